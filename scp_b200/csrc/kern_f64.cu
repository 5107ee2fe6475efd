// kern_f64.cu -- FP64 step kernels (single grid and multi-request).
#include "kern_one.cuh"

namespace scp {
StepFnT<F64> step_fn_f64(int shape, bool g, bool f, bool s, bool d, size_t *smem) {
    return select_one<F64>(shape, g, f, s, d, smem);
}
namespace {
template <int TX, int TY>
StepFnT<F64> pick_diag(bool g, bool d) {
    SCP_PICK4(step_diag_kernel, TX, TY);
}
}  // namespace
StepFnT<F64> step_diag_fn(int shape, bool g, bool d, size_t *smem) {
    switch (shape) {
        case 2: *smem = smem_one<F64, 32, 8>(g); return pick_diag<32, 8>(g, d);
        case 3: *smem = smem_one<F64, 16, 8>(g); return pick_diag<16, 8>(g, d);
        case 4: *smem = smem_one<F64, 64, 2>(g); return pick_diag<64, 2>(g, d);
        default: *smem = smem_one<F64, 32, 4>(g); return pick_diag<32, 4>(g, d);
    }
}
MultiFn<F64> multi_fn_f64(int shape, bool g, bool d, size_t *smem) {
    return select_multi<F64>(shape, g, d, smem);
}
}  // namespace scp
