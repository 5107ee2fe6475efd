// kern_diag.cu -- the first diagnostics reduction on the plane walker (diag_walk.cuh).
#include "diag_walk.cuh"
#include "walk_launch.cuh"

namespace scp {
namespace {

template <bool G, bool COMP>
int plan_of(int N, int nsm, ExtPlan *p) {
    using M = DiagWalk<G, COMP>;
    return walk_plan_fn<M>((const void *)diag_walk_kernel<M, kWalkX, kWalkY>, N, nsm, p);
}
template <bool G, bool COMP>
cudaError_t launch_of(const ExtPlan &p, const DiagWalkArgs &a, cudaStream_t st) {
    using M = DiagWalk<G, COMP>;
    using LY = WalkLayout<M, kWalkX, kWalkY>;
    diag_walk_kernel<M, kWalkX, kWalkY><<<p.grid, LY::NT, LY::smem_bytes, st>>>(a, p.tg);
    return cudaGetLastError();
}

}  // namespace

int diag_walk_plan(bool gauged, bool comp, int N, int nsm, ExtPlan *p) {
    if (comp) return gauged ? plan_of<true, true>(N, nsm, p) : plan_of<false, true>(N, nsm, p);
    return gauged ? plan_of<true, false>(N, nsm, p) : plan_of<false, false>(N, nsm, p);
}

cudaError_t diag_walk(bool gauged, bool comp, const ExtPlan &p, const DiagWalkArgs &a, cudaStream_t st) {
    if (comp) return gauged ? launch_of<true, true>(p, a, st) : launch_of<false, true>(p, a, st);
    return gauged ? launch_of<true, false>(p, a, st) : launch_of<false, false>(p, a, st);
}

}  // namespace scp
