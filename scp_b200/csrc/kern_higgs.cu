// kern_higgs.cu -- the Higgs / second-gauge stepper (higgs_u1.cuh).
#include "higgs_u1.cuh"
#include "walk_launch.cuh"

namespace scp {
namespace {

// the plan of one extension set; every mode of it gets its shared memory
template <bool H, bool G>
int hu_plan_of(int N, int nsm, ExtPlan *p) {
    for (int v = 0; v < 5; v++) {
        const int rc = with_mode(v == 0, v & 1, v >= 3, [&](auto mode) {
            return walk_plan<HiggsU1<decltype(mode), H, G>>(N, nsm, p);
        });
        if (rc) return rc;
    }
    return 0;
}

template <class MODE, bool H, bool G>
cudaError_t hu_launch(const ExtPlan &p, const HuConsts &c, const HuIO &io, cudaStream_t st) {
    using M = HiggsU1<MODE, H, G>;
    typename M::Args a;
    const long long n3 = c.N3, at[2] = {0, 12 * n3};
    a.x = io.x;
    a.N = c.N;
    a.c = c;
    for (int b = 0; b < 2; b++) {
        a.io.win[b] = io.win + at[b];
        a.io.wout[b] = io.wout + at[b];
        a.io.xout[b] = io.xout + at[b];
        a.io.sout[b] = io.sout + at[b];
    }
    a.io.flag = io.flag;
    return walk_launch<M>(p, a, st);
}

template <bool H, bool G>
cudaError_t hu_step_of(const ExtPlan &p, const HuConsts &c, const HuIO &io, cudaStream_t st) {
    return with_mode(io.first, io.sync, io.damp,
                     [&](auto mode) { return hu_launch<decltype(mode), H, G>(p, c, io, st); });
}

}  // namespace

int hu_plan(bool higgs, bool g2, int N, int nsm, ExtPlan *plan) {
    if (higgs && g2) return hu_plan_of<true, true>(N, nsm, plan);
    if (higgs) return hu_plan_of<true, false>(N, nsm, plan);
    return hu_plan_of<false, true>(N, nsm, plan);
}

cudaError_t hu_step(bool higgs, bool g2, const ExtPlan &plan, const HuConsts &c, const HuIO &io, cudaStream_t st) {
    if (higgs && g2) return hu_step_of<true, true>(plan, c, io, st);
    if (higgs) return hu_step_of<true, false>(plan, c, io, st);
    return hu_step_of<false, true>(plan, c, io, st);
}

}  // namespace scp
