// kern_fabric.cu -- the three-fabric stepper (fabrics.cuh).
#include "fabrics.cuh"
#include "walk_launch.cuh"

namespace scp {
namespace {

template <class MODE>
int fabric_plan_of(int N, int nsm, ExtPlan *plan) {
    if (walk_plan<FabricPass<MODE, true, false, false>>(N, nsm, plan)) return -1;
    if (walk_plan<FabricPass<MODE, false, true, false>>(N, nsm, plan)) return -1;
    if (walk_plan<FabricPass<MODE, false, true, true>>(N, nsm, plan)) return -1;
    return walk_plan<FabricPass<MODE, false, false, false>>(N, nsm, plan);
}

template <class MODE, bool SECOND, bool ACC, bool LINKS>
cudaError_t fabric_launch(const ExtPlan &p, const FabConsts &c, const FabIO &io, cudaStream_t st) {
    typename FabricPass<MODE, SECOND, ACC, LINKS>::Args a;
    for (int b = 0; b < 2; b++) {
        a.src[b] = io.src[b];
        a.io.win[b] = io.win[b];
        a.io.wout[b] = io.wout[b];
        a.io.xout[b] = io.xout[b];
        a.io.sout[b] = io.sout[b];
    }
    a.N = c.N;
    a.c = c;
    a.qf = io.qf;
    a.gqf = io.gqf;
    a.qx = io.qx;
    a.gqx = io.gqx;
    a.io.flag = io.flag;
    a.kacc = io.kacc;
    return walk_launch<FabricPass<MODE, SECOND, ACC, LINKS>>(p, a, st);
}

}  // namespace

// the passes share their plan (same staged fields and tile)
int fabric_plan(int N, int nsm, ExtPlan *plan) {
    for (int v = 0; v < 5; v++) {
        const int rc = with_mode(v == 0, v & 1, v >= 3,
                                 [&](auto mode) { return fabric_plan_of<decltype(mode)>(N, nsm, plan); });
        if (rc) return rc;
    }
    return 0;
}

cudaError_t fabric_step(const ExtPlan &plan, const FabConsts &c, const FabIO &io, cudaStream_t st) {
    return with_mode(io.first, io.sync, io.damp, [&](auto mode) {
        using M = decltype(mode);
        if (io.links) return fabric_launch<M, false, true, true>(plan, c, io, st);
        if (io.accumulate) return fabric_launch<M, false, true, false>(plan, c, io, st);
        return io.second ? fabric_launch<M, true, false, false>(plan, c, io, st)
                         : fabric_launch<M, false, false, false>(plan, c, io, st);
    });
}

}  // namespace scp
