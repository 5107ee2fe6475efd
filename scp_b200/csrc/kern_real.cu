// kern_real.cu -- the real mode's optional terms (real6.cuh).
#include "real6.cuh"
#include "walk_launch.cuh"

namespace scp {
namespace {

// 384 threads of 168 registers, one CTA per SM: 113 us a step at 128^3 with
// strain and hardening against 119 with 32 x 8 (the perimeter's C and B weigh
// less) and 182 with two CTAs of 32 x 8, whose 213 KB leave the L1 too few
// lines for the copies in flight.
constexpr int kR6X = 32, kR6Y = 12;

template <class MODE, bool AUX>
int r6_plan_of(int N, int nsm, ExtPlan *p) {
    using LY = R6Layout<AUX, kR6X, kR6Y>;
    auto fn = r6_kernel<MODE, AUX, kR6X, kR6Y>;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LY::smem_bytes) != cudaSuccess)
        return -1;
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, LY::NT, LY::smem_bytes) != cudaSuccess || occ < 1)
        return -1;
    int tw = kR6X, th = kR6Y;
    fit_tile(N, LY::NT, LY::TFS, &tw, &th, {2 * (LY::H - 1), 2 * (LY::H - 1), LY::PFS});
    plan_tiles(N, tw, th, nsm * occ, &p->tg, &p->grid);
    p->tx = tw;
    p->ty = th;
    p->smem = LY::smem_bytes;
    return 0;
}

template <class MODE, bool AUX>
cudaError_t r6_launch(const ExtPlan &p, const R6Args &a, cudaStream_t st) {
    return launch_step_kernel(r6_kernel<MODE, AUX, kR6X, kR6Y>, a.N, p.grid, kR6X * kR6Y, p.smem, st, a, p.tg);
}

}  // namespace

int r6_plan(bool aux, int N, int nsm, ExtPlan *plan) {
    for (int v = 0; v < 5; v++) {
        const int rc = with_mode(v == 0, v & 1, v >= 3, [&](auto mode) {
            using M = decltype(mode);
            return aux ? r6_plan_of<M, true>(N, nsm, plan) : r6_plan_of<M, false>(N, nsm, plan);
        });
        if (rc) return rc;
    }
    return 0;
}

cudaError_t r6_step(bool aux, const ExtPlan &plan, const R6Consts &c, const R6IO &io, cudaStream_t st) {
    R6Args a;
    a.x = io.x;
    a.N = c.N;
    a.c = c;
    for (int b = 0; b < 2; b++) {   // six arrays: all in the first group
        a.io.win[b] = io.win;
        a.io.wout[b] = io.wout;
        a.io.xout[b] = io.xout;
        a.io.sout[b] = io.sout;
    }
    a.io.flag = io.flag;
    return with_mode(io.first, io.sync, io.damp, [&](auto mode) {
        using M = decltype(mode);
        return aux ? r6_launch<M, true>(plan, a, st) : r6_launch<M, false>(plan, a, st);
    });
}

}  // namespace scp
