// walk_launch.cuh -- plan and launch of the walker models (walk.cuh), for the
// units that instantiate them.
#pragma once
#include "ext_launch.cuh"
#include "plan.cuh"
#include "walk.cuh"

namespace scp {
namespace {

// Tile of the walker models: up to 256 sites, one CTA per SM with 255
// registers a thread, as the gauged FP64 step.
constexpr int kWalkX = 32, kWalkY = 8;

// the tile of a grid edge: its rows, with the columns its staging keeps on
// either side, fit a ring field
template <class LY>
void walk_tile(int N, int *tw, int *th) {
    constexpr int X = LY::TX_, Y = LY::TY_;
    *tw = X;
    *th = Y;
    fit_tile(N, LY::NT, (X + 2) * (Y + 2), tw, th, {2 * (LY::OFF - 1), 0, LY::FS});
}

template <class M>
int walk_plan_fn(const void *fn, int N, int nsm, ExtPlan *p) {
    using LY = WalkLayout<M, kWalkX, kWalkY>;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LY::smem_bytes) != cudaSuccess)
        return -1;
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, LY::NT, LY::smem_bytes) != cudaSuccess || occ < 1)
        return -1;
    int tw, th;
    walk_tile<LY>(N, &tw, &th);
    plan_tiles(N, tw, th, nsm * occ, &p->tg, &p->grid);
    p->tx = tw;
    p->ty = th;
    p->smem = LY::smem_bytes;
    return 0;
}

template <class M>
int walk_plan(int N, int nsm, ExtPlan *p) {
    return walk_plan_fn<M>((const void *)walk_kernel<M, kWalkX, kWalkY>, N, nsm, p);
}

template <class M>
cudaError_t walk_launch(const ExtPlan &p, const typename M::Args &a, cudaStream_t st) {
    using LY = WalkLayout<M, kWalkX, kWalkY>;
    return launch_step_kernel(walk_kernel<M, kWalkX, kWalkY>, a.N, p.grid, LY::NT, LY::smem_bytes, st, a, p.tg);
}

// run f(StepMode) for the launch's mode
template <class F>
auto with_mode(int first, int sync, int damp, F &&f) {
    if (first) return f(StepMode<true, false, false>());   // no closing kick, nothing synchronous
    if (sync) return damp ? f(StepMode<false, true, true>()) : f(StepMode<false, true, false>());
    return damp ? f(StepMode<false, false, true>()) : f(StepMode<false, false, false>());
}

}  // namespace
}  // namespace scp
