// kern_ext.cu -- instantiations and launchers of the plane-ring kernels of the
// real mode's optional terms.
#include "ext_launch.cuh"
#include "real6.cuh"

namespace scp {

namespace {

// Tile of a ring model: 128 threads, so that two CTAs share an SM and one
// CTA's plane barrier overlaps the other's work; 32 x 4 while the 4-slot ring
// of NR fields fits twice in shared memory, 16 x 8 (narrower halo rows) for
// the widest rings.
template <class M>
struct TileOf {
    static constexpr int TX = (M::NR <= 17) ? 32 : 16;
    static constexpr int TY = (M::NR <= 17) ? 4 : 8;
    static constexpr int NT = TX * TY;
};

template <class M>
int ring_plan(int N, int nsm, ExtPlan *p) {
    constexpr int TX = TileOf<M>::TX, TY = TileOf<M>::TY;
    using S = RingShape<M::NR, TX, TY>;
    auto fn = ring_kernel<M, TX, TY>;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::smem_bytes) != cudaSuccess)
        return -1;
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, TX * TY, S::smem_bytes) != cudaSuccess || occ < 1)
        return -1;
    plan_ring_tiles(N, TX, TY, nsm * occ, p);
    p->smem = S::smem_bytes;
    return 0;
}

}  // namespace

int r6_plan(bool aux, int N, int nsm, ExtPlan *aux_plan, ExtPlan *step_plan) {
    if (aux) {
        if (ring_plan<R6Aux>(N, nsm, aux_plan)) return -1;
        return ring_plan<R6Step<true>>(N, nsm, step_plan);
    }
    return ring_plan<R6Step<false>>(N, nsm, step_plan);
}

namespace {
template <bool AUX>
cudaError_t r6_launch(const ExtPlan &p, const R6Consts &c, const R6IO &io, cudaStream_t st) {
    using M = R6Step<AUX>;
    typename M::Args a;
    const long long n3 = c.N3;
    for (int f = 0; f < 6; f++) a.src.f[f] = io.x + f * n3;
    if (AUX)
        for (int f = 0; f < 6; f++) a.src.f[6 + f] = io.aux + f * n3;
    a.N = c.N;
    a.c = c;
    a.win = io.win;
    a.wout = io.wout;
    a.xout = io.xout;
    a.sout = io.sout;
    a.flag = io.flag;
    a.first = io.first;
    a.sync = io.sync;
    a.damp = io.damp;
    ring_kernel<M, TileOf<M>::TX, TileOf<M>::TY><<<p.grid, TileOf<M>::NT, p.smem, st>>>(a, p.tg);
    return cudaGetLastError();
}
}  // namespace

cudaError_t r6_step(const ExtPlan &aux_plan, const ExtPlan &step_plan, const R6Consts &c, const R6IO &io,
                    cudaStream_t st) {
    if (!io.aux) return r6_launch<false>(step_plan, c, io, st);
    R6Aux::Args a;
    for (int f = 0; f < 6; f++) a.src.f[f] = io.x + f * c.N3;
    a.N = c.N;
    a.c = c;
    a.aux = io.aux;
    using T = TileOf<R6Aux>;
    ring_kernel<R6Aux, T::TX, T::TY><<<aux_plan.grid, T::NT, aux_plan.smem, st>>>(a, aux_plan.tg);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return r6_launch<true>(step_plan, c, io, st);
}

}  // namespace scp
