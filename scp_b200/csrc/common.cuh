// common.cuh -- shared device-side definitions of libscpgpu (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace scp {

// Packed field slots used by every device buffer.  Positions X: u0..2 v0..2
// tu0..2 tv0..2 th0..2; momenta W/S: du0..2 dv0..2 dtu0..2 dtv0..2 E0..2.
enum : int { FU = 0, FV = 3, FTU = 6, FTV = 9, FTH = 12 };

// Constants of one stepper instance, passed by value (kernel parameter bank).
struct StepConsts {
    int N;
    long long N3;
    double idx2, idx1, inva;      // 1/dx^2, 1/(2dx), 1/dx
    double m2, mtheta2, eta, mu, kappa;
    double dt, hdt, gad;          // gad = -g*dx*dt (link drift prefactor)
    double g, stp;                // stp = 1/(g dx^3) (staple prefactor)
    double L, dx, damp_width, damp_rate;
    int prefetch;                 // 1: prefetch the next plane's momenta into L2 at the top of a plane
    // diagnostics summed by synchronous FP64 launches: cell volume, core
    // radius^2 of Q_core, plaquette-energy prefactor 1/(g^2 dx^4)
    double dV, R2, bpre;
    // products the gauged site function uses: eta/(2dx), eta dx/2, g/dx
    double ei, cross, gi;
};

// Work decomposition of the persistent step kernels: the grid is cut into
// (TX x TY) columns in (k, j) and segments of seg planes along i.
struct TileGrid {
    int ntx, nty, nseg, seg;
    int nitems;
    int tw, th;   // sites of a tile along k and j
};

// A run of planes [i0, i1) of column (kt, jt).
struct Piece {
    int kt, jt, i0, i1;
};

// Work item -> piece.  Items enumerate the columns fastest and the segments
// last, so the CTAs of one wave start on the same plane and walk i in step.
__device__ __forceinline__ Piece piece_of_item(const TileGrid &tg, int item, int N) {
    Piece p;
    p.kt = item % tg.ntx;
    p.jt = (item / tg.ntx) % tg.nty;
    const int sg = item / (tg.ntx * tg.nty);
    p.i0 = sg * tg.seg;
    p.i1 = min(p.i0 + tg.seg, N);
    return p;
}

// Every piece of this CTA, in order (items blockIdx.x, + gridDim.x, ...).
template <class F>
__device__ __forceinline__ void for_each_piece(const TileGrid &tg, int N, F &&f) {
    for (int item = blockIdx.x; item < tg.nitems; item += gridDim.x) f(piece_of_item(tg, item, N));
}

__device__ __forceinline__ void cp_async8(void *smem, const void *gmem) {
    unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
// 16 bytes past L1 (both addresses 16-byte aligned): no L1 line is held while
// the copy is in flight
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
    unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int NPEND>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(NPEND) : "memory");
}

// Programmatic dependent launch: a step launch's CTAs may become resident while
// the launch before it still runs; griddep_wait returns once that launch has
// completed and its writes are visible (at once where there is none, or for an
// ordinary launch), griddep_launch lets the next one become resident.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// Bring the line holding p into L2 ahead of its use (a hint: no register, no wait).
__device__ __forceinline__ void prefetch_line_l2(const void *p) {
    asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p));
}

// Streaming store (evict-first): outputs are not re-read by this launch.
__device__ __forceinline__ void st_cs(double *p, double v) { __stcs(p, v); }
__device__ __forceinline__ void st_cs(float *p, float v) { __stcs(p, v); }

// Link-angle wrap to (-pi, pi], the reference's v - 2*pi*rint(v/(2*pi))
// (sfa/sim/scp_sim.c:1647).
__device__ __forceinline__ double wrap_angle(double v) {
    const double twopi = 2.0 * 3.14159265358979323846;
    return v - twopi * rint(v / twopi);
}

// link wrap into (-pi, pi] (reference: v - 2*pi*rint(v/(2*pi)), scp_sim.c:1647);
// |v| < 3 never wraps, so the division only runs for the rare large angles
__device__ __forceinline__ double link_wrap(double v) {
    if (fabs(v) < 3.0) return v;
    return wrap_angle(v);
}

// A load that stays where it is written: the compiler does not move it down to
// its first use, so its latency passes under what follows, nor above
// griddep_wait.  An ordinary (coherent) load: a step reads momenta that it
// overwrites itself and, as a dependent launch, that the launch before it may
// still be writing while this one is already resident; the read-only path
// (ld.global.nc, __ldg) promises nothing for such data.
__device__ __forceinline__ double ld_early(const double *p) {
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_early(const float *p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint16_t ld_early(const uint16_t *p) {
    uint16_t v;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}

__device__ __forceinline__ int wrapi(int x, int N) { return x < 0 ? x + N : (x >= N ? x - N : x); }

// (i, j, k) of site idx = (i*N + j)*N + k: 32-bit divisions while the index
// fits (N <= 1625), 64-bit beyond
__device__ __forceinline__ void site_ijk(long long idx, int N, int *i, int *j, int *k) {
    if (idx <= 0xFFFFFFFFll) {
        const unsigned u = (unsigned)idx, n = (unsigned)N, nn = n * n;
        const unsigned ii = u / nn, r = u - ii * nn, jj = r / n;
        *i = (int)ii;
        *j = (int)jj;
        *k = (int)(r - jj * n);
    } else {
        const long long NN = (long long)N * N;
        *i = (int)(idx / NN);
        *j = (int)((idx / N) % N);
        *k = (int)(idx % N);
    }
}

}  // namespace scp
