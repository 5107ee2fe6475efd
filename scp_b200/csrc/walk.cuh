// walk.cuh -- plane walker of the extension steppers (Higgs and second gauge,
// three fabrics).
//
// The work split is the fused step's (step.cuh): tile columns of tw x th
// sites times segments of planes along i; a CTA streams its column through a
// 3-slot shared-memory ring of NR staged fields (plane i, plane i+1, plane
// i+2 in flight), and what a site needs of plane i-1 and its momenta, read
// one plane ahead, stay in registers.
//
// A model supplies
//   NR, CF         staged fields, of which those from CF on are staged at the
//                  two corners (j+1, k-1) and (j-1, k+1) too
//   src(args, f, n3)   the N^3 array of staged field f
//   NR_FEW, few(args)  a launch may stage only the first NR_FEW fields
//   CONVERT        the fields are not FP64 arrays: value(args, f, n3, at) is
//                  field f at element `at`, prefetch() its L2 prefetch; a plane
//                  is then staged through registers, prefetched a plane ahead
//   HALO_APART     own copies of a plane first, then the halo's, instead of
//                  field by field: 375 against 397 us for a step of three
//                  fabrics at 128^3, but 365 against 321 with the 19 fields of
//                  the Higgs and second gauge
//   WIDE           rows in 16-byte copies past L1 where the edge and the tile
//                  are even: 303 against 324 us for the 19 fields of the Higgs
//                  and second gauge, whose 155 KB ring leaves the L1 fewer
//                  lines than their copies hold; 377 against 365 for the three
//                  fabrics' 15
//   Args           kernel arguments, with `int N`
//   State          per-thread state kept along the i walk
//   load(args, st, idx)                first plane's global loads
//   begin(args, st, m, c)              carry from the plane before the first
//   site(args, st, c, p, i, j, k, idx, next)   the work at one site; next:
//                  elements to the next plane's site, 0 on a segment's last
//                  (what is then read ahead is not used: a load behind a
//                  branch would be copied where the branch joins, and wait)
// and runs as walk_kernel<Model, TX, TY>.
#pragma once
#include <type_traits>

#include "gauged.cuh"

namespace scp {

template <class M, int TX, int TY>
struct WalkLayout {
    static constexpr int TX_ = TX, TY_ = TY;
    static constexpr int NR = M::NR;
    static constexpr int OFF = M::WIDE ? 2 : 1;      // columns before the tile's first
    static constexpr int FS = (TX + 2 * OFF) * (TY + 2);   // ring elements of one field
    static constexpr int PLANE = NR * FS;
    static constexpr int NT = TX * TY;
    static constexpr int HPT = (2 * TX + 2 * TY + 2 + NT - 1) / NT;
    static_assert(HPT == 1, "one halo site per thread at most");
    static constexpr size_t smem_bytes = sizeof(double) * 3 * PLANE;
};

template <class M, int TX, int TY>
struct WalkStage {
    using LY = WalkLayout<M, TX, TY>;
    double *xs;
    int tx, ty, pitch, c_s, own_g, h_s, h_g, h_f0;
    bool act, wide, chunk;

    struct View {
        const double *p;
        int pitch;
        __device__ __forceinline__ double get(int f, int dj, int dk) const { return p[f * LY::FS + dj * pitch + dk]; }
        __device__ __forceinline__ double again(int f) const { return get(f, 0, 0); }
    };
    __device__ __forceinline__ View view(int slot) const { return View{xs + slot * LY::PLANE + c_s, pitch}; }

    __device__ __forceinline__ WalkStage(double *ring, int tw) : xs(ring) {
        ty = (int)threadIdx.x / tw;
        tx = (int)threadIdx.x - ty * tw;
        pitch = tw + 2 * LY::OFF;
        c_s = (ty + 1) * pitch + tx + LY::OFF;
    }
    // this thread's own site and its halo copy: rows j0-1 and j0+nj, columns
    // k0-1 and k0+nk, two corners (fields from h_f0 on; M::NR: no copy)
    __device__ __forceinline__ void begin(int N, int k0, int j0, int nk, int nj) {
        act = tx < nk && ty < nj;
        own_g = (j0 + ty) * N + k0 + tx;
        int h = threadIdx.x, r = 0, col = 0;
        h_f0 = M::NR;
        chunk = false;
        // even edges and tiles, WIDE models: rows -1 .. nj in 16-byte chunks
        wide = M::WIDE && ((N | pitch) & 1) == 0;
        if (wide) {
            const int nch = nk / 2, nc = nch * (nj + 2);
            if (h < nc) { r = h / nch; col = 1 + 2 * (h - r * nch); h_f0 = 0; chunk = true; }
            h += 2 * nk - nc;   // the columns and corners follow
        } else if (h < nk) { r = 0; col = h + 1; h_f0 = 0; }
        else if (h < 2 * nk) { r = nj + 1; col = h - nk + 1; h_f0 = 0; }
        if (!chunk && h >= 2 * nk) {
            if (h < 2 * nk + nj) { r = h - 2 * nk + 1; col = 0; h_f0 = 0; }
            else if (h < 2 * nk + 2 * nj) { r = h - 2 * nk - nj + 1; col = nk + 1; h_f0 = 0; }
            else if (h == 2 * nk + 2 * nj) { r = nj + 1; col = 0; h_f0 = M::CF; }
            else if (h == 2 * nk + 2 * nj + 1) { r = 0; col = nk + 1; h_f0 = M::CF; }
        }
        h_s = r * pitch + col + LY::OFF - 1;
        h_g = wrapi(j0 - 1 + r, N) * N + wrapi(k0 - 1 + col, N);
    }
    // f(the number of fields this launch stages, as a constant)
    template <class F>
    __device__ __forceinline__ static void with_staged(const typename M::Args &a, F &&f) {
        if (M::NR_FEW < M::NR && M::few(a)) f(std::integral_constant<int, M::NR_FEW>());
        else f(std::integral_constant<int, M::NR>());
    }
    __device__ __forceinline__ void issue(const typename M::Args &a, long long n3, int plane, int slot) {
        const long long pb = (long long)wrapi(plane, a.N) * a.N * a.N;
        double *sb = xs + slot * LY::PLANE;
        if constexpr (M::CONVERT) {
            static_assert(M::CF == M::NR, "converted staging brings no corners");
            const long long nb = (long long)wrapi(plane + 1, a.N) * a.N * a.N + own_g;
            with_staged(a, [&](auto nf) {   // own sites, the next plane's prefetch, the halo
                constexpr int NF = decltype(nf)::value;
                if (act) {
                    double v[NF];
#pragma unroll
                    for (int f = 0; f < NF; f++) v[f] = M::value(a, f, n3, pb + own_g);
#pragma unroll
                    for (int f = 0; f < NF; f++) M::prefetch(a, f, n3, nb);
#pragma unroll
                    for (int f = 0; f < NF; f++) sb[f * LY::FS + c_s] = v[f];
                }
                if (h_f0 == 0) {
                    double v[NF];
#pragma unroll
                    for (int f = 0; f < NF; f++) v[f] = M::value(a, f, n3, pb + h_g);
#pragma unroll
                    for (int f = 0; f < NF; f++) sb[f * LY::FS + h_s] = v[f];
                }
            });
        } else if (M::WIDE && wide) {
            with_staged(a, [&](auto nf) {
                constexpr int NF = decltype(nf)::value;
                if (chunk) {
#pragma unroll
                    for (int f = 0; f < NF; f++) cp_async16(sb + f * LY::FS + h_s, M::src(a, f, n3) + pb + h_g);
                } else if (h_f0 == 0) {
#pragma unroll
                    for (int f = 0; f < NF; f++) cp_async8(sb + f * LY::FS + h_s, M::src(a, f, n3) + pb + h_g);
                }
            });
            if (M::CF < M::NR && h_f0 == M::CF) {
#pragma unroll
                for (int f = M::CF; f < M::NR; f++) cp_async8(sb + f * LY::FS + h_s, M::src(a, f, n3) + pb + h_g);
            }
        } else if constexpr (M::HALO_APART) {
            with_staged(a, [&](auto nf) {
                constexpr int NF = decltype(nf)::value;
                if (act) {
#pragma unroll
                    for (int f = 0; f < NF; f++) cp_async8(sb + f * LY::FS + c_s, M::src(a, f, n3) + pb + own_g);
                }
                if (h_f0 == 0) {
#pragma unroll
                    for (int f = 0; f < NF; f++) cp_async8(sb + f * LY::FS + h_s, M::src(a, f, n3) + pb + h_g);
                }
            });
            if (M::CF < M::NR && h_f0 == M::CF) {
#pragma unroll
                for (int f = M::CF; f < M::NR; f++) cp_async8(sb + f * LY::FS + h_s, M::src(a, f, n3) + pb + h_g);
            }
        } else {
#pragma unroll
            for (int f = 0; f < M::NR; f++) {
                if (act) cp_async8(sb + f * LY::FS + c_s, M::src(a, f, n3) + pb + own_g);
                if (f >= h_f0) cp_async8(sb + f * LY::FS + h_s, M::src(a, f, n3) + pb + h_g);
            }
        }
        cp_async_commit();
    }
};

// Extra arguments (a reduction's per-thread sums) are passed on to M::site.
template <class M, int TX, int TY, class... Extra>
__device__ __forceinline__ void walk_item(const typename M::Args &a, const TileGrid &tg, const Piece &pc,
                                          WalkStage<M, TX, TY> &stg, Extra &...extra) {
    const int N = a.N;
    const long long NN = (long long)N * N, n3 = NN * N;
    const int k0 = pc.kt * tg.tw, j0 = pc.jt * tg.th, i0 = pc.i0, i1 = pc.i1;
    stg.begin(N, k0, j0, min(tg.tw, N - k0), min(tg.th, N - j0));
    const int j = j0 + stg.ty, k = k0 + stg.tx;
    __syncthreads();   // the previous item's last plane has been read
    stg.issue(a, n3, i0 - 1, 0);
    stg.issue(a, n3, i0, 1);
    stg.issue(a, n3, i0 + 1, 2);
    typename M::State st;
    if (stg.act) M::load(a, st, (long long)i0 * NN + stg.own_g);
    cp_async_wait<1>();
    __syncthreads();
    if (stg.act) M::begin(a, st, stg.view(0), stg.view(1));
    for (int i = i0; i < i1; i++) {
        // plane p sits in slot (p - i0 + 1) mod 3; plane i+2 reuses the slot of i-1
        const int sc = (i - i0 + 1) % 3, sp = (i - i0 + 2) % 3, sn = (i - i0) % 3;
        cp_async_wait<0>();
        __syncthreads();
        if (i + 2 <= i1) stg.issue(a, n3, i + 2, sn);
        if (stg.act)
            M::site(a, st, stg.view(sc), stg.view(sp), i, j, k, (long long)i * NN + stg.own_g, i + 1 < i1 ? NN : 0,
                    extra...);
    }
}

template <class M, int TX, int TY>
__global__ void __launch_bounds__(TX *TY, M::MIN_CTAS) walk_kernel(typename M::Args a, TileGrid tg) {
    extern __shared__ __align__(16) double walk_ring[];
    WalkStage<M, TX, TY> stg(walk_ring, tg.tw);
    griddep_wait();
    griddep_launch();
    for_each_piece(tg, a.N, [&](const Piece &pc) { walk_item<M, TX, TY>(a, tg, pc, stg); });
}

// ---------------------------------------------------------------- leapfrog

// Where a walker model's state lives: slots 0-11 (matter) at [0], the rest
// (links, second links, Higgs) at [1], consecutive N^3 arrays.
struct LeapIO {
    const double *win[2];    // w_n (v_0 on the first launch)
    double *wout[2];         // w_{n+1} (may alias win)
    double *xout[2];         // x_{n+2}
    double *sout[2];         // v_{n+1} (synchronous launches)
    int *flag;
};

// Which step a launch takes: FIRST reads v_0 in place of w and takes no
// closing kick, SYNC also stores v_{n+1}, DAMP has the sponge.
template <bool FIRST_, bool SYNC_, bool DAMP_>
struct StepMode {
    static constexpr bool FIRST = FIRST_, SYNC = SYNC_, DAMP = DAMP_;
};

// Kick, sponge, kick and drift of one slot at one site (the fused scheme of
// the main step: v = (w + hdt a) damp, w' = v + hdt a, x' = x + dt w'),
// explicitly rounded.  w: the site's momenta, read one plane ahead.
template <class MODE, int NM>
struct LeapSite {
    const LeapIO &io;
    double (&w)[NM];
    const long long n3, site, next;
    const double hdt, dt, dmp;
    bool bad = false;

    __device__ __forceinline__ static const double *at(const double *const (&b)[2], int f, long long n3) {
        return f < 12 ? b[0] + f * n3 : b[1] + (f - 12) * n3;
    }
    __device__ __forceinline__ static double *at(double *const (&b)[2], int f, long long n3) {
        return f < 12 ? b[0] + f * n3 : b[1] + (f - 12) * n3;
    }
    __device__ __forceinline__ double kick(int f, double a, double damp, double *wn) {
        double v = MODE::FIRST ? w[f] : rfma(hdt, a, w[f]);
        if (MODE::DAMP && !MODE::FIRST) v = rmul(v, damp);
        *wn = rfma(hdt, a, v);
        return v;
    }
    __device__ __forceinline__ void store(int f, double x, double v, double wn) {
        st_cs(at(io.xout, f, n3) + site, x);
        at(io.wout, f, n3)[site] = wn;
        if (MODE::SYNC) {
            st_cs(at(io.sout, f, n3) + site, v);
            bad |= !isfinite(x) || !isfinite(v);
        }
        // the next plane's momentum, behind the stores, which the compiler does
        // not move it across (ahead of them: Higgs and second gauge 322 against
        // 296 us at 113^3, three fabrics 368 against 352 at 128^3)
        w[f] = ld_early(at(io.win, f, n3) + site + next);
    }
    __device__ __forceinline__ void put(int f, double x, double a, double damp) {
        double wn;
        const double v = kick(f, a, damp, &wn);
        store(f, rfma(dt, wn, x), v, wn);
    }
    __device__ __forceinline__ void put_link(int f, double th, double K, double gad, double damp) {
        double Eh;
        const double E = kick(f, K, damp, &Eh);
        store(f, link_wrap(rfma(gad, Eh, th)), E, Eh);
    }
};

}  // namespace scp
