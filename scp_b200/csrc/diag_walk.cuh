// diag_walk.cuh -- the first diagnostics reduction (energies, charges,
// centroid moments, Gauss residual, E_em; the pass-1 slots of diag.cuh) on the
// plane walker, for FP64 and FP32-compensated states: the state is read once,
// every stencil value comes from shared memory, and every thread keeps its
// sums over all the sites it walks before one block fold at the end.  The
// per-site terms are those of diag_pass1_kernel (compute_energy_complex[_gauge],
// compute_charges, compute_gauss, sfa/sim/scp_sim.c:1823-2243), in FP64 for
// either state; the order of the sums is fixed by the tile plan.
//
// What bounds it: FP64 dependency chains at eight warps per SM beside the one
// read of the state (240 B per site in FP64, 156 B compensated).
#pragma once
#include "step.cuh"
#include "walk.cuh"

namespace scp {

struct DiagWalkArgs {
    int N;
    DiagConsts c;
    // FP64 state: 12 matter positions, th and E (3 each), 12 matter momenta
    const double *x, *th, *E, *mom;
    // compensated state: hi parts (15 arrays), bf16 and fp32 low parts, momenta (15)
    const float *x32;
    const uint16_t *lo;
    const float *tlo, *s32;
    // folding of the CTAs' partials by the last one
    double *part, *fold;
    unsigned *count;
};

// Sums beyond the step's own: the Gauss-law norms, taken here because E of
// the neighbours is staged.
struct DiagWalkSums {
    StepSums s;
    double gl2, nom, fsum, nc, gmax;
};

template <bool GAUGED, bool COMP>
struct DiagWalk {
    static constexpr int TH = 12, EF = 15;
    static constexpr int NR = 18, CF = NR;
    static constexpr int MIN_CTAS = 1;
    static constexpr bool HALO_APART = true, WIDE = false;
    static constexpr bool CONVERT = COMP;     // staged through registers, converted to FP64
    using Args = DiagWalkArgs;
    using MT = typename std::conditional<COMP, float, double>::type;
    struct State {
        double t[12];    // conj(U_0) F (gauged) or F at x - i
        double e0;       // E_0 at x - i
        MT w[12];        // momenta, read one plane ahead
    };

    static constexpr int NR_FEW = 12;         // without links: the matter fields
    __device__ static __forceinline__ bool few(const Args &a) { return !a.c.links; }
    __device__ static __forceinline__ const double *src(const Args &a, int f, long long n3) {
        return f < TH ? a.x + f * n3 : f < EF ? a.th + (f - TH) * n3 : a.E + (f - EF) * n3;
    }
    // staged field f of a compensated state (read-only loads: no launch in
    // flight writes a state whose diagnostics are taken)
    __device__ static __forceinline__ double value(const Args &a, int f, long long n3, long long at) {
        if (f < TH) return (double)__ldg(a.x32 + f * n3 + at) + (double)bf16_to_f(__ldg(a.lo + f * n3 + at));
        if (f < EF) return (double)__ldg(a.x32 + f * n3 + at) + (double)__ldg(a.tlo + (f - TH) * n3 + at);
        return (double)__ldg(a.s32 + (f - EF + TH) * n3 + at);
    }
    __device__ static __forceinline__ void prefetch(const Args &a, int f, long long n3, long long at) {
        prefetch_line_l2(f < EF ? (const void *)(a.x32 + f * n3 + at) : (const void *)(a.s32 + (f - EF + TH) * n3 + at));
        if (f < TH) prefetch_line_l2(a.lo + f * n3 + at);
        else if (f < EF) prefetch_line_l2(a.tlo + (f - TH) * n3 + at);
    }
    __device__ static __forceinline__ MT momentum(const Args &a, int f, long long n3, long long at) {
        if constexpr (COMP) {
            float v;
            asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(a.s32 + f * n3 + at));
            return v;
        } else {
            return ld_early(a.mom + f * n3 + at);
        }
    }

    __device__ static __forceinline__ void load(const Args &a, State &st, long long idx) {
#pragma unroll
        for (int f = 0; f < 12; f++) st.w[f] = momentum(a, f, a.c.N3, idx);
    }
    template <class V>
    __device__ static __forceinline__ void begin(const Args &a, State &st, const V &m, const V &) {
        double ph[1] = {m.get(TH, 0, 0)}, sn[1] = {0.0}, cs[1] = {1.0};
        if (GAUGED) sincos_batch<1, true>(ph, sn, cs);
#pragma unroll
        for (int q = 0; q < 6; q++) {
            const double u = m.get(field_re(q), 0, 0), v = m.get(field_im(q), 0, 0);
            st.t[field_re(q)] = GAUGED ? cs[0] * u + sn[0] * v : u;
            st.t[field_im(q)] = GAUGED ? cs[0] * v - sn[0] * u : v;
        }
        st.e0 = m.get(EF, 0, 0);
    }

    template <class V>
    __device__ static __forceinline__ void site(const Args &a, State &st, const V &c, const V &p, int i, int j, int k,
                                                long long idx, long long next, DiagWalkSums &acc) {
        const DiagConsts &dc = a.c;
        StepSums &S = acc.s;
        double sn[5], cs[5];
        if (GAUGED) {
            double ang[5] = {c.get(TH, 0, 0), c.get(TH + 1, 0, 0), c.get(TH + 2, 0, 0), c.get(TH + 1, -1, 0),
                             c.get(TH + 2, 0, -1)};
            sincos_batch<5, true>(ang, sn, cs);
        }
        double eg = 0.0, etg = 0.0, rho = 0.0, rho2 = 0.0, s3 = 1.0, cr[3], ci[3];
#pragma unroll
        for (int n = 0; n < 6; n++) {
            const int q = (n + 3) % 6;   // Theta first: Phi's coupling needs its curl
            const int fre = field_re(q), fim = field_im(q), b = q % 3;
            const double u = c.get(fre, 0, 0), v = c.get(fim, 0, 0);
#pragma unroll
            for (int d = 0; d < 3; d++) {
                double fr = d == 0 ? p.get(fre, 0, 0) : c.get(fre, d == 1, d == 2);
                double fi = d == 0 ? p.get(fim, 0, 0) : c.get(fim, d == 1, d == 2);
                double br, bi;
                if (d == 0) { br = st.t[fre]; bi = st.t[fim]; }
                else { br = c.get(fre, -(d == 1), -(d == 2)); bi = c.get(fim, -(d == 1), -(d == 2)); }
                if (GAUGED) {
                    const double up = fr, vp = fi;
                    fr = cs[d] * up - sn[d] * vp;
                    fi = cs[d] * vp + sn[d] * up;
                    if (d != 0) {
                        const double um = br, vm = bi;
                        br = cs[2 + d] * um + sn[2 + d] * vm;
                        bi = cs[2 + d] * vm - sn[2 + d] * um;
                    }
                }
                const double dr = fr - br, di = fi - bi;   // central differences, undivided
                if (q < 3) eg += dr * dr + di * di;
                else etg += dr * dr + di * di;
                if (q >= 3 && b != d) {   // curl of Theta
                    const bool plus = (b == (d + 1) % 3);
                    const int t = plus ? (d + 2) % 3 : (d + 1) % 3;
                    const int other = plus ? (t + 1) % 3 : (t + 2) % 3;
                    if (b < other) { cr[t] = plus ? dr : -dr; ci[t] = plus ? di : -di; }
                    else if (plus) { cr[t] += dr; ci[t] += di; }
                    else { cr[t] -= dr; ci[t] -= di; }
                }
            }
            st.t[fre] = GAUGED ? cs[0] * u + sn[0] * v : u;
            st.t[fim] = GAUGED ? cs[0] * v - sn[0] * u : v;
            const double pu = (double)st.w[fre], pv = (double)st.w[fim];
            st.w[fre] = momentum(a, fre, dc.N3, idx + next);
            st.w[fim] = momentum(a, fim, dc.N3, idx + next);
            const double kin = pu * pu + pv * pv, mod = u * u + v * v, ch = u * pv - v * pu;
            rho += ch;
            if (q < 3) {
                S.s[SS_EPK] += kin;
                S.s[SS_EC] += u * cr[b] + v * ci[b];
                S.s[SS_QP0 + b] += ch;
                S.pm = fmax(S.pm, mod);
                rho2 += mod;
                s3 *= mod;
            } else {
                S.s[SS_ETK] += kin;
                S.s[SS_TRS] += mod;
                S.s[SS_QT] += ch;
            }
        }
        S.s[SS_EG] += eg;
        S.s[SS_ETG] += etg;
        S.s[SS_M0] += rho2;
        S.s[SS_EP] += s3 / (1.0 + dc.kappa * s3);
        S.s[SS_PINT] += sqrt(s3);
        S.smax = fmax(S.smax, s3);
        const double x = -dc.L + i * dc.dx, y = -dc.L + j * dc.dx, z = -dc.L + k * dc.dx;
        const double r2 = x * x + y * y + z * z;
        S.s[SS_CX] += x * rho2;
        S.s[SS_CY] += y * rho2;
        S.s[SS_CZ] += z * rho2;
        if (r2 <= dc.R2) S.s[SS_QC] += rho;
        if (dc.links) {   // Gauss law and E_em (also with g = 0: then only E^2/2)
            const double E0 = c.get(EF, 0, 0), E1 = c.get(EF + 1, 0, 0), E2 = c.get(EF + 2, 0, 0);
            const double divE = (E0 - st.e0 + E1 - c.get(EF + 1, -1, 0) + E2 - c.get(EF + 2, 0, -1)) / dc.dx;
            st.e0 = E0;
            const double G = divE - dc.g * rho - dc.G_offset;
            if (r2 < dc.Rint2) {
                acc.gmax = fmax(acc.gmax, fabs(G));
                acc.gl2 += G * G;
                acc.nom += 1.0;
            }
            S.s[SS_EE] += E0 * E0 + E1 * E1 + E2 * E2;
            if (GAUGED) {   // 1 - cos of the plaquettes, as 2 sin^2 of the half angle
                double h[3] = {0.5 * plaq_angle(c, p, TH, 0, 0, 0), 0.5 * plaq_angle(c, p, TH, 1, 0, 0),
                               0.5 * plaq_angle(c, p, TH, 2, 0, 0)};
                sin_batch(h);
                S.s[SS_BB] += 2.0 * (h[0] * h[0] + h[1] * h[1] + h[2] * h[2]);
            }
            if (fabs(x) <= dc.Rcube && fabs(y) <= dc.Rcube && fabs(z) <= dc.Rcube) {
                acc.fsum += divE;
                acc.nc += 1.0;
            }
        }
    }
};

template <class M, int TX, int TY>
__global__ void __launch_bounds__(TX *TY, M::MIN_CTAS) diag_walk_kernel(DiagWalkArgs a, TileGrid tg) {
    extern __shared__ __align__(16) double walk_ring[];
    WalkStage<M, TX, TY> stg(walk_ring, tg.tw);
    DiagWalkSums acc;
    acc.s.clear();
    acc.gl2 = acc.nom = acc.fsum = acc.nc = acc.gmax = 0.0;
    for_each_piece(tg, a.N, [&](const Piece &pc) { walk_item<M, TX, TY>(a, tg, pc, stg, acc); });
    __syncthreads();   // the ring is free: scratch of the fold
    DiagSums o;
    step_sums(acc.s, a.c, o);
    o.S[DS_GL2] = acc.gl2;
    o.S[DS_NOM] = acc.nom;
    o.S[DS_FSUM] = acc.fsum * a.c.dV;
    o.S[DS_NC] = acc.nc;
    o.M[DM_GMAX] = acc.gmax;
    block_fold<DS_NSUM, DM_NMAX>(o.S, o.M, walk_ring, a.part);
    if (last_block_done(a.count)) fold_rows_block<DS_NSUM, DM_NMAX>(a.part, gridDim.x, walk_ring, a.fold);
}

}  // namespace scp
