// step2.cuh -- the FP32-compensated leapfrog step with two neighbouring sites
// (k, k+1) per thread, computed with the packed FP32 instructions of sm_100
// (vec2.cuh).  Same time integration, state layout and compensated
// bookkeeping as step_item<F32C> in step.cuh; what changes is the work split:
//
//  * a thread owns the site pair (k, k+1), k even, so every field of the pair
//    is one 8-byte word in global and shared memory (one cp.async, one
//    LDS.64, one STG.64 per field and pair; the bf16 low parts of a pair are
//    one 32-bit word);
//  * the arithmetic of both sites is one FFMA2 / FADD2 / FMUL2 stream, which
//    halves the instructions that bound the one-site FP32C kernel;
//  * the k +- 1 neighbours come from the pair itself plus one scalar load.
//
// Requirements: N even (pairs never straddle a row end and every pair is
// 8-byte aligned) and an even tile width.  The host picks this kernel for
// FP32C grids with even N and the one-site kernel otherwise.
//
// Shared-memory ring: [3 slots][NR fields][TY + 2 rows][TX + 4 columns];
// interior sites sit in columns 2..TX+1 so pairs start on even columns, the
// k-1 / k+1 halo columns are 1 and TX+2.
#pragma once
#include "step.cuh"
#include "vec2.cuh"

#ifndef SCP_PAIR_THREADS_PER_SM
#define SCP_PAIR_THREADS_PER_SM 256
#endif

namespace scp {

template <int TX, int TY, bool GAUGED>
struct Step2Layout {
    static_assert(TX % 2 == 0, "site pairs along k need an even tile width");
    static constexpr int NF = GAUGED ? 15 : 12;
    static constexpr int NR = NF + (GAUGED ? 3 : 0);     // ring fields (+ link low parts)
    static constexpr int PX = TX + 4, PY = TY + 2;
    static constexpr int FS = PY * PX;                     // ring elements of one field (tw + 4) x (th + 2)
    static constexpr int PLANE = NR * FS;
    static constexpr int NT = (TX / 2) * TY;
    static constexpr int NHALO = TX + 2 * TY + (GAUGED ? 2 : 0);   // pair rows + single columns + corners
    static constexpr int HPT = (NHALO + NT - 1) / NT;
    static constexpr size_t smem_bytes = sizeof(float) * (size_t)(3 * PLANE);
    // resident threads per SM the register allocation is sized for
    // (256: up to 255 registers a thread)
    static constexpr int MIN_BLOCKS = (SCP_PAIR_THREADS_PER_SM / NT) > 0 ? SCP_PAIR_THREADS_PER_SM / NT : 1;
};

__device__ __forceinline__ V2 bf16x2_to_v2(uint32_t u) {
    return V2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}
__device__ __forceinline__ uint32_t v2_to_bf16x2(V2 a) {
    return (uint32_t)f_to_bf16(a.v.x) | ((uint32_t)f_to_bf16(a.v.y) << 16);
}
__device__ __forceinline__ void st_cs2(float *p, V2 a) { __stcs(reinterpret_cast<float2 *>(p), a.v); }

// Link angle drift with the 2 pi wrap, one lane (th, lo: compensated pair).
__device__ __forceinline__ void link_wrap_c(float *th, float *lo) {
    if (fabsf(*th) > 3.0f) {
        const float kq = rintf(*th * 0.159154943091895336f);
        float t1, e1;
        two_sum(*th, -kq * 6.28318548202514648f, &t1, &e1);   // 2 pi (fp32) times |kq| <= 1
        const float l = *lo + e1 + kq * 1.74845553e-7f;        // 2 pi = 6.2831855f - 1.748e-7
        two_sum(t1, l, th, lo);
    }
}

// The values around one site pair in one ring slot.
template <class LY>
struct PairView {
    const float *p;
    int pitch;
    __device__ __forceinline__ V2 get(int f, int dj, int dk) const {
        const float *q = p + f * LY::FS + dj * pitch;
        if (dk == 0) return V2(*reinterpret_cast<const float2 *>(q));
        if (dk > 0) return V2(q[1], q[2]);
        return V2(q[-1], q[0]);
    }
};

// The pair's momenta and position low parts, read one plane ahead: each is
// replaced by the next plane's behind the stores that follow its use, which the
// compiler does not move the load across (ahead of them: 153 against 148 us a
// gauged step at 128^3, 175 against 151 at 144^3 without links).
template <bool GAUGED>
struct PairAhead {
    V2 w[GAUGED ? 15 : 12];
    uint32_t lo[12];
};

__device__ __forceinline__ V2 ld_early2(const float *p) {
    float2 v;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return V2(v);
}
__device__ __forceinline__ uint32_t ld_early_u32(const uint16_t *p) {
    uint32_t v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// Kicks, damping and compensated drift of one site pair (scp_sim.c:1591-1715,
// fused) as the accelerations come in.
template <bool GAUGED, bool FIRST>
struct PairUpdate {
    const StepIO<F32C> &io;
    const StepConsts &c;
    PairAhead<GAUGED> &m;
    const long long site, next;
    const bool SYNC, DAMP;
    V2 dt, hdt, dt_lo, hdt_lo, dmp;
    bool bad = false;

    // kicks with dt and dt/2 as fp32 pairs: the increment is formed first and
    // added in one rounding (lo*a folded into w first would be lost below half
    // an ulp and run the kick with fp32(dt))
    __device__ __forceinline__ V2 kick(int f, V2 a, V2 *wn) {
        const V2 w = m.w[f];
        const V2 ha = fma2(hdt, a, hdt_lo * a);
        V2 v = FIRST ? w : w + ha;
        if (DAMP && !FIRST) v = v * dmp;
        *wn = (DAMP || FIRST) ? v + ha : w + fma2(dt, a, dt_lo * a);
        return v;
    }
    __device__ __forceinline__ void store(int f, V2 x, V2 v, V2 wn) {
        st_cs2(io.xout + f * c.N3 + site, x);
        *reinterpret_cast<float2 *>(io.wout + f * c.N3 + site) = wn.v;
        if (SYNC && !FIRST) {
            st_cs2(io.sout + f * c.N3 + site, v);
            bad |= !isfinite(x.v.x) || !isfinite(x.v.y) || !isfinite(v.v.x) || !isfinite(v.v.y);
        }
        m.w[f] = ld_early2(io.win + f * c.N3 + site + next);
    }
    __device__ __forceinline__ void matter(int f, V2 x, V2 a) {
        V2 wn;
        const V2 v = kick(f, a, &wn);
        // compensated drift (hi, lo) += dt*w_{n+1}
        const V2 y = fma2(dt, wn, fma2(dt_lo, wn, bf16x2_to_v2(m.lo[f])));
        V2 xn, e;
        two_sum2(x, y, &xn, &e);
        *reinterpret_cast<uint32_t *>(io.loout + f * c.N3 + site) = v2_to_bf16x2(e);
        store(f, xn, v, wn);
        m.lo[f] = ld_early_u32(io.loin + f * c.N3 + site + next);
    }
    __device__ __forceinline__ void link(int d, V2 th0, V2 th0_lo, V2 K) {
        const V2 gad((float)c.gad), gad_lo((float)(c.gad - (double)(float)c.gad));
        V2 Eh;
        const V2 E = kick(FTH + d, K, &Eh);
        const V2 y = fma2(gad, Eh, fma2(gad_lo, Eh, th0_lo));
        V2 th, lnew;
        two_sum2(th0, y, &th, &lnew);
        link_wrap_c(&th.v.x, &lnew.v.x);
        link_wrap_c(&th.v.y, &lnew.v.y);
        st_cs2(io.tloout + d * c.N3 + site, lnew);
        store(FTH + d, th, E, Eh);
    }
};

// angle of the plaquette of plane (a, b) = (q, q+1 mod 3) at row / column
// offset (dj, dk): the sum of hi differences plus the sum of lo differences
// (compute_forces_complex_gauge pass B, scp_sim.c:1090-1109)
template <class LY>
__device__ __forceinline__ V2 plaq_pair(const PairView<LY> &c, const PairView<LY> &p, int q, int dj, int dk) {
    const int a = q, b = (q + 1) % 3, lo = LY::NF;
    auto at = [&](int f, int dir) { return dir == 0 ? p.get(f, dj, dk) : c.get(f, dj + (dir == 1), dk + (dir == 2)); };
    const V2 hi = (c.get(FTH + a, dj, dk) - at(FTH + a, b)) + (at(FTH + b, a) - c.get(FTH + b, dj, dk));
    const V2 l = (c.get(lo + a, dj, dk) - at(lo + a, b)) + (at(lo + b, a) - c.get(lo + b, dj, dk));
    return hi + l;
}

// What the pair carries from plane i-1: conj(U_0) F of every field (gauged) or
// x(i-1), and the (0,1), (2,0) plaquette sines.
struct PairCarry {
    V2 t[12];
    V2 p0, p2;
};

// The gauged force of one pair, field by field in gauged_site's order (Phi,
// then Theta, each Theta field finished at once).  The Laplacian sums and the
// current's own part take (transported - centre) differences, which removes
// the cancellation an FP32 stencil suffers against O(|f|) values.
//
// Rounding.  Every sum is formed from the same rounded terms in the same order
// as compute_forces_complex_gauge visits them direction by direction (Phi_0,
// Theta_0, Phi_1, ... in the current; T12 and T21 of the cross term as two sums
// of two products): the link angles are two time integrals of these roundings,
// so a run keeps its bits under another order of the work.
template <class LY, class Out>
__device__ __forceinline__ void gauged_pair(const PairView<LY> &c, const PairView<LY> &p, PairCarry &cy,
                                            const StepConsts &k, Out &out) {
    V2 ang[5] = {c.get(FTH, 0, 0), c.get(FTH + 1, 0, 0), c.get(FTH + 2, 0, 0), c.get(FTH + 1, -1, 0),
                 c.get(FTH + 2, 0, -1)};
    V2 sn[5], cs[5], ns[5];
    sincos2_batch(ang, sn, cs);
#pragma unroll
    for (int i = 0; i < 5; i++) ns[i] = -sn[i];
    const V2 idx1((float)k.idx1), idx2((float)k.idx2), eta((float)k.eta);
    V2 jphi[3][3], Jg[3];                 // Phi_a's current terms [d][a], waiting for their place in the sum
    V2 T12[3], T21[3];
    V2 crP[3], ciP[3], crT[3], ciT[3], lapU[3], lapV[3];
    auto field = [&](int q, V2 *cr, V2 *ci, V2 &lu, V2 &lv) {
        const int fre = field_re(q), fim = field_im(q), a = q % 3;
        const V2 u = c.get(fre, 0, 0), v = c.get(fim, 0, 0);
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const V2 up = d == 0 ? p.get(fre, 0, 0) : c.get(fre, d == 1, d == 2);
            const V2 vp = d == 0 ? p.get(fim, 0, 0) : c.get(fim, d == 1, d == 2);
            const V2 fr = fma2(cs[d], up, ns[d] * vp), fi = fma2(cs[d], vp, sn[d] * up);
            V2 br, bi;
            if (d == 0) {
                br = cy.t[fre];
                bi = cy.t[fim];
                cy.t[fre] = fma2(cs[0], u, sn[0] * v);
                cy.t[fim] = fma2(cs[0], v, ns[0] * u);
            } else {
                const V2 um = c.get(fre, -(d == 1), -(d == 2)), vm = c.get(fim, -(d == 1), -(d == 2));
                br = fma2(cs[2 + d], um, sn[2 + d] * vm);
                bi = fma2(cs[2 + d], vm, ns[2 + d] * um);
            }
            const V2 du = fr - u, dv = fi - v;
            const V2 su = du + (br - u), sv = dv + (bi - v);
            if (d == 0) { lu = su; lv = sv; }
            else { lu = lu + su; lv = lv + sv; }
            // lattice current (scp_sim.c:1232-1249): u*TI - v*TR written as
            // u*(TI - v) - v*(TR - u), differences of neighbouring values
            const V2 j = u * dv - v * du;
            if (q < 3) jphi[d][a] = j;
            else if (a == 0) Jg[d] = jphi[d][0] + j;
            else Jg[d] = (Jg[d] + jphi[d][a]) + j;
            if (a == d) continue;
            // cross terms: Phi_a with Theta_b own, Theta_a(x+d) with Phi_b
            // transported back, b the third index; T12 has (Theta, Phi) =
            // (d+1, d+2), T21 the reverse
            const int b = 3 - d - a;
            V2 x;
            if (q < 3) {
                x = c.get(FTU + b, 0, 0) * fi - c.get(FTV + b, 0, 0) * fr;
            } else {
                const V2 pu = c.get(FU + b, 0, 0), pv = c.get(FV + b, 0, 0);
                const V2 wr = d == 0 ? cy.t[FU + b] : fma2(cs[d], pu, sn[d] * pv);
                const V2 wi = d == 0 ? cy.t[FV + b] : fma2(cs[d], pv, ns[d] * pu);
                x = up * wi - vp * wr;
            }
            V2 *T = ((q < 3) == (a == (d + 2) % 3)) ? T12 : T21;
            T[d] = q < 3 ? x : T[d] + x;
            // central covariant differences enter the curls: component t gets
            // +D[d = t+1][field t+2] - D[d = t+2][field t+1] (indices mod 3)
            const V2 dr = (fr - br) * idx1, di = (fi - bi) * idx1;
            const bool plus = (a == (d + 1) % 3);
            const int t = plus ? (d + 2) % 3 : (d + 1) % 3;
            const int other = plus ? (t + 1) % 3 : (t + 2) % 3;   // field of the other term
            if (a < other) { cr[t] = dr; ci[t] = di; }
            else if (plus) { cr[t] = dr - cr[t]; ci[t] = di - ci[t]; }
            else { cr[t] = cr[t] - dr; ci[t] = ci[t] - di; }
        }
    };
#pragma unroll
    for (int a = 0; a < 3; a++) field(a, crP, ciP, lapU[a], lapV[a]);
    const V2 nmt2(-(float)k.mtheta2), nm2(-(float)k.m2);
#pragma unroll
    for (int a = 0; a < 3; a++) {
        V2 lu, lv;
        field(3 + a, crT, ciT, lu, lv);
        const V2 u = c.get(FTU + a, 0, 0), v = c.get(FTV + a, 0, 0);
        out.matter(FTU + a, u, fma2(eta, crP[a], fma2(nmt2, u, lu * idx2)));
        out.matter(FTV + a, v, fma2(eta, ciP[a], fma2(nmt2, v, lv * idx2)));
    }
    V2 s[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const V2 u = c.get(FU + a, 0, 0), v = c.get(FV + a, 0, 0);
        s[a] = fma2(u, u, v * v);
    }
    const V2 den = fma2(V2((float)k.kappa), s[0] * s[1] * s[2], V2(1.f)), dd = den * den;
    const float hmu = 0.5f * (float)k.mu;
    const V2 Vp2(2.f * (hmu / dd.v.x), 2.f * (hmu / dd.v.y));     // 2 V'
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const V2 vr = Vp2 * (a == 0 ? s[1] * s[2] : a == 1 ? s[0] * s[2] : s[0] * s[1]);
        const V2 u = c.get(FU + a, 0, 0), v = c.get(FV + a, 0, 0);
        out.matter(FU + a, u, fma2(eta, crT[a], fma2(nm2, u, lapU[a] * idx2) - vr * u));
        out.matter(FV + a, v, fma2(eta, ciT[a], fma2(nm2, v, lapV[a] * idx2) - vr * v));
    }
    // staples (scp_sim.c:1214-1220)
    V2 pa[7] = {plaq_pair(c, p, 0, 0, 0), plaq_pair(c, p, 1, 0, 0), plaq_pair(c, p, 2, 0, 0), plaq_pair(c, p, 0, -1, 0),
                plaq_pair(c, p, 1, -1, 0), plaq_pair(c, p, 1, 0, -1), plaq_pair(c, p, 2, 0, -1)};
    sin2_batch(pa);
    const V2 st[3] = {(pa[0] - pa[3]) - (pa[2] - pa[6]), (pa[1] - pa[5]) - (pa[0] - cy.p0),
                      (pa[2] - cy.p2) - (pa[1] - pa[4])};
    cy.p0 = pa[0];
    cy.p2 = pa[2];
    const V2 stp((float)k.stp), gg((float)k.g);
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const V2 K = fma2(V2((float)k.inva), Jg[d], V2(-0.5f * (float)k.eta) * (T12[d] - T21[d]));   // Jlat
        out.link(d, c.get(FTH + d, 0, 0), c.get(LY::NF + d, 0, 0), fma2(stp, st[d], gg * K));
    }
}

// compute_forces_complex (scp_sim.c:931-994) of one pair, field by field;
// cy.t: x(i-1), left holding x(i)
template <class LY, class Out>
__device__ __forceinline__ void free_pair(const PairView<LY> &c, const PairView<LY> &p, PairCarry &cy,
                                          const StepConsts &k, Out &out) {
    const V2 idx2((float)k.idx2), ei((float)k.ei), nmt2(-(float)k.mtheta2), nm2(-(float)k.m2);
    V2 crP[6], crT[6], lap[6];
    // Laplacian of neighbour differences (no cancellation against 6*centre)
    // and the central differences into the curl (part 0: real, 3: imaginary)
    auto field = [&](int f, int a, int part, V2 *cr) -> V2 {
        const V2 x = c.get(f, 0, 0);
        const V2 n[3] = {p.get(f, 0, 0), c.get(f, 1, 0), c.get(f, 0, 1)};
        const V2 m[3] = {cy.t[f], c.get(f, -1, 0), c.get(f, 0, -1)};
        V2 l(0.f);
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const V2 up = n[d] - x, dn = m[d] - x;
            l = d == 0 ? up + dn : (l + up) + dn;
            if (a != d) {
                const V2 df = n[d] - m[d];
                const bool plus = (a == (d + 1) % 3);
                const int s = plus ? (d + 2) % 3 : (d + 1) % 3;
                const int other = plus ? (s + 1) % 3 : (s + 2) % 3;
                if (a < other) cr[part + s] = plus ? df : -df;
                else cr[part + s] = plus ? cr[part + s] + df : cr[part + s] - df;
            }
        }
        cy.t[f] = x;
        return l;
    };
#pragma unroll
    for (int a = 0; a < 3; a++) {
        lap[a] = field(FU + a, a, 0, crP);
        lap[3 + a] = field(FV + a, a, 3, crP);
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const V2 lu = field(FTU + a, a, 0, crT), lv = field(FTV + a, a, 3, crT);
        const V2 u = cy.t[FTU + a], v = cy.t[FTV + a];
        out.matter(FTU + a, u, fma2(ei, crP[a], fma2(nmt2, u, lu * idx2)));
        out.matter(FTV + a, v, fma2(ei, crP[3 + a], fma2(nmt2, v, lv * idx2)));
    }
    V2 s[3];
#pragma unroll
    for (int a = 0; a < 3; a++) s[a] = fma2(cy.t[FU + a], cy.t[FU + a], cy.t[FV + a] * cy.t[FV + a]);
    const V2 den = fma2(V2((float)k.kappa), s[0] * s[1] * s[2], V2(1.f)), dd = den * den;
    const float nmu = -(float)k.mu;
    const V2 nV2(nmu / dd.v.x, nmu / dd.v.y);   // -2 V'
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const V2 t = nV2 * (s[(a + 1) % 3] * s[(a + 2) % 3]);
        const V2 u = cy.t[FU + a], v = cy.t[FV + a];
        out.matter(FU + a, u, fma2(ei, crT[a], fma2(t, u, fma2(nm2, u, lap[a] * idx2))));
        out.matter(FV + a, v, fma2(ei, crT[3 + a], fma2(t, v, fma2(nm2, v, lap[3 + a] * idx2))));
    }
}

template <int TX, int TY, bool GAUGED, bool FIRST>
__device__ __forceinline__ void step_item2(const StepIO<F32C> &io, const StepConsts &c, const TileGrid &tg,
                                           const Piece &pc, const bool SYNC, const bool DAMP, unsigned char *smem_raw) {
    using LY = Step2Layout<TX, TY, GAUGED>;
    constexpr int NF = LY::NF, NR = LY::NR, FS = LY::FS, NT = LY::NT;
    float *xs = reinterpret_cast<float *>(smem_raw);
    const int N = c.N;
    const long long N3 = c.N3;
    const int tid = threadIdx.x, hx = tg.tw / 2, pitch = tg.tw + 4;
    const int ty = tid / hx, tx2 = tid - ty * hx;

    const int k0 = pc.kt * tg.tw, j0 = pc.jt * tg.th;
    const int i0 = pc.i0, i1 = pc.i1;
    const int k = k0 + 2 * tx2, j = j0 + ty;
    const int nk = min(k0 + tg.tw, N) - k0, nj = min(j0 + tg.th, N) - j0;   // nk is even
    const bool act = (2 * tx2 < nk) && (ty < nj);
    const int oc = j * N + k;
    const int jlo = wrapi(j0 - 1, N), jhi = wrapi(j0 + nj, N);
    const int klo = wrapi(k0 - 1, N), khi = wrapi(k0 + nk, N);
    const int hk = nk / 2;
    const int c_s = (ty + 1) * pitch + 2 + 2 * tx2;                    // the pair in a slot

    // halo copies of this thread.  kind 1: a pair of the j-1 / j+1 rows (all
    // ring fields); 2: one site of the k-1 / k+1 columns; 3: a corner site
    // (link angles only, for the plaquettes of the neighbour rows)
    int h_s[LY::HPT], h_g[LY::HPT], h_kind[LY::HPT];
#pragma unroll
    for (int q = 0; q < LY::HPT; q++) {
        const int h = tid + q * NT;
        int r = 0, col = 0, gj = 0, gk = 0, kind = 0;
        if (h < hk) { r = 0; col = 2 + 2 * h; gj = jlo; gk = k0 + 2 * h; kind = 1; }
        else if (h < 2 * hk) { r = nj + 1; col = 2 + 2 * (h - hk); gj = jhi; gk = k0 + 2 * (h - hk); kind = 1; }
        else if (h < 2 * hk + nj) { r = h - 2 * hk + 1; col = 1; gj = j0 + h - 2 * hk; gk = klo; kind = 2; }
        else if (h < 2 * hk + 2 * nj) { r = h - 2 * hk - nj + 1; col = nk + 2; gj = j0 + h - 2 * hk - nj; gk = khi; kind = 2; }
        else if (GAUGED && h == 2 * hk + 2 * nj) { r = nj + 1; col = 1; gj = jhi; gk = klo; kind = 3; }
        else if (GAUGED && h == 2 * hk + 2 * nj + 1) { r = 0; col = nk + 2; gj = jlo; gk = khi; kind = 3; }
        h_s[q] = r * pitch + col;
        h_g[q] = gj * N + gk;
        h_kind[q] = kind;
    }

    auto issue_plane = [&](int p, int slot) {
        const long long pb = (long long)wrapi(p, N) * N * N;
        float *sbase = xs + slot * LY::PLANE;
        // ring field f: the positions, then the links' low parts
        auto src = [&](int f) { return (f < NF ? io.xin + f * N3 : io.tloin + (f - NF) * N3) + pb; };
        if (act) {
#pragma unroll
            for (int f = 0; f < NR; f++) cp_async8(sbase + f * FS + c_s, src(f) + oc);
        }
#pragma unroll
        for (int q = 0; q < LY::HPT; q++) {
            const int kind = h_kind[q];
            if (kind == 1) {
#pragma unroll
                for (int f = 0; f < NR; f++) cp_async8(sbase + f * FS + h_s[q], src(f) + h_g[q]);
            } else if (kind != 0) {
                const int f0 = (kind == 2) ? 0 : FTH;
#pragma unroll
                for (int f = 0; f < NR; f++)
                    if (f >= f0) cp_async4(sbase + f * FS + h_s[q], src(f) + h_g[q]);
            }
        }
        cp_async_commit();
    };
    auto view = [&](int slot) { return PairView<LY>{xs + slot * LY::PLANE + c_s, pitch}; };

    __syncthreads();   // previous item finished reading the ring
    issue_plane(i0 - 1, 0);
    issue_plane(i0, 1);
    issue_plane(i0 + 1, 2);
    PairAhead<GAUGED> m;
    if (act) {
        const long long site = (long long)i0 * N * N + oc;
#pragma unroll
        for (int f = 0; f < NF; f++) m.w[f] = ld_early2(io.win + f * N3 + site);
#pragma unroll
        for (int f = 0; f < 12; f++) m.lo[f] = ld_early_u32(io.loin + f * N3 + site);
    }
    cp_async_wait<1>();
    __syncthreads();
    PairCarry cy;
    if (act) {
        const PairView<LY> vm = view(0), vc = view(1);
        if constexpr (GAUGED) {
            V2 a0[1] = {vm.get(FTH, 0, 0)}, sn[1], cs[1];
            sincos2_batch(a0, sn, cs);
            const V2 ns = -sn[0];
#pragma unroll
            for (int q = 0; q < 6; q++) {
                const V2 u = vm.get(field_re(q), 0, 0), v = vm.get(field_im(q), 0, 0);
                cy.t[field_re(q)] = fma2(cs[0], u, sn[0] * v);
                cy.t[field_im(q)] = fma2(cs[0], v, ns * u);
            }
            V2 pa[2] = {plaq_pair(vm, vc, 0, 0, 0), plaq_pair(vm, vc, 2, 0, 0)};
            sin2_batch(pa);
            cy.p0 = pa[0];
            cy.p2 = pa[1];
        } else {
#pragma unroll
            for (int f = 0; f < 12; f++) cy.t[f] = vm.get(f, 0, 0);
        }
    }

    for (int i = i0; i < i1; i++) {
        const int sc = (i - i0 + 1) % 3, sp = (i - i0 + 2) % 3, sn = (i - i0) % 3;
        cp_async_wait<0>();
        __syncthreads();
        if (i + 2 <= i1) issue_plane(i + 2, sn);
        if (!act) continue;
        const long long site = (long long)i * N * N + oc;
        PairUpdate<GAUGED, FIRST> out{io, c, m, site, i + 1 < i1 ? (long long)N * N : 0, SYNC, DAMP,
                                      V2((float)c.dt), V2((float)c.hdt), V2((float)(c.dt - (double)(float)c.dt)),
                                      V2((float)(c.hdt - (double)(float)c.hdt)), V2(1.f)};
        if (DAMP && !FIRST)
            out.dmp = V2((float)sponge_factor(i, j, k, c.L, c.dx, c.damp_width, c.damp_rate),
                         (float)sponge_factor(i, j, k + 1, c.L, c.dx, c.damp_width, c.damp_rate));
        if constexpr (GAUGED) gauged_pair<LY>(view(sc), view(sp), cy, c, out);
        else free_pair<LY>(view(sc), view(sp), cy, c, out);
        if (SYNC && out.bad) atomicOr(io.flag, 1);
    }
}

template <int TX, int TY, bool GAUGED, bool FIRST, bool SYNC, bool DAMP>
__global__ void __launch_bounds__(Step2Layout<TX, TY, GAUGED>::NT, Step2Layout<TX, TY, GAUGED>::MIN_BLOCKS)
step2_kernel(StepIO<F32C> io, StepConsts c, TileGrid tg) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    griddep_wait();
    griddep_launch();
    for_each_piece(tg, c.N, [&](const Piece &pc) { step_item2<TX, TY, GAUGED, FIRST>(io, c, tg, pc, SYNC, DAMP, smem_raw); });
}

// many FP32C requests of even N per launch (table semantics as step_multi_kernel)
template <int TX, int TY, bool GAUGED, bool DAMP>
__global__ void __launch_bounds__(Step2Layout<TX, TY, GAUGED>::NT, Step2Layout<TX, TY, GAUGED>::MIN_BLOCKS)
step2_multi_kernel(const ReqTable<F32C> *tab, int k) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int nitems = tab->nitems, nreq = tab->nreq;
    const long long s = tab->step + k;
    for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
        const ReqSlot<F32C> &q = tab->r[req_of_item(tab, nreq, item)];
        if (s < q.s0 || s >= q.s1) continue;       // uniform over the CTA
        const StepIO<F32C> io = q.io[(int)((s - q.s0) & 1)];
        const StepConsts c = q.c;
        const TileGrid tg = q.tg;
        step_item2<TX, TY, GAUGED, false>(io, c, tg, piece_of_item(tg, item - q.item0, c.N), false, DAMP, smem_raw);
    }
}

}  // namespace scp
