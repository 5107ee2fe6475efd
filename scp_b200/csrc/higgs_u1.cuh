// higgs_u1.cuh -- the gauged stepper with the Higgs condensate and/or the
// second compact U(1) (the reference's v71 extensions of the gauged force,
// sfa/sim/scp_sim.c:1053-1263; its energy :1970-1975; the second Gauss
// projection :2400-2458), as one fused kernel per time step.
//
// Physics.  The Higgs field H is a real scalar with
//     V_H = (lambda/4)(H^2 - v^2)^2 + (kappa_H/2) s H^2,   s = prod_a |Phi_a|^2,
// so it pushes the matter with -kappa_H H^2 Phi_a prod_{b!=a} |Phi_b|^2 and
// feels lap H - lambda H (H^2 - v^2) - kappa_H s H.  The second gauge has its
// own links th2, field E2, coupling g2, and per-component charges q_a: the
// matter component a is transported by the phase th_d + q_a th2_d, the E2
// kick is its plaquette term plus g2 sum_a q_a Im[f_a^* T+_a] / dx, and the
// E kick keeps the first gauge's plaquette term and current (whose cross term
// pairs the Theta and Phi components through the first gauge's link alone).
// The sponge damps the matter momenta and E, not E2 or dH/dt.
//
// Layout.  Position buffers (two, alternating) and momentum buffers hold, as
// N^3 arrays: the 12 matter fields and th (the 15-field order of the fused
// step, so diagnostics and snapshots read them the same way), then th2 (3)
// with the second gauge, then H with the Higgs field; the momenta follow the
// same order (matter, E, [E2], [dH/dt]).  One launch per step reads every
// position of the resident planes through the ring, so each word moves once
// per step.
//
// What bounds it: latency at eight warps per SM.  608 B per site; with both
// extensions a warp issues some 2000 instructions per plane (two sets of link
// phases, two gauges' staples), 0.65 of a plain copy's rate at 128^3: 303 us a
// step against 614 with four resident planes, a sine and cosine of every
// plaquette and the momenta loaded at their own plane.
#pragma once
#include "walk.cuh"

namespace scp {

struct HuConsts {
    int N;
    long long N3;
    double L, dx, dV, idx1, idx2, inva, hdt, dt;
    double mu, kappa, m2, mtheta2, eta;
    double g, stp, gad;               // first gauge: coupling, 1/(g dx^3), -g dx dt
    double g2, stp2, gad2, q[3];      // second gauge
    double hv, hlam, hkap;            // Higgs
    double damp_width, damp_rate;
    double ei, cross, gi;             // eta/(2dx), eta dx/2, g/dx
};

constexpr int kTh2Slot = 15;   // second gauge links, after matter and th

template <class MODE, bool HIGGS, bool G2>
struct HiggsU1 {
    static constexpr int TH = 12;                        // first gauge links
    static constexpr int TH2 = kTh2Slot;                      // second gauge links
    static constexpr int HF = G2 ? 18 : 15;              // the Higgs field
    static constexpr int NR = 15 + (G2 ? 3 : 0) + (HIGGS ? 1 : 0), CF = 12;
    static constexpr int MIN_CTAS = 1;
    static constexpr bool HALO_APART = false, CONVERT = false, WIDE = true;

    struct Args {
        const double *x;        // positions x_{n+1}, NR arrays
        int N;
        HuConsts c;
        LeapIO io;
    };

    static constexpr int NR_FEW = NR;   // always all of them
    __device__ static __forceinline__ bool few(const Args &) { return false; }
    __device__ static __forceinline__ const double *src(const Args &A, int f, long long n3) { return A.x + f * n3; }

    struct State {
        GaugedCarry cy;
        double p0, p2;          // plaquette sines of the second gauge at x - i
        double hm;              // H at x - i
        double w[NR];
    };

    __device__ static __forceinline__ void load(const Args &A, State &st, long long idx) {
#pragma unroll
        for (int f = 0; f < NR; f++) st.w[f] = ld_early(LeapSite<MODE, NR>::at(A.io.win, f, A.c.N3) + idx);
    }

    template <class V>
    __device__ static __forceinline__ void begin(const Args &A, State &st, const V &m, const V &c) {
        if constexpr (G2) {   // a phase per component: th + q_a th2
#pragma unroll
            for (int a = 0; a < 3; a++) {
                double ph[1] = {rfma(A.c.q[a], m.get(TH2, 0, 0), m.get(TH, 0, 0))}, sn[1], cs[1];
                sincos_batch<1, true>(ph, sn, cs);
#pragma unroll
                for (int q = a; q < 6; q += 3) {
                    const double u = m.get(field_re(q), 0, 0), v = m.get(field_im(q), 0, 0);
                    st.cy.t[field_re(q)] = rfma(sn[0], v, rmul(cs[0], u));
                    st.cy.t[field_im(q)] = rfma(-sn[0], u, rmul(cs[0], v));
                }
            }
            staples_begin(m, c, TH, st.cy.p0, st.cy.p2);
            staples_begin(m, c, TH2, st.p0, st.p2);
        } else {
            gauged_begin<false, true>(m, c, TH, st.cy);
        }
        if (HIGGS) st.hm = m.get(HF, 0, 0);
    }

    struct Out {
        const Args &A;
        LeapSite<MODE, NR> &leap;
        double s;               // prod_a |Phi_a|^2
        __device__ __forceinline__ void theta(int a, double u, double v, double au, double av) {
            leap.put(FTU + a, u, au, leap.dmp);
            leap.put(FTV + a, v, av, leap.dmp);
        }
        __device__ __forceinline__ void phi(int a, double u, double v, double au, double av) {
            leap.put(FU + a, u, au, leap.dmp);
            leap.put(FV + a, v, av, leap.dmp);
        }
        __device__ __forceinline__ void moduli(const double (&m)[3], double) { s = rmul(rmul(m[0], m[1]), m[2]); }
        __device__ __forceinline__ void angles(double, double, double) {}
        __device__ __forceinline__ double current(int, double K) { return K; }
        __device__ __forceinline__ void link(int d, double th, double K) {
            leap.put_link(TH + d, th, K, A.c.gad, leap.dmp);
        }
    };

    // The force with the second gauge: the components have phases of their
    // own, so a component's Phi and Theta go through their directions together
    // (one set of phases live at a time, shared by components of equal charge)
    // and every kick waits for the last of them.
    template <class V>
    __device__ static __forceinline__ void two_gauge_site(const Args &A, State &st, const V &c, const V &p, Out &out,
                                                          double nhh) {
        const HuConsts &h = A.c;
        const GaugedConsts k(h);
        double wang[3] = {c.get(TH, 0, 0), c.get(TH + 1, 0, 0), c.get(TH + 2, 0, 0)}, sw[3], cw[3];
        sincos_batch(wang, sw, cw);
        double K[3] = {0.0, 0.0, 0.0}, Kw[3] = {0.0, 0.0, 0.0};
        double crP[3], ciP[3], crT[3], ciT[3], lap[12], none = 0.0;
        double sn[5], cs[5];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            if (a == 0 || h.q[a] != h.q[a - 1]) {
                double ang[5];
#pragma unroll
                for (int n = 0; n < 5; n++) {
                    const int d = n < 3 ? n : n - 2, dj = n == 3 ? -1 : 0, dk = n == 4 ? -1 : 0;
                    ang[n] = rfma(h.q[a], c.get(TH2 + d, dj, dk), c.get(TH + d, dj, dk));
                }
                sincos_batch<5, true>(ang, sn, cs);
            }
            const TwoGauge g2{cw, sw, h.q[a], Kw};
            transport_field<false, true>(c, p, a, cs, sn, st.cy.t, K, k.r, crP, ciP, lap[FU + a], lap[FV + a], none, g2);
            transport_field<false, true>(c, p, 3 + a, cs, sn, st.cy.t, K, k.r, crT, ciT, lap[FTU + a], lap[FTV + a],
                                         none, g2);
        }
        double s[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const double u = c.again(FU + a), v = c.again(FV + a);
            s[a] = rfma(u, u, rmul(v, v));
        }
        const double den = rfma(k.kappa, rmul(rmul(s[0], s[1]), s[2]), 1.0);
        const double nV2 = radd(-k.mu / rmul(den, den), nhh);
        out.moduli(s, den);
        auto acc = [&](double x, double l, double t, double cu) {
            return rfma(k.ei, cu, rfma(rfma(-6.0, x, l), k.idx2, rmul(t, x)));
        };
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const double t = rfma(nV2, rmul(s[(a + 1) % 3], s[(a + 2) % 3]), k.nm2);
            const double u = c.again(FU + a), v = c.again(FV + a);
            out.phi(a, u, v, acc(u, lap[FU + a], t, crT[a]), acc(v, lap[FV + a], t, ciT[a]));
            const double tu = c.again(FTU + a), tv = c.again(FTV + a);
            out.theta(a, tu, tv, acc(tu, lap[FTU + a], k.nmt2, crP[a]), acc(tv, lap[FTV + a], k.nmt2, ciP[a]));
        }
        double stp[3], own[3];
        staples(c, p, TH, st.cy.p0, st.cy.p2, stp, own);
#pragma unroll
        for (int d = 0; d < 3; d++) out.link(d, c.again(TH + d), rfma(k.stp, stp[d], rmul(k.gi, K[d])));
        staples(c, p, TH2, st.p0, st.p2, stp, own);
        const double g2i = rmul(h.g2, h.inva);
#pragma unroll
        for (int d = 0; d < 3; d++)   // E2 is not damped by the sponge
            out.leap.put_link(TH2 + d, c.again(TH2 + d), rfma(h.stp2, stp[d], rmul(g2i, Kw[d])), h.gad2, 1.0);
    }

    template <class V>
    __device__ static __forceinline__ void site(const Args &A, State &st, const V &c, const V &p, int i, int j, int k,
                                                long long idx, long long next) {
        const HuConsts &h = A.c;
        const double dmp = (MODE::DAMP && !MODE::FIRST)
                               ? sponge_factor(i, j, k, h.L, h.dx, h.damp_width, h.damp_rate) : 1.0;
        LeapSite<MODE, NR> leap{A.io, st.w, h.N3, idx, next, h.hdt, h.dt, dmp};
        Out out{A, leap, 0.0};
        const double H = HIGGS ? c.get(HF, 0, 0) : 0.0;
        const double nhh = HIGGS ? rmul(-h.hkap, rmul(H, H)) : 0.0;
        if constexpr (G2) {
            two_gauge_site(A, st, c, p, out, nhh);
        } else {
            GaugedSums none;
            gauged_site<false, false, true>(c, p, TH, st.cy, GaugedConsts(h), out, none, 1.0, nhh);
        }
        if (HIGGS) {   // lap H - lambda H (H^2 - v^2) - kappa_H s H, not damped
            double l = radd(p.get(HF, 0, 0), st.hm);
            l = radd(radd(l, c.get(HF, 1, 0)), c.get(HF, -1, 0));
            l = radd(radd(l, c.get(HF, 0, 1)), c.get(HF, 0, -1));
            st.hm = H;
            const double v2 = rfma(H, H, rmul(-h.hv, h.hv));
            const double t = rfma(-h.hlam, v2, rmul(-h.hkap, out.s));
            leap.put(HF, H, rfma(rfma(-6.0, H, l), h.idx2, rmul(t, H)), 1.0);
        }
        if (MODE::SYNC && leap.bad) atomicOr(A.io.flag, 1);
    }
};

}  // namespace scp
