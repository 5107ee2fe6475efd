// gauged.cuh -- the gauged FP64 force at one site, in explicitly rounded
// operations, visited field by field.
//
// What a site needs (compute_forces_complex_gauge, sfa/sim/scp_sim.c:1053-1263):
// every complex field F_q (Phi_a: q = a, Theta_a: q = 3 + a) is parallel-
// transported along both links of each direction,
//     T+_d = U_d(x) F(x + d),   T-_d = conj(U_d(x - d)) F(x - d),
// and the transports feed its covariant Laplacian, the curl of its triplet
// (differences T+ - T-) and the lattice current
//     J_d = sum_q Im[F_q^* T+_d F_q] / dx - (eta/2) (T12 - T21),
// whose cross terms pair Theta_{d+1} with Phi_{d+2} and Theta_{d+2} with
// Phi_{d+1}: Im[Theta_e^* T+ Phi_f] - Im[Phi_f^* T+ Theta_e].
//
// Order of the work.  The three Phi fields come first, then the three Theta
// fields, each taken through all its directions before the next: what stays
// live is the running curls, the currents and one field's sums, about 100
// registers less than holding every field's sums direction by direction.  A
// Theta field is finished (kicked, drifted, stored) as soon as its directions
// are done, since the curl of Phi is complete by then.  The cross terms ride
// on the transports as they appear: J_d gains Im[(F_q + r G)^* T+] with G the
// partner's own value and r = -+ eta dx / 2, so no transport is kept or formed
// twice.  The backward transport along i is formed at the plane before, from
// that plane's own site, and carried (T-_0: 12 values) in place of the field.
//
// Rounding.  Every operation that reaches the state is an explicit
// multiply, add or fused multiply-add: the compiler has no freedom to fuse
// them differently, so every kernel built on this function (stagings, tile
// shapes, with or without the diagnostics sums, which reuse the transports'
// differences) advances the state with the same bits.
#pragma once
#include "common.cuh"
#include "trig.cuh"

namespace scp {

__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double radd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double rsub(double a, double b) { return __dadd_rn(a, -b); }
__device__ __forceinline__ double rfma(double a, double b, double c) { return __fma_rn(a, b, c); }

// sponge factor 1 - rate * s^2 of the absorbing boundary at site (i, j, k),
// 1 inside radius L - width (apply_damping, sfa/sim/scp_sim.c:1440-1473)
__device__ __forceinline__ double sponge_factor(int i, int j, int k, double L, double dx, double width, double rate) {
    const double x = rfma(i, dx, -L), y = rfma(j, dx, -L), z = rfma(k, dx, -L);
    const double r = sqrt(rfma(z, z, rfma(y, y, rmul(x, x))));
    const double inner = rsub(L, width);
    if (!(r > inner)) return 1.0;
    const double s = fmin(rsub(r, inner) / width, 1.0);
    return rfma(rmul(-rate, s), s, 1.0);
}

// Constants derived from StepConsts that only the site function uses.
struct GaugedConsts {
    double idx2, ei, nm2, nmt2, kappa, mu, r, gi, stp;
    template <class C>
    __device__ __forceinline__ explicit GaugedConsts(const C &c)
        : idx2(c.idx2), ei(c.ei), nm2(-c.m2), nmt2(-c.mtheta2), kappa(c.kappa), mu(c.mu), r(c.cross), gi(c.gi),
          stp(c.stp) {}
};

// What a thread carries from plane i-1 to plane i at its site.
struct GaugedCarry {
    double t[12];      // conj(U_0) F of every field at x - i (slots u, v, tu, tv)
    double p0, p2;     // plaquette sines (0,1) and (2,0) at x - i
};

// Per-site sums that the diagnostics take from the transports.
struct GaugedSums {
    double eg, etg;    // sum of squared differences (T+ - T-) of Phi and of Theta
    double ec;         // Phi . curl Theta, differences undivided
};

// angle of the plaquette of plane (a, b) = (q, q+1 mod 3) at the site offset
// (dj, dk) of view c (next plane: p): th_a(y) + th_b(y+a) - th_a(y+b) - th_b(y)
template <class V>
__device__ __forceinline__ double plaq_angle(const V &c, const V &p, int fth, int q, int dj, int dk) {
    const int a = q, b = (q + 1) % 3;
    const double tay = c.get(fth + a, dj, dk), tby = c.get(fth + b, dj, dk);
    const double tb_ya = (a == 0) ? p.get(fth + b, dj, dk) : c.get(fth + b, dj + (a == 1), dk + (a == 2));
    const double ta_yb = (b == 0) ? p.get(fth + a, dj, dk) : c.get(fth + a, dj + (b == 1), dk + (b == 2));
    return rsub(rsub(radd(tay, tb_ya), ta_yb), tby);
}

// field slot of Phi_a / Theta_a's real part; the imaginary part is 3 further
__device__ __forceinline__ constexpr int field_re(int q) { return q < 3 ? FU + q : FTU + q - 3; }
__device__ __forceinline__ constexpr int field_im(int q) { return q < 3 ? FV + q : FTV + q - 3; }

// plaquette sines (0,1) and (2,0) of the plane viewed by m (next: c)
template <class V>
__device__ __forceinline__ void staples_begin(const V &m, const V &c, int fth, double &p0, double &p2) {
    double pa[2] = {plaq_angle(m, c, fth, 0, 0, 0), plaq_angle(m, c, fth, 2, 0, 0)};
    sin_batch(pa);
    p0 = pa[0];
    p2 = pa[1];
}

// The carry of the plane before the first one of a segment: m views plane
// i0-1, c plane i0.
template <bool CHARGED, bool LINKS, class V>
__device__ __forceinline__ void gauged_begin(const V &m, const V &c, int fth, GaugedCarry &cy, double charge = 1.0) {
    double a0[1] = {m.get(fth, 0, 0)}, sn[1], cs[1];
    if (CHARGED) a0[0] = rmul(charge, a0[0]);
    sincos_batch<1, CHARGED>(a0, sn, cs);
#pragma unroll
    for (int q = 0; q < 6; q++) {
        const double u = m.get(field_re(q), 0, 0), v = m.get(field_im(q), 0, 0);
        cy.t[field_re(q)] = rfma(sn[0], v, rmul(cs[0], u));
        cy.t[field_im(q)] = rfma(-sn[0], u, rmul(cs[0], v));
    }
    if constexpr (LINKS) staples_begin(m, c, fth, cy.p0, cy.p2);
}

// One complex field q through its three directions.  cs, sn: the phases of
// its links at x (0..2), at x - j (3) and at x - k (4); t: the carried
// backward transports along i.  Adds to the currents K (in units of 1/dx,
// cross terms with the factor r = eta dx / 2 included), to the curl of its
// triplet (cr, ci: differences undivided) and, with SUMS, to esum (squared
// differences); returns the Laplacian's sum of transports in lu, lv.
//
// With G2 the components have phases of their own and the cross terms take
// the first gauge's link alone on their Theta(x + d) side (cw, sw); Kw sums
// the current weighted by the component's second charge w.
struct TwoGauge {
    const double *cw, *sw;   // first gauge's link phases at x, per direction
    double w;                // second charge of this component
    double *Kw;
};
template <bool SUMS, bool G2, class V>
__device__ __forceinline__ void transport_field(const V &c, const V &p, const int q, const double *cs,
                                                const double *sn, double *t, double *K, const double rx, double *cr,
                                                double *ci, double &lu, double &lv, double &esum,
                                                const TwoGauge &g2) {
    const int fre = field_re(q), fim = field_im(q), a = q % 3;
    const double u = c.get(fre, 0, 0), v = c.get(fim, 0, 0);
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const double cP = cs[d], sP = sn[d];
        const double up = d == 0 ? p.get(fre, 0, 0) : c.get(fre, d == 1, d == 2);
        const double vp = d == 0 ? p.get(fim, 0, 0) : c.get(fim, d == 1, d == 2);
        const double fr = rfma(-sP, vp, rmul(cP, up)), fi = rfma(sP, up, rmul(cP, vp));
        double br, bi;
        if (d == 0) {
            br = t[fre];
            bi = t[fim];
            t[fre] = rfma(sP, v, rmul(cP, u));
            t[fim] = rfma(-sP, u, rmul(cP, v));
        } else {
            const double cM = cs[2 + d], sM = sn[2 + d];
            const double um = c.get(fre, -(d == 1), -(d == 2)), vm = c.get(fim, -(d == 1), -(d == 2));
            br = rfma(sM, vm, rmul(cM, um));
            bi = rfma(-sM, um, rmul(cM, vm));
        }
        if (d == 0) { lu = radd(fr, br); lv = radd(fi, bi); }
        else { lu = radd(radd(lu, fr), br); lv = radd(radd(lv, fi), bi); }
        // the current; Phi_a meets Theta_b and Theta_a meets Phi_b, b the third
        // index, with sign + where a = d+1
        const int b = 3 - d - a, o = q < 3 ? 3 + b : b;
        const double r = (a == (d + 1) % 3) ? rx : -rx;
        if constexpr (!G2) {
            double gu = u, gv = v;
            if (a != d) {   // the own value plus r times the partner's
                gu = rfma(r, c.again(field_re(o)), u);
                gv = rfma(r, c.again(field_im(o)), v);
            }
            K[d] = rfma(gu, fi, K[d]);
            K[d] = rfma(-gv, fr, K[d]);
        } else {
            const double j = rfma(-v, fr, rmul(u, fi));
            K[d] = radd(K[d], j);
            g2.Kw[d] = rfma(g2.w, j, g2.Kw[d]);
            if (a != d) {
                double xr = fr, xi = fi;
                if (q >= 3) {
                    xr = rfma(-g2.sw[d], vp, rmul(g2.cw[d], up));
                    xi = rfma(g2.sw[d], up, rmul(g2.cw[d], vp));
                }
                const double x = rfma(-c.again(field_im(o)), xr, rmul(c.again(field_re(o)), xi));
                K[d] = rfma(r, x, K[d]);
            }
        }
        // curl_c = D_{c+1} f_{c+2} - D_{c+2} f_{c+1}
        if (a != d || SUMS) {
            const double dr = rsub(fr, br), di = rsub(fi, bi);
            if (SUMS) esum += dr * dr + di * di;
            if (a != d) {
                const bool plus = (a == (d + 1) % 3);
                const int s = plus ? (d + 2) % 3 : (d + 1) % 3;
                const int other = plus ? (s + 1) % 3 : (s + 2) % 3;   // field of the other term
                if (a < other) { cr[s] = plus ? dr : -dr; ci[s] = plus ? di : -di; }
                else if (plus) { cr[s] = radd(cr[s], dr); ci[s] = radd(ci[s], di); }
                else { cr[s] = rsub(cr[s], dr); ci[s] = rsub(ci[s], di); }
            }
        }
    }
}

// Field kick of one gauge's plaquettes (scp_sim.c:1214-1220): staples from
// the sines at x and at x less the other direction of the plane; p0, p2: the
// sines at x - i, replaced by this plane's.  pa receives the site's angles.
template <class V>
__device__ __forceinline__ void staples(const V &c, const V &p, int fth, double &p0, double &p2, double (&st)[3],
                                        double (&own)[3]) {
    double pa[7] = {plaq_angle(c, p, fth, 0, 0, 0), plaq_angle(c, p, fth, 1, 0, 0), plaq_angle(c, p, fth, 2, 0, 0),
                    plaq_angle(c, p, fth, 0, -1, 0), plaq_angle(c, p, fth, 1, -1, 0),
                    plaq_angle(c, p, fth, 1, 0, -1), plaq_angle(c, p, fth, 2, 0, -1)};
    own[0] = pa[0];
    own[1] = pa[1];
    own[2] = pa[2];
    sin_batch(pa);
    st[0] = rsub(rsub(pa[0], pa[3]), rsub(pa[2], pa[6]));
    st[1] = rsub(rsub(pa[1], pa[5]), rsub(pa[0], p0));
    st[2] = rsub(rsub(pa[2], p2), rsub(pa[1], pa[4]));
    p0 = pa[0];
    p2 = pa[2];
}

// The force at one site: c views plane i, p plane i+1, cy carries plane i-1
// and leaves with plane i.  Results go to `out` as they are complete:
//   out.theta(a, u, v, au, av)   Theta_a and its accelerations, once Phi's directions are done
//   out.moduli(s, den)           |Phi_a|^2 and 1 + kappa s
//   out.phi(a, u, v, au, av)     Phi_a and its accelerations
//   out.angles(p0, p1, p2)       the site's own plaquette angles
//   out.link(d, th, K)           link angle d and the kick of E_d
// Variants: the links carry the charge `charge` (CHARGED); LINKS = false
// leaves the plaquettes out and hands the bare currents to out.current(d, K);
// nhh adds nhh prod_{b != a} |Phi_b|^2 Phi_a to Phi's force (the Higgs).
template <bool SUMS, bool CHARGED, bool LINKS, class V, class Out>
__device__ __forceinline__ void gauged_site(const V &c, const V &p, int fth, GaugedCarry &cy, const GaugedConsts &k,
                                            Out &out, GaugedSums &sums, double charge = 1.0, double nhh = 0.0) {
    // link phases at x (U_0, U_1, U_2) and at x - j, x - k
    double ang[5] = {c.get(fth, 0, 0), c.get(fth + 1, 0, 0), c.get(fth + 2, 0, 0), c.get(fth + 1, -1, 0),
                     c.get(fth + 2, 0, -1)};
    double sn[5], cs[5];
    if (CHARGED) {
#pragma unroll
        for (int i = 0; i < 5; i++) ang[i] = rmul(charge, ang[i]);
        sincos_batch<5, true>(ang, sn, cs);
    } else {
        sincos_batch(ang, sn, cs);
    }
    double K[3] = {0.0, 0.0, 0.0};
    double crP[3], ciP[3], crT[3], ciT[3], lapU[3], lapV[3];
    double eg = 0.0, etg = 0.0;
    const TwoGauge none{};
#pragma unroll
    for (int a = 0; a < 3; a++)
        transport_field<SUMS, false>(c, p, a, cs, sn, cy.t, K, k.r, crP, ciP, lapU[a], lapV[a], eg, none);
#pragma unroll
    for (int a = 0; a < 3; a++) {
        double lu, lv;
        transport_field<SUMS, false>(c, p, 3 + a, cs, sn, cy.t, K, k.r, crT, ciT, lu, lv, etg, none);
        const double u = c.again(FTU + a), v = c.again(FTV + a);
        out.theta(a, u, v, rfma(k.ei, crP[a], rfma(rfma(-6.0, u, lu), k.idx2, rmul(k.nmt2, u))),
                  rfma(k.ei, ciP[a], rfma(rfma(-6.0, v, lv), k.idx2, rmul(k.nmt2, v))));
    }
    {   // Phi: potential (scp_sim.c:946-958) and the finished sums
        double u[3], v[3], s[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            u[a] = c.again(FU + a);
            v[a] = c.again(FV + a);
            s[a] = rfma(u[a], u[a], rmul(v[a], v[a]));
        }
        const double den = rfma(k.kappa, rmul(rmul(s[0], s[1]), s[2]), 1.0);
        const double nV2 = radd(-k.mu / rmul(den, den), nhh);   // -2 V' [- kappa_H H^2]
        out.moduli(s, den);
        double ec = 0.0;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const double t = rfma(nV2, rmul(s[(a + 1) % 3], s[(a + 2) % 3]), k.nm2);
            if (SUMS) ec += u[a] * crT[a] + v[a] * ciT[a];
            out.phi(a, u[a], v[a], rfma(k.ei, crT[a], rfma(rfma(-6.0, u[a], lapU[a]), k.idx2, rmul(t, u[a]))),
                    rfma(k.ei, ciT[a], rfma(rfma(-6.0, v[a], lapV[a]), k.idx2, rmul(t, v[a]))));
        }
        if (SUMS) sums.ec = ec;
    }
    if (SUMS) { sums.eg = eg; sums.etg = etg; }
    if constexpr (LINKS) {
        double st[3], own[3];
        staples(c, p, fth, cy.p0, cy.p2, st, own);
        out.angles(own[0], own[1], own[2]);
#pragma unroll
        for (int d = 0; d < 3; d++)
            out.link(d, c.again(fth + d), rfma(k.stp, st[d], CHARGED ? out.current(d, K[d]) : rmul(k.gi, K[d])));
    } else {
#pragma unroll
        for (int d = 0; d < 3; d++) out.current(d, K[d]);
    }
}

}  // namespace scp
