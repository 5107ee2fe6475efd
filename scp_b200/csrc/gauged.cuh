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

// Constants derived from StepConsts that only the site function uses.
struct GaugedConsts {
    double idx2, ei, nm2, nmt2, kappa, mu, r, gi, stp;
    __device__ __forceinline__ explicit GaugedConsts(const StepConsts &c)
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

// The carry of the plane before the first one of a segment: m views plane
// i0-1, c plane i0.
template <class V>
__device__ __forceinline__ void gauged_begin(const V &m, const V &c, int fth, GaugedCarry &cy) {
    double a0[1] = {m.get(fth, 0, 0)}, sn[1], cs[1];
    sincos_batch(a0, sn, cs);
#pragma unroll
    for (int q = 0; q < 6; q++) {
        const double u = m.get(field_re(q), 0, 0), v = m.get(field_im(q), 0, 0);
        cy.t[field_re(q)] = rfma(sn[0], v, rmul(cs[0], u));
        cy.t[field_im(q)] = rfma(-sn[0], u, rmul(cs[0], v));
    }
    double pa[2] = {plaq_angle(m, c, fth, 0, 0, 0), plaq_angle(m, c, fth, 2, 0, 0)};
    sin_batch(pa);
    cy.p0 = pa[0];
    cy.p2 = pa[1];
}

// The force at one site: c views plane i, p plane i+1, cy carries plane i-1
// and leaves with plane i.  Results go to `out` as they are complete:
//   out.theta(a, u, v, au, av)   Theta_a and its accelerations, once Phi's directions are done
//   out.moduli(s, den)           |Phi_a|^2 and 1 + kappa s
//   out.phi(a, u, v, au, av)     Phi_a and its accelerations
//   out.angles(p0, p1, p2)       the site's own plaquette angles
//   out.link(d, th, K)           link angle d and the kick of E_d
template <bool SUMS, class V, class Out>
__device__ __forceinline__ void gauged_site(const V &c, const V &p, int fth, GaugedCarry &cy, const GaugedConsts &k,
                                            Out &out, GaugedSums &sums) {
    // link phases at x (U_0, U_1, U_2) and at x - j, x - k
    double ang[5] = {c.get(fth, 0, 0), c.get(fth + 1, 0, 0), c.get(fth + 2, 0, 0), c.get(fth + 1, -1, 0),
                     c.get(fth + 2, 0, -1)};
    double sn[5], cs[5];
    sincos_batch(ang, sn, cs);
    double K[3] = {0.0, 0.0, 0.0};
    double crP[3], ciP[3], crT[3], ciT[3], lapU[3], lapV[3];
    double eg = 0.0, etg = 0.0;
    // one field through its three directions
    auto field = [&](int q, double *lu_out, double *lv_out, double *cr, double *ci, double &esum) {
        const int fre = field_re(q), fim = field_im(q), a = q % 3;
        const double u = c.get(fre, 0, 0), v = c.get(fim, 0, 0);
        double lu = 0.0, lv = 0.0;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const double cP = cs[d], sP = sn[d];
            const double up = d == 0 ? p.get(fre, 0, 0) : c.get(fre, d == 1, d == 2);
            const double vp = d == 0 ? p.get(fim, 0, 0) : c.get(fim, d == 1, d == 2);
            const double fr = rfma(-sP, vp, rmul(cP, up)), fi = rfma(sP, up, rmul(cP, vp));
            double br, bi;
            if (d == 0) {
                br = cy.t[fre];
                bi = cy.t[fim];
                cy.t[fre] = rfma(sP, v, rmul(cP, u));
                cy.t[fim] = rfma(-sP, u, rmul(cP, v));
            } else {
                const double cM = cs[2 + d], sM = sn[2 + d];
                const double um = c.get(fre, -(d == 1), -(d == 2)), vm = c.get(fim, -(d == 1), -(d == 2));
                br = rfma(sM, vm, rmul(cM, um));
                bi = rfma(-sM, um, rmul(cM, vm));
            }
            if (d == 0) { lu = radd(fr, br); lv = radd(fi, bi); }
            else { lu = radd(radd(lu, fr), br); lv = radd(radd(lv, fi), bi); }
            // the current, cross terms included: the own value plus r times the partner's
            double gu = u, gv = v;
            if (a != d) {
                // Phi_a meets Theta_b, Theta_a meets Phi_b, b the third index;
                // sign + for (Phi, a = d+1) and (Theta, a = d+1) with reversed roles
                const int b = 3 - d - a;
                const int o = q < 3 ? 3 + b : b;
                const bool plus = (a == (d + 1) % 3);
                const double r = plus ? k.r : -k.r;
                gu = rfma(r, c.again(field_re(o)), u);
                gv = rfma(r, c.again(field_im(o)), v);
            }
            K[d] = rfma(gu, fi, K[d]);
            K[d] = rfma(-gv, fr, K[d]);
            // curl_c = D_{c+1} f_{c+2} - D_{c+2} f_{c+1}, differences undivided
            if (a != d || SUMS) {
                const double dr = rsub(fr, br), di = rsub(fi, bi);
                if (SUMS) esum += dr * dr + di * di;
                if (a != d) {
                    const bool plus = (a == (d + 1) % 3);
                    const int t = plus ? (d + 2) % 3 : (d + 1) % 3;
                    const int other = plus ? (t + 1) % 3 : (t + 2) % 3;   // field of the other term
                    if (a < other) { cr[t] = plus ? dr : -dr; ci[t] = plus ? di : -di; }
                    else if (plus) { cr[t] = radd(cr[t], dr); ci[t] = radd(ci[t], di); }
                    else { cr[t] = rsub(cr[t], dr); ci[t] = rsub(ci[t], di); }
                }
            }
        }
        *lu_out = lu;
        *lv_out = lv;
    };
#pragma unroll
    for (int a = 0; a < 3; a++) field(a, &lapU[a], &lapV[a], crP, ciP, eg);
#pragma unroll
    for (int a = 0; a < 3; a++) {
        double lu, lv;
        field(3 + a, &lu, &lv, crT, ciT, etg);
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
        const double nV2 = -k.mu / rmul(den, den);   // -2 V'
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
    // staples (scp_sim.c:1214-1220): plaquette sines at x, and at x less the
    // other direction of the plane
    double pa[7] = {plaq_angle(c, p, fth, 0, 0, 0), plaq_angle(c, p, fth, 1, 0, 0), plaq_angle(c, p, fth, 2, 0, 0),
                    plaq_angle(c, p, fth, 0, -1, 0), plaq_angle(c, p, fth, 1, -1, 0),
                    plaq_angle(c, p, fth, 1, 0, -1), plaq_angle(c, p, fth, 2, 0, -1)};
    out.angles(pa[0], pa[1], pa[2]);
    sin_batch(pa);
    const double st0 = rsub(rsub(pa[0], pa[3]), rsub(pa[2], pa[6]));
    const double st1 = rsub(rsub(pa[1], pa[5]), rsub(pa[0], cy.p0));
    const double st2 = rsub(rsub(pa[2], cy.p2), rsub(pa[1], pa[4]));
    cy.p0 = pa[0];
    cy.p2 = pa[2];
    out.link(0, c.again(fth), rfma(k.stp, st0, rmul(k.gi, K[0])));
    out.link(1, c.again(fth + 1), rfma(k.stp, st1, rmul(k.gi, K[1])));
    out.link(2, c.again(fth + 2), rfma(k.stp, st2, rmul(k.gi, K[2])));
}

}  // namespace scp
