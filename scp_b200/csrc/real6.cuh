// real6.cuh -- the real six-field stepper (phi_a, theta_a real) with the
// reference's optional terms (compute_forces, sfa/sim/scp_sim.c:743-929;
// compute_energy, :1722-1801; theta_rms and P_integrated, :1803-1816):
//
//   mass mode 1    m_eff^2 = inv_alpha / (1 + inv_beta |phi|^2)
//   mass mode 3    kappa_eff = kappa / (1 + kappa_gamma |phi|^2), which adds
//                  -mu kappa_gamma kappa P^4 / D^2 phi_a,  D = 1 + kappa_gamma |phi|^2 + kappa P^2
//   Cosserat strain  alpha |C|^2,  C = curl(phi)/2 - theta
//   hardening        (beta/2) |theta|^2 |curl phi|^2
//   chiral helicity  kappa_h P^2 phi . curl(phi)
// with P = phi_0 phi_1 phi_2.  Varying the strain and hardening energies gives
// -alpha curl(C) and -2 curl(B), B = (beta/2)|theta|^2 curl(phi), on phi: the
// curl of a field that itself holds a curl, a stencil two sites wide.
//
// Structure.  A step is one launch: a CTA streams its tile column plane by
// plane through a shared-memory ring of phi and theta, and with strain or
// hardening (AUX) forms C and B of plane i+1 -- on its tile and one site
// around it -- into a two-slot table while it updates plane i, whose curls of
// C and B it reads from the table (in the plane) and from its own site's
// values of planes i-1 and i+1 (registers).  So phi is staged two sites wide
// and four planes deep (i, i+1, i+2 resident, i+3 in flight), theta one site
// wide, and C and B never leave the SM.  Momenta are read one plane ahead.
// Buffers: positions X[0..1] and momenta W, S of 6 arrays (phi_0..2,
// theta_0..2).
//
// What bounds it: dependency chains at twelve warps per SM beside DRAM, 192 B
// per site: 0.55 of a plain copy's rate at 128^3, 113 us a step against 197
// with C and B written by a launch of their own (336 B).  Every operation that reaches the
// state is explicitly rounded, so a run's bits do not depend on its launches.
#pragma once
#include "walk.cuh"

namespace scp {

struct R6Consts {
    int N;
    long long N3;
    double L, dx, dV, idx1, idx2, hdt, dt;
    double mu, kappa, m2, mtheta2, eta;
    double kh, alpha, beta, kg, ia, ib;
    int mode;
    double damp_width, damp_rate;
};

// Kernel arguments: positions x_{n+1} and the leapfrog's arrays, 6 each.
struct R6Args {
    const double *x;
    int N;
    R6Consts c;
    LeapIO io;
};

template <bool AUX, int TX, int TY>
struct R6Layout {
    static constexpr int H = AUX ? 2 : 1;                          // halo of phi
    static constexpr int NS = AUX ? 4 : 3;                         // ring slots
    static constexpr int PFS = (TX + 2 * H) * (TY + 2 * H);        // phi, one field of a slot
    static constexpr int TFS = (TX + 2) * (TY + 2);                // theta, C, B
    static constexpr int SLOT = 3 * PFS + 3 * TFS;
    static constexpr int NT = TX * TY;
    static constexpr int CP = (PFS + NT - 1) / NT, CT = (TFS + NT - 1) / NT;   // copies per thread and field
    static constexpr int AUXN = AUX ? 2 * 6 * TFS : 0;
    static constexpr size_t smem_bytes = sizeof(double) * (size_t)(NS * SLOT + AUXN);
};

template <class MODE, bool AUX, int TX, int TY>
struct R6Tile {
    using LY = R6Layout<AUX, TX, TY>;
    static constexpr int H = LY::H, NS = LY::NS, L = NS - 2;   // planes beyond i that are resident
    const R6Args &a;
    double *ring, *aux;
    int N, tx, ty, pp, pt;                // pitches of phi and theta rows
    long long NN, n3;
    int own_p, own_t;                     // own site in a phi field / a theta field
    int ps[LY::CP], pg[LY::CP], ts[LY::CT], tg_[LY::CT];   // copies: slot offset (-1: none), plane offset
    bool act;
    int halo_p, halo_t;                   // the site around the tile whose C, B this thread forms (-1: none)

    __device__ __forceinline__ R6Tile(const R6Args &args, double *smem, int tw)
        : a(args), ring(smem), aux(smem + NS * LY::SLOT), N(args.N) {
        ty = (int)threadIdx.x / tw;
        tx = (int)threadIdx.x - ty * tw;
        pp = tw + 2 * H;
        pt = tw + 2;
        NN = (long long)N * N;
        n3 = NN * N;
        own_p = (ty + H) * pp + tx + H;
        own_t = (ty + 1) * pt + tx + 1;
    }
    __device__ __forceinline__ void begin(int k0, int j0, int nk, int nj) {
        act = tx < nk && ty < nj;
        const int wp = nk + 2 * H, wt = nk + 2;
#pragma unroll
        for (int q = 0; q < LY::CP; q++) {
            const int h = (int)threadIdx.x + q * LY::NT, r = h / wp, col = h - r * wp;
            ps[q] = r < nj + 2 * H ? r * pp + col : -1;
            pg[q] = wrapi(j0 - H + r, N) * N + wrapi(k0 - H + col, N);
        }
#pragma unroll
        for (int q = 0; q < LY::CT; q++) {
            const int h = (int)threadIdx.x + q * LY::NT, r = h / wt, col = h - r * wt;
            ts[q] = r < nj + 2 ? r * pt + col : -1;
            tg_[q] = wrapi(j0 - 1 + r, N) * N + wrapi(k0 - 1 + col, N);
        }
        halo_p = halo_t = -1;
        if (AUX) {   // rows -1 and nj, columns -1 and nk (no corners)
            const int h = threadIdx.x;
            int r = 0, col = -2;
            if (h < nk) { r = -1; col = h; }
            else if (h < 2 * nk) { r = nj; col = h - nk; }
            else if (h < 2 * nk + nj) { r = h - 2 * nk; col = -1; }
            else if (h < 2 * nk + 2 * nj) { r = h - 2 * nk - nj; col = nk; }
            if (col > -2) {
                halo_p = (r + H) * pp + col + H;
                halo_t = (r + 1) * pt + col + 1;
            }
        }
    }
    __device__ __forceinline__ void issue(int plane, int slot) {
        const double *g = a.x + (long long)wrapi(plane, N) * NN;
        double *sp = ring + slot * LY::SLOT, *st = sp + 3 * LY::PFS;
#pragma unroll
        for (int q = 0; q < LY::CP; q++)
            if (ps[q] >= 0) {
#pragma unroll
                for (int f = 0; f < 3; f++) cp_async8(sp + f * LY::PFS + ps[q], g + f * n3 + pg[q]);
            }
#pragma unroll
        for (int q = 0; q < LY::CT; q++)
            if (ts[q] >= 0) {
#pragma unroll
                for (int f = 0; f < 3; f++) cp_async8(st + f * LY::TFS + ts[q], g + (3 + f) * n3 + tg_[q]);
            }
        cp_async_commit();
    }
    __device__ __forceinline__ const double *phi(int slot) const { return ring + slot * LY::SLOT; }
    __device__ __forceinline__ const double *theta(int slot) const { return ring + slot * LY::SLOT + 3 * LY::PFS; }

    // curl of phi at offset o of slot c, neighbours along i in slots m and p
    __device__ __forceinline__ void curl_phi(const double *m, const double *c, const double *p, int o,
                                             double (&cp)[3]) const {
        const double idx1 = a.c.idx1;
        auto d = [&](int dir, int f) {
            const int at = f * LY::PFS + o;
            return dir == 0 ? rsub(p[at], m[at])
                            : dir == 1 ? rsub(c[at + pp], c[at - pp]) : rsub(c[at + 1], c[at - 1]);
        };
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const int b = (q + 1) % 3, e = (q + 2) % 3;
            cp[q] = rmul(rsub(d(b, e), d(e, b)), idx1);
        }
    }
    // C and B from the curl of phi and theta at one site
    __device__ __forceinline__ void fields(const double (&cp)[3], double t0, double t1, double t2, double (&C)[3],
                                           double (&B)[3]) const {
        const double w = rmul(0.5 * a.c.beta, rfma(t2, t2, rfma(t1, t1, rmul(t0, t0))));
        C[0] = rfma(0.5, cp[0], -t0);
        C[1] = rfma(0.5, cp[1], -t1);
        C[2] = rfma(0.5, cp[2], -t2);
#pragma unroll
        for (int q = 0; q < 3; q++) B[q] = rmul(w, cp[q]);
    }
    // C, B of one plane (slot c; m, p beside it) at phi offset op / theta offset ot into table slot s
    __device__ __forceinline__ void table(int m, int c, int p, int op, int ot, int s, double (&cp)[3], double (&C)[3],
                                          double (&B)[3]) const {
        curl_phi(phi(m), phi(c), phi(p), op, cp);
        const double *t = theta(c) + ot;
        fields(cp, t[0], t[LY::TFS], t[2 * LY::TFS], C, B);
        double *o = aux + s * 6 * LY::TFS + ot;
#pragma unroll
        for (int q = 0; q < 3; q++) {
            o[q * LY::TFS] = C[q];
            o[(3 + q) * LY::TFS] = B[q];
        }
    }
};

template <class MODE, bool AUX, int TX, int TY>
__device__ __forceinline__ void r6_item(R6Tile<MODE, AUX, TX, TY> &T, const TileGrid &tg, const Piece &pc) {
    using LY = R6Layout<AUX, TX, TY>;
    constexpr int NS = LY::NS, L = NS - 2, FS = LY::PFS, TS = LY::TFS;
    const R6Args &A = T.a;
    const R6Consts &c = A.c;
    const int N = T.N, k0 = pc.kt * tg.tw, j0 = pc.jt * tg.th, i0 = pc.i0, i1 = pc.i1;
    T.begin(k0, j0, min(tg.tw, N - k0), min(tg.th, N - j0));
    const int j = j0 + T.ty, k = k0 + T.tx, own_g = j * N + k;
    // plane q sits in slot (q - i0 + L) mod NS
    auto slot = [&](int q) { return (q - i0 + L) % NS; };
    __syncthreads();   // the previous item's last plane has been read
#pragma unroll
    for (int q = 0; q < NS; q++) T.issue(i0 - L + q, q);   // planes i0-L .. i0+1
    double w[6], xm[6], cpc[3], Cm[2], Bm[2];   // momenta; x, and C_1, C_2, B_1, B_2 at x - i; curl phi at x
    if (T.act) {
#pragma unroll
        for (int f = 0; f < 6; f++) w[f] = ld_early(A.io.win[0] + f * T.n3 + (long long)i0 * T.NN + own_g);
    }
    cp_async_wait<0>();
    __syncthreads();
    {
        const int sm = slot(i0 - 1), sc = slot(i0), sp = slot(i0 + 1);
        double cp[3], C[3], B[3];
        if (T.act) {
#pragma unroll
            for (int f = 0; f < 3; f++) {
                xm[f] = T.phi(sm)[f * FS + T.own_p];
                xm[3 + f] = T.theta(sm)[f * TS + T.own_t];
            }
            if constexpr (AUX) {
                T.curl_phi(T.phi(slot(i0 - 2)), T.phi(sm), T.phi(sc), T.own_p, cp);
                T.fields(cp, xm[3], xm[4], xm[5], C, B);
                Cm[0] = C[1]; Cm[1] = C[2]; Bm[0] = B[1]; Bm[1] = B[2];
                T.table(sm, sc, sp, T.own_p, T.own_t, 0, cpc, C, B);
            }
        }
        if constexpr (AUX) {
            if (T.halo_p >= 0) T.table(sm, sc, sp, T.halo_p, T.halo_t, 0, cp, C, B);
            __syncthreads();   // plane i0-2 has been read: its slot takes plane i0+2
            T.issue(i0 + 2, slot(i0 + 2));
        }
    }
    for (int i = i0; i < i1; i++) {
        const int sc = slot(i), sp = slot(i + 1);
        if constexpr (AUX) cp_async_wait<0>();   // plane i+2 (without AUX the prologue or the last round waited)
        else if (i > i0) cp_async_wait<0>();
        __syncthreads();   // copies and the table of plane i are visible; plane i-1 and its table are free
        if (i + L + 1 <= i1 + L - 1) T.issue(i + L + 1, slot(i + L + 1));
        double Cn[3], Bn[3], cpn[3];
        const int an = (i + 1 - i0) & 1;         // table slot of plane i+1
        if constexpr (AUX) {
            const int s2 = slot(i + 2);
            if (T.act) T.table(sc, sp, s2, T.own_p, T.own_t, an, cpn, Cn, Bn);
            if (T.halo_p >= 0 && i + 1 < i1) {
                double cp[3], C[3], B[3];
                T.table(sc, sp, s2, T.halo_p, T.halo_t, an, cp, C, B);
            }
        }
        if (!T.act) continue;
        const double *ph = T.phi(sc) + T.own_p, *php = T.phi(sp) + T.own_p;
        const double *th = T.theta(sc) + T.own_t, *thp = T.theta(sp) + T.own_t;
        const double p[3] = {ph[0], ph[FS], ph[2 * FS]}, t[3] = {th[0], th[TS], th[2 * TS]};
        // neighbours of field f (phi 0-2, theta 3-5): direction d, side s
        auto nbr = [&](int f, int d, int s) -> double {
            if (d == 0) return s < 0 ? xm[f] : (f < 3 ? php[f * FS] : thp[(f - 3) * TS]);
            if (f < 3) return ph[f * FS + s * (d == 1 ? T.pp : 1)];
            return th[(f - 3) * TS + s * (d == 1 ? T.pt : 1)];
        };
        const double sig = rfma(p[2], p[2], rfma(p[1], p[1], rmul(p[0], p[0])));
        const double m2e = (c.mode == 1) ? c.ia / rfma(c.ib, sig, 1.0) : c.m2;
        const double ke = (c.mode == 3) ? c.kappa / rfma(c.kg, sig, 1.0) : c.kappa;
        const double P = rmul(rmul(p[0], p[1]), p[2]), P2 = rmul(P, P);
        const double q = rfma(ke, P2, 1.0);
        const double dVdP = rmul(c.mu, P) / rmul(q, q);
        double extra = 0.0;   // mode 3's additional -extra * phi_a
        if (c.mode == 3 && c.kg > 0) {
            const double D = rfma(c.kappa, P2, rfma(c.kg, sig, 1.0));
            extra = rmul(rmul(rmul(rmul(c.mu, c.kg), c.kappa), P2), P2) / rmul(D, D);
        }
        double ct[3], cp[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const int b = (a + 1) % 3, e = (a + 2) % 3;
            ct[a] = rmul(rsub(rsub(nbr(3 + e, b, 1), nbr(3 + e, b, -1)), rsub(nbr(3 + b, e, 1), nbr(3 + b, e, -1))),
                         c.idx1);
            cp[a] = AUX ? cpc[a]
                        : rmul(rsub(rsub(nbr(e, b, 1), nbr(e, b, -1)), rsub(nbr(b, e, 1), nbr(b, e, -1))), c.idx1);
        }
        const double cp2 = rfma(cp[2], cp[2], rfma(cp[1], cp[1], rmul(cp[0], cp[0])));
        double hel = 0.0, gP2[3] = {0.0, 0.0, 0.0};   // phi . curl phi, gradient of P^2
        if (c.kh != 0.0) {
            hel = rfma(p[2], cp[2], rfma(p[1], cp[1], rmul(p[0], cp[0])));
#pragma unroll
            for (int d = 0; d < 3; d++) {
                const double Pp = rmul(rmul(nbr(0, d, 1), nbr(1, d, 1)), nbr(2, d, 1));
                const double Pm = rmul(rmul(nbr(0, d, -1), nbr(1, d, -1)), nbr(2, d, -1));
                gP2[d] = rmul(rfma(Pp, Pp, -rmul(Pm, Pm)), c.idx1);
            }
        }
        // curls of C and B: in the plane from the table, along i from this
        // site's own values
        double cC[3] = {0.0, 0.0, 0.0}, cB[3] = {0.0, 0.0, 0.0};
        if constexpr (AUX) {
            const double *ax = T.aux + ((i - i0) & 1) * 6 * TS + T.own_t;
            auto curl = [&](const double *f, const double (&n)[3], const double (&m)[2], double (&o)[3]) {
                auto dj = [&](int q2) { return rsub(f[q2 * TS + T.pt], f[q2 * TS - T.pt]); };
                auto dk = [&](int q2) { return rsub(f[q2 * TS + 1], f[q2 * TS - 1]); };
                o[0] = rmul(rsub(dj(2), dk(1)), c.idx1);
                o[1] = rmul(rsub(dk(0), rsub(n[2], m[1])), c.idx1);
                o[2] = rmul(rsub(rsub(n[1], m[0]), dj(0)), c.idx1);
            };
            curl(ax, Cn, Cm, cC);
            curl(ax + 3 * TS, Bn, Bm, cB);
        }
        const double dmp = (MODE::DAMP && !MODE::FIRST) ? sponge_factor(i, j, k, c.L, c.dx, c.damp_width, c.damp_rate)
                                                        : 1.0;
        const long long site = (long long)i * T.NN + own_g;
        LeapSite<MODE, 6> leap{A.io, w, T.n3, site, i + 1 < i1 ? T.NN : 0, c.hdt, c.dt, dmp};
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const int b = (a + 1) % 3, e = (a + 2) % 3;
            auto lap = [&](int f, double x) {
                double l = radd(nbr(f, 0, 1), nbr(f, 0, -1));
                l = radd(radd(l, nbr(f, 1, 1)), nbr(f, 1, -1));
                l = radd(radd(l, nbr(f, 2, 1)), nbr(f, 2, -1));
                return rmul(rfma(-6.0, x, l), c.idx2);
            };
            const double dPa = rmul(p[b], p[e]);   // dP / dphi_a
            double f = rfma(-m2e, p[a], lap(a, p[a]));
            f = rfma(-dVdP, dPa, f);
            f = rfma(-extra, p[a], f);
            f = rfma(c.eta, ct[a], f);
            if (c.kh != 0.0) {
                // kappa_h [2 P dP/dphi_a (phi.curl phi) + 2 P^2 curl_a phi + (grad P^2 x phi)_a]
                const double cross = rfma(gP2[b], p[e], -rmul(gP2[e], p[b]));
                const double ch = rfma(rmul(rmul(2.0, P), dPa), hel, rfma(rmul(2.0, P2), cp[a], cross));
                f = rfma(c.kh, ch, f);
            }
            if constexpr (AUX) {
                f = rfma(-c.alpha, cC[a], f);
                f = rfma(-2.0, cB[a], f);
            }
            double g = rfma(-c.mtheta2, t[a], lap(3 + a, t[a]));
            g = rfma(c.eta, cp[a], g);
            if constexpr (AUX) {
                g = rfma(rmul(2.0, c.alpha), rfma(0.5, cp[a], -t[a]), g);   // 2 alpha C_a
                g = rfma(rmul(-c.beta, cp2), t[a], g);
            }
            leap.put(a, p[a], f, dmp);
            leap.put(3 + a, t[a], g, dmp);
        }
        if (MODE::SYNC && leap.bad) atomicOr(A.io.flag, 1);
#pragma unroll
        for (int f = 0; f < 3; f++) {
            xm[f] = p[f];
            xm[3 + f] = t[f];
        }
        if constexpr (AUX) {
            // plane i's own C, B become those at x - i
            const double *ax = T.aux + ((i - i0) & 1) * 6 * TS + T.own_t;
            Cm[0] = ax[TS]; Cm[1] = ax[2 * TS]; Bm[0] = ax[4 * TS]; Bm[1] = ax[5 * TS];
#pragma unroll
            for (int a = 0; a < 3; a++) cpc[a] = cpn[a];
        }
    }
}

template <class MODE, bool AUX, int TX, int TY>
__global__ void __launch_bounds__(TX *TY, 1) r6_kernel(R6Args a, TileGrid tg) {
    extern __shared__ __align__(16) double r6_smem[];
    R6Tile<MODE, AUX, TX, TY> T(a, r6_smem, tg.tw);
    griddep_wait();
    griddep_launch();
    for_each_piece(tg, a.N, [&](const Piece &pc) { r6_item<MODE, AUX, TX, TY>(T, tg, pc); });
}

}  // namespace scp
