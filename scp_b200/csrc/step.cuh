// step.cuh -- fused leapfrog step for the complex (v66) and gauged (v69)
// Cosserat Q-ball lattice, one launch per time step, in two precisions:
//   F64   all state and arithmetic in FP64 (the drop-in mode);
//   F32C  FP32 state and arithmetic; positions carried as a compensated pair
//         (hi: fp32, lo: bf16 for the matter fields, fp32 for the link
//         angles) so the drift accumulates without loss.
//         F32C evaluates Laplacians, currents and plaquette angles as sums of
//         neighbour differences, which removes the cancellation that FP32
//         would otherwise suffer against O(|f|) values.
//
// Time integration.  The reference runs kick / drift / force / kick as about
// ten separate sweeps per step (sfa/sim/scp_sim.c:1583-1716, GPU launch
// sequence sfa/sim/scp_sim.cu:2971-3208) and keeps an acceleration array.
// Here the state between launches is (x_{n+1}, w_n) with the half-step
// momentum w_n = v_n + hdt*a_n, and launch n+1 performs, per site,
//     a_{n+1} = F(x_{n+1})                    (stencil of x_{n+1})
//     v_{n+1} = w_n + hdt*a_{n+1}             (reference stage-4 kick)
//     [v_{n+1} *= damp(r)]                    (reference stage 5, bc_type 0)
//     w_{n+1} = v_{n+1} + hdt*a_{n+1}         (next step's stage-1 kick)
//     x_{n+2} = x_{n+1} + dt*w_{n+1}          (next step's drift)
// so no acceleration array exists and each state word is read once and written
// once per step.  (The terms are the reference's; in FP64 they are summed field
// by field, gauged.cuh, to roundoff of the reference's order.)  Links follow the same pattern with E and the wrapped drift
// th += -g*dx*dt*E.  The launch that starts a run (FIRST) reads v_0 instead
// of w and skips the stage-4 kick; a SYNC launch also stores v_{n+1} and
// E_{n+1} for diagnostics and snapshots.
//
// Data movement.  Persistent CTAs walk work items = tile columns (tw x th
// sites in k and j, chosen per grid) times segments of `seg` planes in i.  A
// CTA streams its column plane by plane through a 3-slot shared-memory ring
// (plane i, plane i+1, and plane i+2 in flight via cp.async).  Every thread
// copies its own site; the halo rows and columns (periodic wrap) are spread
// over the CTA's threads so each thread issues the same copies with no
// per-field branches.  What a site needs of plane i-1 is carried in registers
// (FP64: the backward transports along i, or x(i-1) without links; F32C:
// x(i-1)), and so are the momenta, read one plane ahead.  In gauged mode every
// thread evaluates the link cos/sin and plaquette sines it needs itself: its
// own site, the j-1 and k-1 neighbours (recomputed from the ring), and the
// i-1 values carried from the previous plane -- more sines than sharing them
// through shared memory, but no extra barrier per plane.
//
// FP64, what bounds it: DRAM.  A gauged step moves 480 B per site (every state
// word read and written once) and ran at 0.69 of a plain copy's rate while its
// momenta were loaded at the top of the plane that uses them: with 8 warps an
// SM, the warps sat on those loads (2 of 5.4 cycles per issue) whatever the
// arithmetic cost.  Loading them one plane ahead (gauged.cuh frees the
// registers that takes), and 256-site tiles with their smaller halo, bring it
// to 0.85 at 128^3 (182 us against 227) and 0.88 at 256^3 (1.41 ms against
// 1.78).  Three CTAs of 168 registers were slower (278 us at 128^3): the ring
// of three leaves the L1 too few lines for the copies in flight.  So were
// 16-byte copies past L1 (206 against 198 us on 32 x 4 tiles).
#pragma once
#include <cuda_bf16.h>

#include <type_traits>

#include "common.cuh"
#include "diag.cuh"
#include "gauged.cuh"
#include "trig.cuh"

namespace scp {

struct F64 {
    using T = double;
    static constexpr bool COMP = false;
};
struct F32C {
    using T = float;
    static constexpr bool COMP = true;
};

template <class P>
struct StepIO {
    using T = typename P::T;
    const T *xin;           // NF arrays of N^3: positions x_{n+1} (hi part in F32C)
    T *xout;                // NF arrays: x_{n+2}
    const uint16_t *loin;   // F32C: bf16 low parts of the 12 matter positions
    uint16_t *loout;
    const float *tloin;     // F32C gauged: low parts of the 3 link angles
    float *tloout;
    const T *win;           // NF arrays: w_n (or v_0, E_0 when FIRST)
    T *wout;                // NF arrays: w_{n+1} (may alias win)
    T *sout;                // NF arrays: v_{n+1}, E_{n+1} (SYNC only)
    int *flag;              // nonfinite flag (SYNC only)
    // FP64 SYNC launches of the single-grid kernel: when set, the launch also
    // sums the first diagnostics pass at (x_{n+1}, v_{n+1}) -- one partial of
    // DS_NSUM + DM_NMAX slots per CTA into dpart -- and stores the Gauss-law
    // charge density of every site into drho (gauged)
    double *dpart = nullptr;
    double *drho = nullptr;
    double *dfold = nullptr;      // the last CTA folds the partials here
    unsigned *dcount = nullptr;   // CTAs done
};

template <class P, int TX, int TY, bool GAUGED>
struct StepLayout {
    using T = typename P::T;
    static constexpr int NF = GAUGED ? 15 : 12;
    static constexpr int NR = NF + ((P::COMP && GAUGED) ? 3 : 0);   // ring fields (+ link lo parts)
    static constexpr int PX = TX + 2, PY = TY + 2;
    static constexpr int PLANE = NR * PY * PX;            // elements per ring slot
    static constexpr int NT = TX * TY;
    static constexpr int NHALO = 2 * TX + 2 * TY + (GAUGED ? 2 : 0);
    static constexpr int HPT = (NHALO + NT - 1) / NT;      // halo sites per thread (max)
    static constexpr size_t smem_bytes = sizeof(T) * (size_t)(3 * PLANE);
};

__device__ __forceinline__ void cp_async_elem(double *s, const double *g) { cp_async8(s, g); }
__device__ __forceinline__ void cp_async_elem(float *s, const float *g) { cp_async4(s, g); }

__device__ __forceinline__ float bf16_to_f(uint16_t h) { return __uint_as_float((uint32_t)h << 16); }
__device__ __forceinline__ uint16_t f_to_bf16(float f) {
    return __bfloat16_as_ushort(__float2bfloat16_rn(f));
}

// exact sum: s + e = a + b (Knuth two-sum)
__device__ __forceinline__ void two_sum(float a, float b, float *s, float *e) {
    const float t = a + b;
    const float bb = t - a;
    *e = (a - (t - bb)) + (b - bb);
    *s = t;
}

// Plane staging of the classic ring: every thread copies its own site with
// cp.async, and the halo rows and columns (periodic wrap, two corners for
// the gauged plaquettes) are spread over the CTA's threads.  Slot layout
// [NR][PY][PX] of StepLayout; any grid size.
template <class P, int TX, int TY, bool GAUGED>
struct CpStage {
    using T = typename P::T;
    using LY = StepLayout<P, TX, TY, GAUGED>;
    static constexpr int NSLOT = 3;   // ring slots: planes i, i+1 resident, i+2 in flight
    static constexpr bool MOM = false;   // momenta read from global memory at the site
    __device__ __forceinline__ void issue_mom(int, int) {}
    __device__ __forceinline__ void wait_mom(int) {}
    __device__ __forceinline__ T mom(int, int) const { return T(0); }
    static constexpr int NF = LY::NF, NR = LY::NR, PX = LY::PX, PY = LY::PY, NT = LY::NT;
    T *xs;
    int N;
    long long N3;
    bool act;
    int tx, ty, pitch;
    int oc, c_s;
    int h_s[LY::HPT], h_g[LY::HPT], h_nf[LY::HPT];

    // tw x th sites of a tile, one thread each: at most TX * TY of them, and
    // a ring field of (tw + 2) x (th + 2) fits the layout's PY * PX
    __device__ __forceinline__ CpStage(unsigned char *smem, int tw) : xs(reinterpret_cast<T *>(smem)) {
        ty = (int)threadIdx.x / tw;
        tx = (int)threadIdx.x - ty * tw;
        pitch = tw + 2;
    }

    // per-item set-up: this thread's own site and its halo copies
    __device__ __forceinline__ void begin(const StepConsts &c, int k0, int j0, int nk, int nj) {
        N = c.N;
        N3 = c.N3;
        const int tid = threadIdx.x;
        act = (tx < nk) && (ty < nj);
        oc = (j0 + ty) * N + k0 + tx;
        c_s = (ty + 1) * pitch + tx + 1;
        const int jlo = wrapi(j0 - 1, N), jhi = wrapi(j0 + nj, N);
        const int klo = wrapi(k0 - 1, N), khi = wrapi(k0 + nk, N);
#pragma unroll
        for (int q = 0; q < LY::HPT; q++) {
            const int h = tid + q * NT;
            int r = 0, col = 0, gj = 0, gk = 0, nf = 0;
            if (h < nk) { r = 0; col = h + 1; gj = jlo; gk = k0 + h; nf = NF; }
            else if (h < 2 * nk) { r = nj + 1; col = h - nk + 1; gj = jhi; gk = k0 + h - nk; nf = NF; }
            else if (h < 2 * nk + nj) { r = h - 2 * nk + 1; col = 0; gj = j0 + h - 2 * nk; gk = klo; nf = NF; }
            else if (h < 2 * nk + 2 * nj) { r = h - 2 * nk - nj + 1; col = nk + 1; gj = j0 + h - 2 * nk - nj; gk = khi; nf = NF; }
            else if (GAUGED && h == 2 * nk + 2 * nj) { r = nj + 1; col = 0; gj = jhi; gk = klo; nf = 3; }
            else if (GAUGED && h == 2 * nk + 2 * nj + 1) { r = 0; col = nk + 1; gj = jlo; gk = khi; nf = 3; }
            h_s[q] = r * pitch + col;
            h_g[q] = gj * N + gk;
            h_nf[q] = nf;
        }
    }

    __device__ __forceinline__ void issue(const StepIO<P> &io, int p, int slot) {
        const long long pb = (long long)wrapi(p, N) * N * N;
        T *sbase = xs + slot * LY::PLANE;
        const T *gbase = io.xin + pb;
        if (act) {
#pragma unroll
            for (int f = 0; f < NF; f++)
                cp_async_elem(sbase + f * PY * PX + c_s, gbase + f * N3 + oc);
            if constexpr (NR > NF) {
#pragma unroll
                for (int f = NF; f < NR; f++)
                    cp_async_elem(sbase + f * PY * PX + c_s, io.tloin + pb + (f - NF) * N3 + oc);
            }
        }
#pragma unroll
        for (int q = 0; q < LY::HPT; q++) {
            const int nf = h_nf[q];
            if (nf == 0) continue;
            const int f0 = (nf == NF) ? 0 : FTH;   // corners carry only the link angles
#pragma unroll
            for (int f = 0; f < NF; f++)
                if (f >= f0) cp_async_elem(sbase + f * PY * PX + h_s[q], gbase + f * N3 + h_g[q]);
            if constexpr (NR > NF) {
#pragma unroll
                for (int f = NF; f < NR; f++)
                    cp_async_elem(sbase + f * PY * PX + h_s[q], io.tloin + pb + (f - NF) * N3 + h_g[q]);
            }
        }
    }
    __device__ __forceinline__ void commit() { cp_async_commit(); }
    // this thread's copies have landed, all but the PENDING latest groups (a barrier follows)
    template <int PENDING>
    __device__ __forceinline__ void wait(int) { cp_async_wait<PENDING>(); }
    __device__ __forceinline__ bool failed() const { return false; }
    // the values around this thread's site in one slot
    struct View {
        const T *p;
        int pitch;
        __device__ __forceinline__ T get(int f, int dj, int dk) const { return p[f * (PY * PX) + dj * pitch + dk]; }
        // the own value, read again instead of kept in a register
        __device__ __forceinline__ T again(int f) const { return get(f, 0, 0); }
    };
    __device__ __forceinline__ View view(int slot) const { return View{xs + slot * LY::PLANE + c_s, pitch}; }
};

// ---------------------------------------------------------------- FP64

// Per-thread sums of the first diagnostics pass (energies, charges, core and
// centroid moments, the per-site terms of diag_walk.cuh) over the sites a
// synchronous launch advances, without the constant factors, which step_sums
// applies once per thread.
enum : int {
    SS_EPK = 0, SS_ETK, SS_EG, SS_ETG, SS_EP, SS_EC, SS_EE, SS_BB, SS_PINT, SS_TRS, SS_M0, SS_CX, SS_CY, SS_CZ,
    SS_QP0, SS_QP1, SS_QP2, SS_QT, SS_QC, SS_N
};
struct StepSums {
    double s[SS_N];
    double pm, smax;   // largest |Phi_a|^2 and their product
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int q = 0; q < SS_N; q++) s[q] = 0.0;
        pm = smax = 0.0;
    }
};

// The slots of the first pass from one thread's sums (the Gauss-law slots are
// left to the pass that reads E of the neighbouring sites).
template <class C>
__device__ __forceinline__ void step_sums(const StepSums &t, const C &c, DiagSums &o) {
    o.clear();
    const double hV = 0.5 * c.dV, g2 = c.idx1 * c.idx1;
    o.S[DS_EPK] = hV * t.s[SS_EPK];
    o.S[DS_ETK] = hV * t.s[SS_ETK];
    o.S[DS_EG] = hV * g2 * t.s[SS_EG];
    o.S[DS_ETG] = hV * g2 * t.s[SS_ETG];
    o.S[DS_EM] = hV * c.m2 * t.s[SS_M0];
    o.S[DS_ETM] = hV * c.mtheta2 * t.s[SS_TRS];
    o.S[DS_EP] = hV * c.mu * t.s[SS_EP];
    o.S[DS_EC] = -c.ei * c.dV * t.s[SS_EC];
    o.S[DS_EEM] = c.dV * (0.5 * t.s[SS_EE] + c.bpre * t.s[SS_BB]);
    o.S[DS_PINT] = c.dV * t.s[SS_PINT];
    o.S[DS_TRS] = t.s[SS_TRS];
    o.S[DS_QP] = t.s[SS_QP0] + t.s[SS_QP1] + t.s[SS_QP2];
    o.S[DS_QT] = t.s[SS_QT];
    o.S[DS_M0] = t.s[SS_M0];
    o.S[DS_CX] = t.s[SS_CX];
    o.S[DS_CY] = t.s[SS_CY];
    o.S[DS_CZ] = t.s[SS_CZ];
    o.S[DS_QC] = t.s[SS_QC];
    o.S[DS_QP0] = t.s[SS_QP0];
    o.S[DS_QP1] = t.s[SS_QP1];
    o.S[DS_QP2] = t.s[SS_QP2];
    o.M[DM_PM] = sqrt(t.pm);
    o.M[DM_PMAX] = sqrt(t.smax);
    o.M[DM_SMAX] = t.smax;
}

// The site's momenta w_n, read one plane ahead: each is replaced by the next
// plane's once its kick has used it, so a load has a whole plane of arithmetic
// to pass under.
//
// Where the loads stand.  They are ordinary loads of memory that this launch
// also stores to, so the compiler keeps them where they are written among the
// stores, and the place matters (us a step, loads ahead of a component's stores
// against the form taken): without links each between its component's two
// stores (113^3 138 -> 123, 160^3 292 -> 281, 128^3 144 -> 145); with links
// Phi's like that and Theta's as one batch once the triplet's stores are out
// (128^3 190 -> 183, 192^3 582 -> 563, 113^3 187 -> 185; Theta's like Phi's
// 128^3 189, 192^3 577, 113^3 172).  All of them at the end of the site: 197 at
// 128^3 with links.
template <bool GAUGED>
struct Momenta {
    double v[GAUGED ? 15 : 12];
};

// Kick, damping and drift of one site (scp_sim.c:1591-1715, fused) as the
// accelerations come in; with DIAG also the per-site terms of the sums.
template <bool GAUGED, bool FIRST, bool DIAG, class Stage>
struct SiteUpdate {
    const StepIO<F64> &io;
    const StepConsts &c;
    const Stage &stg;
    StepSums *sums;
    const long long site;
    const int mslot;       // momentum slot of the staging (Stage::MOM)
    const bool SYNC, DAMP;
    Momenta<GAUGED> &w;
    const long long next;   // elements to the next plane's site, 0 on a segment's last plane (what is then
                            // read is not used; a load behind a branch would be copied, and waited
                            // for, where the branch joins)
    double dmp = 1.0;
    bool bad = false;
    double rho = 0.0, rho2 = 0.0;   // charge density and sum of |Phi_a|^2 of the site (DIAG)

    __device__ __forceinline__ double mom(int f) const {
        if constexpr (Stage::MOM) return stg.mom(mslot, f);
        else return w.v[f];
    }
    // the momentum of the next plane, once this plane's is used
    __device__ __forceinline__ void ahead(int f) const {
        if constexpr (!Stage::MOM)
            w.v[f] = ld_early(io.win + f * c.N3 + site + next);
    }
    __device__ __forceinline__ double kick(double w, double a, double *wn) const {
        double v = FIRST ? w : rfma(c.hdt, a, w);
        if (DAMP && !FIRST) v = rmul(v, dmp);
        *wn = rfma(c.hdt, a, v);
        return v;
    }
    __device__ __forceinline__ double put(int f, double x, double a) {
        double wn;
        const double v = kick(mom(f), a, &wn);
        const double xn = rfma(c.dt, wn, x);
        io.wout[f * c.N3 + site] = wn;
        if (!GAUGED || f < FTU) ahead(f);
        st_cs(io.xout + f * c.N3 + site, xn);
        if (SYNC && !FIRST) {
            st_cs(io.sout + f * c.N3 + site, v);
            bad |= !isfinite(xn) || !isfinite(v);
        }
        return v;
    }
    __device__ __forceinline__ void theta(int a, double u, double v, double au, double av) {
        const double pu = put(FTU + a, u, au), pv = put(FTV + a, v, av);
        if constexpr (DIAG) {
            sums->s[SS_ETK] += pu * pu + pv * pv;
            sums->s[SS_TRS] += u * u + v * v;
            const double q = u * pv - v * pu;
            sums->s[SS_QT] += q;
            rho += q;
        }
    }
    __device__ __forceinline__ void phi(int a, double u, double v, double au, double av) {
        const double pu = put(FU + a, u, au), pv = put(FV + a, v, av);
        if constexpr (DIAG) {
            sums->s[SS_EPK] += pu * pu + pv * pv;
            const double q = u * pv - v * pu;
            sums->s[SS_QP0 + a] += q;
            rho += q;
        }
    }
    // potential terms: squared moduli of Phi, den = 1 + kappa s; Theta is done
    __device__ __forceinline__ void moduli(const double (&s)[3], double den) {
        if constexpr (GAUGED) {
#pragma unroll
            for (int f = 0; f < 6; f++) ahead(FTU + f);
        }
        if constexpr (DIAG) {
            const double s3 = s[0] * s[1] * s[2];
            rho2 = s[0] + s[1] + s[2];
            sums->s[SS_M0] += rho2;
            sums->s[SS_EP] += s3 / den;
            sums->s[SS_PINT] += sqrt(s3);
            sums->pm = fmax(sums->pm, fmax(s[0], fmax(s[1], s[2])));
            sums->smax = fmax(sums->smax, s3);
        }
    }
    __device__ __forceinline__ void angles(double p0, double p1, double p2) {
        if constexpr (DIAG) {   // 1 - cos of the site's own plaquettes, as 2 sin^2 of the half angle
            double h[3] = {0.5 * p0, 0.5 * p1, 0.5 * p2};
            sin_batch(h);
            sums->s[SS_BB] += 2.0 * (h[0] * h[0] + h[1] * h[1] + h[2] * h[2]);
        }
    }
    __device__ __forceinline__ double current(int, double K) const { return K; }   // charged links only
    __device__ __forceinline__ void link(int d, double th0, double K) {
        double Eh;
        const double E = kick(mom(FTH + d), K, &Eh);
        const double th = link_wrap(rfma(c.gad, Eh, th0));
        st_cs(io.xout + (FTH + d) * c.N3 + site, th);
        io.wout[(FTH + d) * c.N3 + site] = Eh;
        if (SYNC && !FIRST) {
            st_cs(io.sout + (FTH + d) * c.N3 + site, E);
            bad |= !isfinite(E) || !isfinite(th);
        }
        ahead(FTH + d);
        if constexpr (DIAG) sums->s[SS_EE] += E * E;
    }
};

// compute_forces_complex (scp_sim.c:931-994) at one site, explicitly rounded
// and visited field by field like gauged_site (Phi's neighbours, then Theta's,
// each Theta field finished at once); xm: x(i-1) of the 12 fields, left
// holding x(i)
template <bool SUMS, class V, class Out>
__device__ __forceinline__ void free_site(const V &cv, const V &pv, double (&xm)[12], const StepConsts &k, Out &out,
                                          GaugedSums &sums) {
    double crP[6], crT[6], lap[6];   // curls of Phi and Theta: real part [0..2], imaginary [3..5]
    double eg = 0.0, etg = 0.0;
    // one real field (part 0: real, 3: imaginary) of component a: its sum of
    // neighbours, and its central differences (undivided) into the curl
    auto field = [&](int f, int a, int part, double *cr, double &esum) -> double {
        const double n[3] = {pv.get(f, 0, 0), cv.get(f, 1, 0), cv.get(f, 0, 1)};
        const double m[3] = {xm[f], cv.get(f, -1, 0), cv.get(f, 0, -1)};
        double l = 0.0;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            l = d == 0 ? radd(n[0], m[0]) : radd(radd(l, n[d]), m[d]);
            if (a != d || SUMS) {
                const double df = rsub(n[d], m[d]);
                if (SUMS) esum += df * df;
                if (a != d) {   // + in curl_{d+2} when a = d+1, - in curl_{d+1} when a = d+2
                    const bool plus = (a == (d + 1) % 3);
                    const int t = plus ? (d + 2) % 3 : (d + 1) % 3;
                    const int other = plus ? (t + 1) % 3 : (t + 2) % 3;
                    if (a < other) cr[part + t] = plus ? df : -df;
                    else cr[part + t] = plus ? radd(cr[part + t], df) : rsub(cr[part + t], df);
                }
            }
        }
        xm[f] = cv.get(f, 0, 0);
        return l;
    };
    auto acc = [&](double x, double l, double t, double cu) {
        return rfma(k.ei, cu, rfma(rfma(-6.0, x, l), k.idx2, rmul(t, x)));
    };
#pragma unroll
    for (int a = 0; a < 3; a++) {
        lap[a] = field(FU + a, a, 0, crP, eg);
        lap[3 + a] = field(FV + a, a, 3, crP, eg);
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const double lu = field(FTU + a, a, 0, crT, etg), lv = field(FTV + a, a, 3, crT, etg);
        const double u = xm[FTU + a], v = xm[FTV + a];
        out.theta(a, u, v, acc(u, lu, -k.mtheta2, crP[a]), acc(v, lv, -k.mtheta2, crP[3 + a]));
    }
    double s[3];
#pragma unroll
    for (int a = 0; a < 3; a++) s[a] = rfma(xm[FU + a], xm[FU + a], rmul(xm[FV + a], xm[FV + a]));
    const double den = rfma(k.kappa, rmul(rmul(s[0], s[1]), s[2]), 1.0);
    const double nV2 = -k.mu / rmul(den, den);   // -2 V'
    out.moduli(s, den);
    double ec = 0.0;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const double t = rfma(nV2, rmul(s[(a + 1) % 3], s[(a + 2) % 3]), -k.m2);
        const double u = xm[FU + a], v = xm[FV + a];
        if (SUMS) ec += u * crT[a] + v * crT[3 + a];
        out.phi(a, u, v, acc(u, lap[a], t, crT[a]), acc(v, lap[3 + a], t, crT[3 + a]));
    }
    if (SUMS) { sums.eg = eg; sums.etg = etg; sums.ec = ec; }
}

// One work item (a tile column over one segment of planes) of one FP64 grid.
// sync and damp are uniform per call; the single-grid kernel passes them as
// constants, the multi-request kernel per request.  Stage stages the planes.
template <int TX, int TY, bool GAUGED, bool FIRST, bool DIAG, class Stage>
__device__ __forceinline__ void step_item(const StepIO<F64> &io, const StepConsts &c, const TileGrid &tg,
                                          const Piece &pc, const bool SYNC, const bool DAMP, Stage &stg,
                                          StepSums *sums = nullptr) {
    const int N = c.N;
    const int tx = stg.tx, ty = stg.ty;
    const int k0 = pc.kt * tg.tw, j0 = pc.jt * tg.th;
    const int i0 = pc.i0, i1 = pc.i1;
    const int k = k0 + tx, j = j0 + ty;
    const int nk = min(k0 + tg.tw, N) - k0, nj = min(j0 + tg.th, N) - j0;   // valid extent of the tile
    const bool act = (tx < nk) && (ty < nj);
    const int oc = j * N + k;                                          // in-plane offset (act only)
    stg.begin(c, k0, j0, nk, nj);

    __syncthreads();   // previous item finished reading the ring
    stg.issue(io, i0 - 1, 0);
    stg.issue(io, i0, 1);
    stg.commit();
    // planes i0+1 .. i0+NS-2, one copy group each
    constexpr int NS = Stage::NSLOT;
#pragma unroll
    for (int q = 1; q <= NS - 2; q++) {
        if (i0 + q <= i1) stg.issue(io, i0 + q, q + 1);
        stg.commit();
    }
    Momenta<GAUGED> w;
    if constexpr (Stage::MOM) {
        stg.issue_mom(i0, 0);   // momenta of the first plane
    } else if (act) {
#pragma unroll
        for (int f = 0; f < (GAUGED ? 15 : 12); f++)
            w.v[f] = ld_early(io.win + f * c.N3 + (long long)i0 * N * N + oc);
    }
    stg.template wait<NS - 2>(0);
    stg.template wait<NS - 2>(1);
    __syncthreads();
    GaugedCarry cy;
    double xm[12];
    if (act) {
        if constexpr (GAUGED) {
            gauged_begin<false, true>(stg.view(0), stg.view(1), FTH, cy);
        } else {
            const auto m = stg.view(0);
#pragma unroll
            for (int f = 0; f < 12; f++) xm[f] = m.get(f, 0, 0);
        }
    }

    for (int i = i0; i < i1; i++) {
        // plane p sits in slot (p - i0 + 1) mod NS; plane i + NS - 1 reuses the slot of i - 1
        const int sc = (i - i0 + 1) % NS, sp = (i - i0 + 2) % NS, sn = (i - i0) % NS;
        stg.template wait<NS - 3>(sp);   // the copies of planes beyond i+1 may stay in flight
        if constexpr (Stage::MOM) stg.wait_mom((i - i0) & 1);
        __syncthreads();
        if (i + NS - 1 <= i1) stg.issue(io, i + NS - 1, sn);
        if constexpr (Stage::MOM) {   // momenta of the next plane, into the slot plane i-1 used
            if (i + 1 < i1) stg.issue_mom(i + 1, (i + 1 - i0) & 1);
        }
        stg.commit();
        if (!act) continue;
        const long long site = (long long)i * N * N + oc;
        if (c.prefetch && i + 1 < i1) {
#pragma unroll
            for (int f = 0; f < (GAUGED ? 15 : 12); f++)
                prefetch_line_l2(io.win + f * c.N3 + site + (long long)N * N);
        }
        SiteUpdate<GAUGED, FIRST, DIAG, Stage> out{io, c, stg, sums, site, (i - i0) & 1, SYNC, DAMP, w,
                                                    i + 1 < i1 ? (long long)N * N : 0};
        if (DAMP && !FIRST) out.dmp = sponge_factor(i, j, k, c.L, c.dx, c.damp_width, c.damp_rate);
        GaugedSums gs;
        if constexpr (GAUGED) gauged_site<DIAG, false, true>(stg.view(sc), stg.view(sp), FTH, cy, GaugedConsts(c), out, gs);
        else free_site<DIAG>(stg.view(sc), stg.view(sp), xm, c, out, gs);
        if (SYNC && out.bad) atomicOr(io.flag, 1);
        if constexpr (DIAG) {
            sums->s[SS_EG] += gs.eg;
            sums->s[SS_ETG] += gs.etg;
            sums->s[SS_EC] += gs.ec;
            const double x = -c.L + i * c.dx, y = -c.L + j * c.dx, z = -c.L + k * c.dx;
            sums->s[SS_CX] += x * out.rho2;
            sums->s[SS_CY] += y * out.rho2;
            sums->s[SS_CZ] += z * out.rho2;
            if (x * x + y * y + z * z <= c.R2) sums->s[SS_QC] += out.rho;
            if constexpr (GAUGED) io.drho[site] = out.rho;
        }
    }
}

// ---------------------------------------------------------------- compensated FP32, one site per thread

template <int TX, int TY, bool GAUGED, bool FIRST>
__device__ __forceinline__ void step_item_c(const StepIO<F32C> &io, const StepConsts &c, const TileGrid &tg,
                                            const Piece &pc, const bool SYNC, const bool DAMP,
                                            CpStage<F32C, TX, TY, GAUGED> &stg) {
    using T = float;
    using LY = StepLayout<F32C, TX, TY, GAUGED>;
    constexpr int NF = LY::NF;
    constexpr int NR = LY::NR;
    const int N = c.N;
    const long long N3 = c.N3;
    const int tx = stg.tx, ty = stg.ty;
    auto XS = [&](int slot, int f, int r, int col) -> T { return stg.view(slot).get(f, r - ty - 1, col - tx - 1); };
    const T hdt = (T)c.hdt, idx1 = (T)c.idx1, idx2 = (T)c.idx2;
    const float dt_lo = (float)(c.dt - (double)(float)c.dt);
    const float hdt_lo = (float)(c.hdt - (double)(float)c.hdt);

    {
        const int k0 = pc.kt * tg.tw, j0 = pc.jt * tg.th;
        const int i0 = pc.i0, i1 = pc.i1;
        const int k = k0 + tx, j = j0 + ty;
        const int nk = min(k0 + tg.tw, N) - k0, nj = min(j0 + tg.th, N) - j0;   // valid extent of the tile
        const bool act = (tx < nk) && (ty < nj);
        const int oc = j * N + k;                                          // in-plane offset (act only)
        stg.begin(c, k0, j0, nk, nj);
        auto issue_plane = [&](int p, int slot) { stg.issue(io, p, slot); };

        // sine of the plaquette angle th_a(y) + th_b(y+a) - th_a(y+b) - th_b(y) of plane
        // (a,b) = (0,1) (1,2) (2,0) [q = 0, 1, 2] at ring position (r, col) of slot sc,
        // the next plane in slot sp (compute_forces_complex_gauge pass B, scp_sim.c:1090-1109)
        auto plaq_sin = [&](int q, int sc, int sp, int r, int col) -> T {
            const int a = q, b = (q + 1) % 3;
            // th_b(y+a): the next plane for a = 0, else the neighbour row (a = 1) or column (a = 2)
            const int sa = (a == 0) ? sp : sc, ra = r + (a == 1 ? 1 : 0), ca = col + (a == 2 ? 1 : 0);
            const int sb = (b == 0) ? sp : sc, rb = r + (b == 1 ? 1 : 0), cb = col + (b == 2 ? 1 : 0);
            const T tay = XS(sc, FTH + a, r, col), tby = XS(sc, FTH + b, r, col);
            const T tbya = XS(sa, FTH + b, ra, ca), tayb = XS(sb, FTH + a, rb, cb);
            // hi differences plus lo differences
            const T hi = (tay - tayb) + (tbya - tby);
            const T lo = (XS(sc, NF + a, r, col) - XS(sb, NF + a, rb, cb)) +
                         (XS(sa, NF + b, ra, ca) - XS(sc, NF + b, r, col));
            return sin_bounded(hi + lo);
        };

        __syncthreads();   // previous item finished reading the ring
        issue_plane(i0 - 1, 0);
        issue_plane(i0, 1);
        stg.commit();
        stg.template wait<0>(0);
        stg.template wait<0>(1);
        __syncthreads();
        T xm[12];          // x(i-1) at this thread's site, matter fields
#pragma unroll
        for (int f = 0; f < 12; f++) xm[f] = act ? XS(0, f, ty + 1, tx + 1) : T(0);
        // link 0 and the (0,1), (2,0) plaquettes at x - i (carried from plane to plane)
        T c0m = T(1), s0m = T(0), P0m = T(0), P2m = T(0);
        if (GAUGED && act) {
            sincos_bounded(XS(0, FTH + 0, ty + 1, tx + 1), &s0m, &c0m);
            P0m = plaq_sin(0, 0, 1, ty + 1, tx + 1);
            P2m = plaq_sin(2, 0, 1, ty + 1, tx + 1);
        }
        issue_plane(i0 + 1, 2);
        stg.commit();

        for (int i = i0; i < i1; i++) {
            // plane p sits in slot (p - i0 + 1) mod 3; plane i + 2 reuses the slot of i - 1
            const int sc = (i - i0 + 1) % 3, sp = (i - i0 + 2) % 3, sn = (i - i0) % 3;
            stg.template wait<0>(sp);
            __syncthreads();
            if (i + 2 <= i1) issue_plane(i + 2, sn);
            stg.commit();
            const long long site = (long long)i * N * N + oc;
            if (c.prefetch && act && i + 1 < i1) {
#pragma unroll
                for (int f = 0; f < NF; f++) prefetch_line_l2(io.win + f * N3 + site + (long long)N * N);
            }
            // momenta and low parts of this plane, kept at its top: where the
            // compiler may place them it sinks some to their use (without links
            // 113^3 119 us a step against 115, 151^3 233 against 224; with links
            // 95^3 82.6 against 79.1, 111^3 156 against 147; only 97^3, 105
            // against 109, and 127^3, 198 against 199, are the better for it)
            T w[NF];
            uint16_t lo[12];
            if (act) {
#pragma unroll
                for (int f = 0; f < NF; f++) w[f] = ld_early(io.win + f * N3 + site);
#pragma unroll
                for (int f = 0; f < 12; f++) lo[f] = ld_early(io.loin + f * N3 + site);
            }
            if (!act) continue;
            T acc[12];
            T K[3] = {T(0), T(0), T(0)};
            T ctr[NF];
#pragma unroll
            for (int f = 0; f < NF; f++) ctr[f] = XS(sc, f, ty + 1, tx + 1);
            // potential pieces (scp_sim.c:946-958)
            const T s0 = ctr[FU + 0] * ctr[FU + 0] + ctr[FV + 0] * ctr[FV + 0];
            const T s1 = ctr[FU + 1] * ctr[FU + 1] + ctr[FV + 1] * ctr[FV + 1];
            const T s2 = ctr[FU + 2] * ctr[FU + 2] + ctr[FV + 2] * ctr[FV + 2];
            const T sp3 = s0 * s1 * s2;
            const T den = T(1) + (T)c.kappa * sp3;
            const T Vp = T(0.5) * (T)c.mu / (den * den);
            const T rest[3] = {s1 * s2, s0 * s2, s0 * s1};
            const T m2 = (T)c.m2, mt2 = (T)c.mtheta2, eta = (T)c.eta;

            if (!GAUGED) {
                // compute_forces_complex, scp_sim.c:931-994
                auto nb = [&](int f, int which) -> T {   // 0 ip 1 im 2 jp 3 jm 4 kp 5 km
                    switch (which) {
                        case 0: return XS(sp, f, ty + 1, tx + 1);
                        case 1: return xm[f];
                        case 2: return XS(sc, f, ty + 2, tx + 1);
                        case 3: return XS(sc, f, ty, tx + 1);
                        case 4: return XS(sc, f, ty + 1, tx + 2);
                        default: return XS(sc, f, ty + 1, tx);
                    }
                };
                auto lap = [&](int f) -> T {   // neighbour differences: no cancellation against 6*centre
                    const T x0 = ctr[f];
                    return ((nb(f, 0) - x0) + (nb(f, 1) - x0) + (nb(f, 2) - x0) + (nb(f, 3) - x0) +
                            (nb(f, 4) - x0) + (nb(f, 5) - x0)) * idx2;
                };
                auto curl = [&](int g0, int a) -> T {
                    if (a == 0) return (nb(g0 + 2, 2) - nb(g0 + 2, 3) - nb(g0 + 1, 4) + nb(g0 + 1, 5)) * idx1;
                    if (a == 1) return (nb(g0 + 0, 4) - nb(g0 + 0, 5) - nb(g0 + 2, 0) + nb(g0 + 2, 1)) * idx1;
                    return (nb(g0 + 1, 0) - nb(g0 + 1, 1) - nb(g0 + 0, 2) + nb(g0 + 0, 3)) * idx1;
                };
#pragma unroll
                for (int a = 0; a < 3; a++) {
                    T x = ctr[FU + a];
                    acc[FU + a] = lap(FU + a) - m2 * x - T(2) * Vp * x * rest[a] + eta * curl(FTU, a);
                    x = ctr[FV + a];
                    acc[FV + a] = lap(FV + a) - m2 * x - T(2) * Vp * x * rest[a] + eta * curl(FTV, a);
                    x = ctr[FTU + a];
                    acc[FTU + a] = lap(FTU + a) - mt2 * x + eta * curl(FU, a);
                    x = ctr[FTV + a];
                    acc[FTV + a] = lap(FTV + a) - mt2 * x + eta * curl(FV, a);
                }
            } else {
                // compute_forces_complex_gauge pass C, scp_sim.c:1112-1262
                // complex fields q=0..2 Phi_a, q=3..5 Theta_a
                const T fu[6] = {ctr[FU], ctr[FU + 1], ctr[FU + 2], ctr[FTU], ctr[FTU + 1], ctr[FTU + 2]};
                const T fv[6] = {ctr[FV], ctr[FV + 1], ctr[FV + 2], ctr[FTV], ctr[FTV + 1], ctr[FTV + 2]};
                T lapU[6], lapV[6];
                // covariant curls, built as the directions come in: component a is
                // D[d = a+1][field a+2] - D[d = a+2][field a+1] (indices mod 3) of the
                // central differences D = (transported(x+d) - transported(x-d))/(2dx);
                // one subtraction either way round, as the reference forms it
                T crT[3], ciT[3], crP[3], ciP[3];
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    // link d at x (pass A, scp_sim.c:1072-1079) and at x - d
                    T cP, sP, cM, sM;
                    sincos_bounded(ctr[FTH + d], &sP, &cP);
                    if (d == 0) { cM = c0m; sM = s0m; c0m = cP; s0m = sP; }
                    else if (d == 1) sincos_bounded(XS(sc, FTH + 1, ty, tx + 1), &sM, &cM);
                    else sincos_bounded(XS(sc, FTH + 2, ty + 1, tx), &sM, &cM);
                    T TRpP[3], TIpP[3];   // forward transports of Phi
                    T tup[3], tvp[3];     // raw Theta at x+d (current and seagull)
#pragma unroll
                    for (int q = 0; q < 6; q++) {
                        const int fre = q < 3 ? FU + q : FTU + q - 3;
                        const int fim = q < 3 ? FV + q : FTV + q - 3;
                        T up, vp, um, vm;
                        if (d == 0) {
                            up = XS(sp, fre, ty + 1, tx + 1); vp = XS(sp, fim, ty + 1, tx + 1);
                            um = xm[fre]; vm = xm[fim];
                        } else if (d == 1) {
                            up = XS(sc, fre, ty + 2, tx + 1); vp = XS(sc, fim, ty + 2, tx + 1);
                            um = XS(sc, fre, ty, tx + 1);     vm = XS(sc, fim, ty, tx + 1);
                        } else {
                            up = XS(sc, fre, ty + 1, tx + 2); vp = XS(sc, fim, ty + 1, tx + 2);
                            um = XS(sc, fre, ty + 1, tx);     vm = XS(sc, fim, ty + 1, tx);
                        }
                        const T TRp = cP * up - sP * vp, TIp = cP * vp + sP * up;
                        const T TRm = cM * um + sM * vm, TIm = cM * vm - sM * um;
                        const T cu = fu[q], cv = fv[q];   // (transported - centre) differences
                        if (d == 0) { lapU[q] = (TRp - cu) + (TRm - cu); lapV[q] = (TIp - cv) + (TIm - cv); }
                        else { lapU[q] = lapU[q] + (TRp - cu) + (TRm - cu); lapV[q] = lapV[q] + (TIp - cv) + (TIm - cv); }
                        const int qa = q < 3 ? q : q - 3;
                        if (qa != d) {
                            const T DR = (TRp - TRm) * idx1, DI = (TIp - TIm) * idx1;
                            T *cr = q < 3 ? crP : crT, *ci = q < 3 ? ciP : ciT;
                            if (qa == (d + 1) % 3) {            // plus term of a = d + 2
                                const int a = (d + 2) % 3;
                                if (d < (a + 2) % 3) { cr[a] = DR; ci[a] = DI; }
                                else { cr[a] = DR - cr[a]; ci[a] = DI - ci[a]; }
                            } else {                            // minus term of a = d + 1
                                const int a = (d + 1) % 3;
                                if (d < (a + 1) % 3) { cr[a] = DR; ci[a] = DI; }
                                else { cr[a] = cr[a] - DR; ci[a] = ci[a] - DI; }
                            }
                        }
                        if (q < 3) { TRpP[q] = TRp; TIpP[q] = TIp; }
                        else { tup[q - 3] = up; tvp[q - 3] = vp; }
                    }
                    // lattice current J (scp_sim.c:1232-1249); the Theta transports are
                    // recomputed from the cached raw neighbours to keep the live set small
                    T Jg = T(0);
#pragma unroll
                    for (int a = 0; a < 3; a++) {
                        const T TIt = cP * tvp[a] + sP * tup[a];
                        const T TRt = cP * tup[a] - sP * tvp[a];
                        // u*TI - v*TR = u*(TI - v) - v*(TR - u): differences of neighbouring
                        // values instead of a difference of two O(|f|^2) products
                        Jg += fu[a] * (TIpP[a] - fv[a]) - fv[a] * (TRpP[a] - fu[a]);
                        Jg += fu[3 + a] * (TIt - fv[3 + a]) - fv[3 + a] * (TRt - fu[3 + a]);
                    }
                    const int d1 = (d + 1) % 3, d2 = (d + 2) % 3;
                    const T WpR1 = cP * fu[d2] + sP * fv[d2], WpI1 = cP * fv[d2] - sP * fu[d2];
                    const T WpR2 = cP * fu[d1] + sP * fv[d1], WpI2 = cP * fv[d1] - sP * fu[d1];
                    const T T12 = (fu[3 + d1] * TIpP[d2] - fv[3 + d1] * TRpP[d2])
                                + (tup[d1] * WpI1 - tvp[d1] * WpR1);
                    const T T21 = (fu[3 + d2] * TIpP[d1] - fv[3 + d2] * TRpP[d1])
                                + (tup[d2] * WpI2 - tvp[d2] * WpR2);
                    K[d] = (T)c.inva * Jg - T(0.5) * eta * (T12 - T21);   // Jlat; staple added below
                }
                // staples (scp_sim.c:1214-1220)
                const T P0 = plaq_sin(0, sc, sp, ty + 1, tx + 1), P1 = plaq_sin(1, sc, sp, ty + 1, tx + 1);
                const T P2 = plaq_sin(2, sc, sp, ty + 1, tx + 1);
                const T P0jm = plaq_sin(0, sc, sp, ty, tx + 1), P1jm = plaq_sin(1, sc, sp, ty, tx + 1);
                const T P1km = plaq_sin(1, sc, sp, ty + 1, tx), P2km = plaq_sin(2, sc, sp, ty + 1, tx);
                const T st0 = (P0 - P0jm) - (P2 - P2km);
                const T st1 = -(P0 - P0m) + (P1 - P1km);
                const T st2 = (P2 - P2m) - (P1 - P1jm);
                P0m = P0; P2m = P2;   // x - i of the next plane
                const T stp = (T)c.stp, gg = (T)c.g;
                K[0] = stp * st0 + gg * K[0];
                K[1] = stp * st1 + gg * K[1];
                K[2] = stp * st2 + gg * K[2];
#pragma unroll
                for (int a = 0; a < 3; a++) {
                    const T lUP = lapU[a] * idx2, lVP = lapV[a] * idx2;
                    const T lUT = lapU[3 + a] * idx2, lVT = lapV[3 + a] * idx2;
                    acc[FU + a] = lUP - m2 * fu[a] - T(2) * Vp * fu[a] * rest[a] + eta * crT[a];
                    acc[FV + a] = lVP - m2 * fv[a] - T(2) * Vp * fv[a] * rest[a] + eta * ciT[a];
                    acc[FTU + a] = lUT - mt2 * fu[3 + a] + eta * crP[a];
                    acc[FTV + a] = lVT - mt2 * fv[3 + a] + eta * ciP[a];
                }
            }

            // kicks, damping, drift (scp_sim.c:1591-1715, fused)
            T dmp = T(1);
            if (DAMP && !FIRST) {
                const double x = -c.L + i * c.dx, y = -c.L + j * c.dx, z = -c.L + k * c.dx;
                const double r = sqrt(x * x + y * y + z * z);
                const double Rd = c.L - c.damp_width;
                if (r > Rd) {
                    double sc2 = (r - Rd) / c.damp_width;
                    if (sc2 > 1) sc2 = 1;
                    dmp = (T)(1.0 - c.damp_rate * sc2 * sc2);
                }
            }
            bool bad = false;
#pragma unroll
            for (int f = 0; f < 12; f++) {
                T v, wn, xn;
                // kicks with dt and dt/2 as fp32 pairs: the increment h*a is formed
                // first (hi*a + lo*a), then added to the momentum in one rounding --
                // folding lo*a into the momentum first would lose it below half an
                // ulp and run the kick with fp32(dt), a systematic energy drift
                const float ha = fmaf(hdt, acc[f], hdt_lo * acc[f]);
                v = FIRST ? w[f] : w[f] + ha;
                if (DAMP && !FIRST) v *= dmp;
                if (DAMP || FIRST) wn = v + ha;
                else wn = w[f] + fmaf((float)c.dt, acc[f], dt_lo * acc[f]);   // w_n + dt*a, no damping
                // compensated drift (hi, lo) += dt*w_{n+1}
                const float y = fmaf((float)c.dt, wn, fmaf(dt_lo, wn, bf16_to_f(lo[f])));
                float e;
                two_sum(ctr[f], y, &xn, &e);
                io.loout[f * N3 + site] = f_to_bf16(e);
                st_cs(io.xout + f * N3 + site, xn);
                io.wout[f * N3 + site] = wn;
                if (SYNC && !FIRST) {
                    st_cs(io.sout + f * N3 + site, v);
                    bad |= !isfinite(xn) || !isfinite(v);
                }
            }
            if (GAUGED) {
                const T gad = (T)c.gad;
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    T E, Eh, th;
                    const float hK = fmaf(hdt, K[d], hdt_lo * K[d]);
                    E = FIRST ? w[FTH + d] : w[FTH + d] + hK;
                    if (DAMP && !FIRST) E *= dmp;
                    if (DAMP || FIRST) Eh = E + hK;
                    else Eh = w[FTH + d] + fmaf((float)c.dt, K[d], dt_lo * K[d]);
                    const float gad_lo = (float)(c.gad - (double)(float)c.gad);
                    const float y = fmaf(gad, Eh, fmaf(gad_lo, Eh, XS(sc, NR - 3 + d, ty + 1, tx + 1)));
                    float lnew;
                    two_sum(ctr[FTH + d], y, &th, &lnew);
                    if (fabsf(th) > 3.0f) {   // wrap by 2 pi, carried as an fp32 pair
                        const float kq = rintf(th * 0.159154943091895336f);
                        float t1, e1;
                        two_sum(th, -kq * 6.28318548202514648f, &t1, &e1);   // 2 pi (fp32) times |kq| <= 1
                        lnew = lnew + e1 + kq * 1.74845553e-7f;              // 2 pi = 6.2831855f - 1.748e-7
                        two_sum(t1, lnew, &th, &lnew);
                    }
                    io.tloout[d * N3 + site] = lnew;
                    st_cs(io.xout + (FTH + d) * N3 + site, th);
                    io.wout[(FTH + d) * N3 + site] = Eh;
                    if (SYNC && !FIRST) {
                        st_cs(io.sout + (FTH + d) * N3 + site, E);
                        bad |= !isfinite(E) || !isfinite(th);
                    }
                }
            }
            if (SYNC && bad) atomicOr(io.flag, 1);
#pragma unroll
            for (int f = 0; f < 12; f++) xm[f] = ctr[f];
        }
    }
}

// Single grid: persistent CTAs over the grid's work items.
// Resident CTAs per SM the register allocation is sized for.
template <class P, int TX, int TY, bool GAUGED>
struct MinBlocks {
    static constexpr int value = (TX * TY > 128) ? 1 : (P::COMP ? 3 : 2);
};

template <class P, int TX, int TY, bool GAUGED, bool FIRST, class Stage>
__device__ __forceinline__ void step_one(const StepIO<P> &io, const StepConsts &c, const TileGrid &tg, const Piece &pc,
                                         const bool SYNC, const bool DAMP, Stage &stg) {
    if constexpr (P::COMP) step_item_c<TX, TY, GAUGED, FIRST>(io, c, tg, pc, SYNC, DAMP, stg);
    else step_item<TX, TY, GAUGED, FIRST, false>(io, c, tg, pc, SYNC, DAMP, stg);
}

template <class P, int TX, int TY, bool GAUGED, bool FIRST, bool SYNC, bool DAMP>
__global__ void __launch_bounds__(TX * TY, (MinBlocks<P, TX, TY, GAUGED>::value))
step_kernel(StepIO<P> io, StepConsts c, TileGrid tg) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CpStage<P, TX, TY, GAUGED> stg(smem_raw, tg.tw);
    griddep_wait();
    griddep_launch();
    for_each_piece(tg, c.N, [&](const Piece &pc) {
        step_one<P, TX, TY, GAUGED, FIRST>(io, c, tg, pc, SYNC, DAMP, stg);
    });
}

// The synchronous FP64 launch that also sums the first diagnostics pass: the
// sums stay in registers (two CTAs per SM hold them without spills) and are
// folded to one partial per CTA at the end, the ring serving as scratch.
template <int TX, int TY, bool GAUGED, bool DAMP>
__global__ void __launch_bounds__(TX * TY, (MinBlocks<F64, TX, TY, GAUGED>::value))
step_diag_kernel(StepIO<F64> io, StepConsts c, TileGrid tg) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CpStage<F64, TX, TY, GAUGED> stg(smem_raw, tg.tw);
    griddep_wait();
    griddep_launch();
    StepSums sums;
    sums.clear();
    for_each_piece(tg, c.N, [&](const Piece &pc) {
        step_item<TX, TY, GAUGED, false, true>(io, c, tg, pc, true, DAMP, stg, &sums);
    });
    __syncthreads();
    DiagSums acc;
    step_sums(sums, c, acc);
    block_fold<DS_NSUM, DM_NMAX>(acc.S, acc.M, reinterpret_cast<double *>(smem_raw), io.dpart);
    if (last_block_done(io.dcount))
        fold_rows_block<DS_NSUM, DM_NMAX>(io.dpart, gridDim.x, reinterpret_cast<double *>(smem_raw), io.dfold);
}

// ---------------------------------------------------------------- many grids per launch
//
// The serving loop advances every admitted request by one step per launch.
// Requests live in a device-resident table; request r is active for global
// steps s0 <= s < s1 and its buffers swap roles by the parity of s - s0.
// Because all of that is derived from the step counter in the table, the
// launches can be captured once in a CUDA graph and replayed while requests
// come and go: the host only rewrites the table between replays.  These
// launches never store the synchronous momenta: a request's final step (the
// one that does) runs through the single-grid kernel when it retires.  All
// requests of one launch share the damping mode (a template parameter).

constexpr int kMaxReq = 256;

template <class P>
struct ReqSlot {
    StepIO<P> io[2];      // io[p]: the step taken at parity p
    StepConsts c;
    TileGrid tg;
    int item0;            // first global work item of this request
    int pad;
    long long s0, s1;     // active global steps [s0, s1)
};

template <class P>
struct ReqTable {
    int nreq;
    int nitems;
    long long step;       // global step of launch k = 0 of the current replay
    ReqSlot<P> r[kMaxReq];
};

// last request of the table whose first item is <= item
template <class P>
__device__ __forceinline__ int req_of_item(const ReqTable<P> *tab, int nreq, int item) {
    int lo = 0, hi = nreq - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (tab->r[mid].item0 <= item) lo = mid; else hi = mid - 1;
    }
    return lo;
}

template <class P, int TX, int TY, bool GAUGED, bool DAMP>
__global__ void __launch_bounds__(TX * TY, (MinBlocks<P, TX, TY, GAUGED>::value))
step_multi_kernel(const ReqTable<P> *tab, int k) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int nitems = tab->nitems, nreq = tab->nreq;
    const long long s = tab->step + k;
    for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
        const ReqSlot<P> &q = tab->r[req_of_item(tab, nreq, item)];
        if (s < q.s0 || s >= q.s1) continue;       // uniform over the CTA
        // the request's arguments in registers: the table is global memory the
        // stores of the step could alias, so reading it in place reloads it
        const StepIO<P> io = q.io[(int)((s - q.s0) & 1)];
        const StepConsts c = q.c;
        const TileGrid tg = q.tg;
        CpStage<P, TX, TY, GAUGED> stg(smem_raw, tg.tw);
        step_one<P, TX, TY, GAUGED, false>(io, c, tg, piece_of_item(tg, item - q.item0, c.N), false, DAMP, stg);
    }
}

}  // namespace scp
