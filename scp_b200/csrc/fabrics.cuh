// fabrics.cuh -- the gauged stepper with three matter fabrics C, Q, L under
// one shared compact U(1) (the reference's multi-fabric model: per-fabric
// force force_fabric_gauged_accum and its driver compute_forces_complex_
// gauge_mf, sfa/sim/scp_sim.c:1274-1433; the EM charge density em_rho_at,
// :184-197; per-fabric charges compute_mf_charges, :2247-2261).
//
// Physics.  Every fabric is a complex Cosserat multiplet with its own bag
// potential, transported by the charge-q_f links e^{i q_f th}; the field
// kick is the plaquette term plus sum_f g q_f J_f, and the Gauss law uses
// rho_em = sum_f q_f rho_f.  With the C-Q lock Q equals C at every step: the
// reference copies C into Q after each force and kick, so C moves under the
// q_Q force (the Q pass overwrites C's accelerations) while both fabrics add
// their currents, g q_C J_C(C) + g q_Q J_Q(C).  Here Q's arrays are C's.
//
// Structure.  One time step is one walker launch (walk.cuh) per moving fabric:
// it stages the fabric's 12 matter fields and the three link angles, advances
// the fabric's matter by the fused leapfrog, and adds its currents g q J to a
// per-site accumulator; the last fabric's launch takes the sum instead, forms
// the plaquette term from the angles it staged anyway, kicks E and drifts the
// angles.  Positions (two alternating buffers) and momenta hold C with the
// links (15 arrays, the fused step's order), then L (12), then Q (12) when it
// is not locked.
//
// What bounds it: DRAM, 936 B per site with Q locked (432 for C, 504 for L
// with the links) against 864 that no split can avoid; 363 us a step at 128^3
// (0.77 of a plain copy's rate on the 864 B) against 524 with four resident
// planes, momenta loaded at their own plane and a launch of its own for the
// links.
#pragma once
#include "walk.cuh"

namespace scp {

struct FabConsts {
    int N;
    long long N3;
    double L, dx, dV, idx1, idx2, inva, hdt, dt;
    double mu, kappa, m2, mtheta2, eta;
    double g, stp, gad;
    double damp_width, damp_rate;
    double ei, cross, gi;   // eta/(2dx), eta dx/2, and (unused here) g/dx
};

// Forward-transport current of one fabric under links of charge qx, in units
// of 1/dx, cross terms included (the locked pair's C current).
template <class V>
__device__ __forceinline__ void fabric_current(const V &c, const V &p, int fth, double qx, double r0, double (&K)[3]) {
    double ang[3], sn[3], cs[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        ang[d] = rmul(qx, c.get(fth + d, 0, 0));
        K[d] = 0.0;
    }
    sincos_batch<3, true>(ang, sn, cs);
#pragma unroll
    for (int q = 0; q < 6; q++) {
        const int fre = field_re(q), fim = field_im(q), a = q % 3;
        const double u = c.get(fre, 0, 0), v = c.get(fim, 0, 0);
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const double up = d == 0 ? p.get(fre, 0, 0) : c.get(fre, d == 1, d == 2);
            const double vp = d == 0 ? p.get(fim, 0, 0) : c.get(fim, d == 1, d == 2);
            const double fr = rfma(-sn[d], vp, rmul(cs[d], up)), fi = rfma(sn[d], up, rmul(cs[d], vp));
            double gu = u, gv = v;
            if (a != d) {
                const int b = 3 - d - a, o = q < 3 ? 3 + b : b;
                const double r = (a == (d + 1) % 3) ? r0 : -r0;
                gu = rfma(r, c.again(field_re(o)), u);
                gv = rfma(r, c.again(field_im(o)), v);
            }
            K[d] = rfma(gu, fi, K[d]);
            K[d] = rfma(-gv, fr, K[d]);
        }
    }
}

// One fabric's matter step.  The force uses links of charge qf; the current
// g qf J(qf) goes to the accumulator, joined, with SECOND, by g qx J(qx)
// over the same fields (the locked pair's C current), and with ACC added to
// what the fabrics before left there.  With LINKS the launch
// also steps the shared links with the accumulated currents.
template <class MODE, bool SECOND, bool ACC, bool LINKS>
struct FabricPass {
    static_assert(!LINKS || ACC, "the links come with the last fabric");
    static_assert(!SECOND || !ACC, "the locked pair comes first");
    static constexpr int TH = 12;
    static constexpr int NR = 15, CF = LINKS ? 12 : 15;
    static constexpr int NM = LINKS ? 15 : 12;
    static constexpr int MIN_CTAS = 1;
    static constexpr bool HALO_APART = true, CONVERT = false, WIDE = false;

    struct Args {
        const double *src[2];   // this fabric's 12 matter positions; th
        int N;
        FabConsts c;
        double qf, gqf;         // force charge, current weight g qf / dx
        double qx, gqx;         // second current (SECOND)
        LeapIO io;              // matter; E and th (LINKS)
        double *kacc;           // 3 arrays: accumulated currents
    };

    static constexpr int NR_FEW = NR;   // always all of them
    __device__ static __forceinline__ bool few(const Args &) { return false; }
    __device__ static __forceinline__ const double *src(const Args &A, int f, long long n3) {
        return f < 12 ? A.src[0] + f * n3 : A.src[1] + (f - 12) * n3;
    }

    struct State {
        GaugedCarry cy;
        double w[NM];
        double kin[3];          // the accumulated currents, read one plane ahead
    };

    __device__ static __forceinline__ void load(const Args &A, State &st, long long idx) {
#pragma unroll
        for (int f = 0; f < NM; f++) st.w[f] = ld_early(LeapSite<MODE, NM>::at(A.io.win, f, A.c.N3) + idx);
#pragma unroll
        for (int d = 0; d < 3; d++) st.kin[d] = ACC ? ld_early(A.kacc + d * A.c.N3 + idx) : 0.0;
    }
    template <class V>
    __device__ static __forceinline__ void begin(const Args &A, State &st, const V &m, const V &c) {
        gauged_begin<true, LINKS>(m, c, TH, st.cy, A.qf);
    }

    struct Out {
        const Args &A;
        State &st;
        LeapSite<MODE, NM> &leap;
        double (&k0)[3];        // SECOND: J(qf), until J(qx) joins it
        __device__ __forceinline__ void theta(int a, double u, double v, double au, double av) {
            leap.put(FTU + a, u, au, leap.dmp);
            leap.put(FTV + a, v, av, leap.dmp);
        }
        __device__ __forceinline__ void phi(int a, double u, double v, double au, double av) {
            leap.put(FU + a, u, au, leap.dmp);
            leap.put(FV + a, v, av, leap.dmp);
        }
        __device__ __forceinline__ void moduli(const double (&)[3], double) {}
        __device__ __forceinline__ void angles(double, double, double) {}
        // the fabric's current on top of what the others left
        __device__ __forceinline__ double current(int d, double K) {
            if (SECOND) {
                k0[d] = K;
                return K;
            }
            double t = rmul(A.gqf, K);
            if (ACC) t = radd(st.kin[d], t);
            if (ACC) st.kin[d] = ld_early(A.kacc + d * A.c.N3 + leap.site + leap.next);
            if (!LINKS) A.kacc[d * A.c.N3 + leap.site] = t;
            return t;
        }
        __device__ __forceinline__ void link(int d, double th, double K) {
            leap.put_link(FTH + d, th, K, A.c.gad, leap.dmp);
        }
    };

    template <class V>
    __device__ static __forceinline__ void site(const Args &A, State &st, const V &c, const V &p, int i, int j, int k,
                                                long long idx, long long next) {
        const FabConsts &fc = A.c;
        const double dmp = (MODE::DAMP && !MODE::FIRST)
                               ? sponge_factor(i, j, k, fc.L, fc.dx, fc.damp_width, fc.damp_rate) : 1.0;
        LeapSite<MODE, NM> leap{A.io, st.w, fc.N3, idx, next, fc.hdt, fc.dt, dmp};
        double k0[3];
        Out out{A, st, leap, k0};
        GaugedSums none;
        gauged_site<false, true, LINKS>(c, p, TH, st.cy, GaugedConsts(fc), out, none, A.qf);
        if (SECOND) {
            // The current under qx follows the force, behind a fence that keeps
            // the compiler from holding the neighbours it reads in registers
            // meanwhile: ahead of the force it spilled 256 bytes a thread
            // (locked pair with q_C != 0, a step at 128^3 559 us against 378,
            // at 113^3 498 against 381)
            asm volatile("" ::: "memory");
            double kx[3];
            fabric_current(c, p, TH, A.qx, fc.cross, kx);
#pragma unroll
            for (int d = 0; d < 3; d++) A.kacc[d * fc.N3 + idx] = rfma(A.gqx, kx[d], rmul(A.gqf, k0[d]));
        }
        if (MODE::SYNC && leap.bad) atomicOr(A.io.flag, 1);
    }
};

}  // namespace scp
