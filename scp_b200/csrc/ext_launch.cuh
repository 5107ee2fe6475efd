// ext_launch.cuh -- host-side launchers of the extension steppers' kernels
// (higgs_u1.cuh in kern_higgs.cu, fabrics.cuh in kern_fabric.cu, real6.cuh in
// kern_real.cu: each compiles in its own nvcc process).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include "common.cuh"

namespace scp {

struct HuConsts;
struct FabConsts;
struct R6Consts;

// Launch geometry of one such kernel: tile shape, work items, CTAs.
struct ExtPlan {
    int tx = 0, ty = 0;
    TileGrid tg{};
    int grid = 0;
    size_t smem = 0;
};

// Higgs condensate and / or second gauge: positions and momenta are NR
// consecutive N^3 arrays (matter, th, [th2], [H]; matter, E, [E2], [dH/dt]).
struct HuIO {
    const double *x;      // x_{n+1}
    double *xout;         // x_{n+2}
    const double *win;    // w_n, or v_0 on the first launch
    double *wout, *sout;
    int *flag;
    int first, sync, damp;
};
int hu_plan(bool higgs, bool g2, int N, int nsm, ExtPlan *plan);
cudaError_t hu_step(bool higgs, bool g2, const ExtPlan &plan, const HuConsts &c, const HuIO &io, cudaStream_t st);

// One fabric's matter step, with the shared links' step in the last one.
// Array groups: [0] the fabric's 12 matter arrays, [1] the links (th; E).
struct FabIO {
    const double *src[2];   // positions x_{n+1}
    double *xout[2];
    const double *win[2];
    double *wout[2], *sout[2];
    double *kacc;           // 3 arrays of accumulated currents
    int *flag;
    double qf, gqf;         // force charge and current weight g qf / dx
    double qx, gqx;         // second current over the same fields (second != 0)
    int first, sync, damp, accumulate, second, links;
};
int fabric_plan(int N, int nsm, ExtPlan *plan);
cudaError_t fabric_step(const ExtPlan &plan, const FabConsts &c, const FabIO &io, cudaStream_t st);

// Real mode with the optional terms: positions / momenta are 6 arrays (phi,
// theta); aux: the strain or hardening term is on.
struct R6IO {
    const double *x;
    double *xout;
    const double *win;
    double *wout, *sout;
    int *flag;
    int first, sync, damp;
};
int r6_plan(bool aux, int N, int nsm, ExtPlan *plan);
cudaError_t r6_step(bool aux, const ExtPlan &plan, const R6Consts &c, const R6IO &io, cudaStream_t st);

// First diagnostics reduction on the plane walker (diag_walk.cuh).
struct DiagWalkArgs;
int diag_walk_plan(bool gauged, bool comp, int N, int nsm, ExtPlan *plan);
cudaError_t diag_walk(bool gauged, bool comp, const ExtPlan &plan, const DiagWalkArgs &a, cudaStream_t st);

}  // namespace scp
