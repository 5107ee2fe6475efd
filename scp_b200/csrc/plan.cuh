// plan.cuh -- host-side work plans of the plane-ring steppers: the tile shape
// that suits a grid edge, and its cut into work items.
#pragma once
#include "common.cuh"

namespace scp {

// Launch a step kernel of a grid of edge N; up to 112^3 as a programmatic
// dependent of the launch before it on the stream: its CTAs take free slots and
// set up while that launch drains, which hides the launch gap (gauged 32^3 6.7
// against 8.2 us a step).  Never slower up to there on any stepper: gauged 5 %
// at 64^3, 1 % at 96^3 and 112^3; without links 14, 2 and 2; FP32C 12 to 17, 3
// to 4 and 2 to 4; Higgs and second gauge 5, 2 and 1; three fabrics 7, 2 and 1;
// real mode with its terms 10, 3 and 3.  From 128^3 it depends on the stepper:
// FP64 with links, without, and three fabrics lose 1 %, FP32C and the real mode
// gain 1 to 2.
constexpr int kDependentMaxN = 112;
template <class... P, class... A>
inline cudaError_t launch_step_kernel(void (*fn)(P...), int N, int grid, int threads, size_t smem, cudaStream_t st,
                                      const A &...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = N <= kDependentMaxN ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, fn, P(args)...);
}

// Cut a grid of edge N into tiles of tw x th sites and segments along i, for
// `slots` resident CTAs: the segment length minimises (waves x planes per
// item), planes per item counting the two halo planes a segment re-reads.
// All CTAs start their items on the same plane and walk i in step, so
// neighbouring columns read each other's halo rows while they are in L2.
// (Equal shares of all (column, plane) pairs, which leave no slot idle, were
// measured slower: neighbours drift apart in i and the halo rows come from
// DRAM again, 837 against 470 MB read per 128^3 step.)
inline void plan_tiles(int N, int tw, int th, int slots, TileGrid *out, int *grid) {
    TileGrid tg;
    tg.tw = tw;
    tg.th = th;
    tg.ntx = (N + tw - 1) / tw;
    tg.nty = (N + th - 1) / th;
    const int ntiles = tg.ntx * tg.nty;
    double best = 1e300;
    int best_nseg = 1;
    for (int ns = 1; ns <= N; ns++) {
        const int seg = (N + ns - 1) / ns;
        if (ns > 1 && (N + seg - 1) / seg != ns) continue;   // the same cut as a smaller ns
        const long long waves = ((long long)ntiles * ns + slots - 1) / slots;
        const double cost = (double)waves * (seg + 2);
        if (cost < best - 1e-9) { best = cost; best_nseg = ns; }
    }
    tg.seg = (N + best_nseg - 1) / best_nseg;
    tg.nseg = (N + tg.seg - 1) / tg.seg;
    tg.nitems = ntiles * tg.nseg;
    *out = tg;
    *grid = tg.nitems < slots ? tg.nitems : slots;
}

// Tile of the one-site cp.async kernels for a grid of edge N: up to nt sites
// whose staged rows (halo included) fit `area` ring elements, least
// (padded sites) x (cost of the width).  Rows of 32 sites move whole 128-byte
// lines: width 32 costs 1.  Gauged FP64 measured against it: 16-site rows
// 192 against 184 us at 128^3 (counted 1.08), rows that start inside a line
// 362 against 320 us at 150^3 with 7 % fewer padded sites (1.22; 1.12 where an
// odd N leaves every row unaligned anyway).  So 32-site rows stay except where
// they pad: 16 x 16 takes 54 us at 80^3 against 62, 25 x 10 takes 107 us at
// 97^3 (whose fourth column of 32-site tiles holds one site) against 123.
// FP32C with one site a thread (odd N) pays more for leaving 32-site rows, which
// are one line: with the sponge 27 x 4 tiles 59 against 56 us at 81^3, 22 x 5 76
// against 69 at 85^3 and 19 x 6 168 against 155 at 113^3 with 16, 11 and 12 %
// fewer padded sites, 17 x 7 106 against 111 at 97^3 (no sponge) with 22 %
// fewer; 16 x 8 has no advantage there (52 against 46 us of 25 x 5 at 73^3).
// All counted 1.25.
// more: a second limit, for fields staged further out (or rows of more columns).
struct WiderStage {
    int cols = 0, rows = 0;   // staged beyond the tile's (w + 2) x (h + 2)
    int area = 1 << 30;       // ring elements of one such field
};
inline void fit_tile(int N, int nt, int area, int *tw, int *th, const WiderStage &more = {}, bool fp32 = false) {
    double best = 1e300;
    for (int w = 32; w >= 16; w--) {
        int h = nt / w;
        while (h > 1 && ((w + 2) * (h + 2) > area || (w + 2 + more.cols) * (h + 2 + more.rows) > more.area)) h--;
        const double pad = (double)((N + w - 1) / w) * w * ((N + h - 1) / h) * h;
        const double cost = pad * (w == 32 ? 1.0 : fp32 ? 1.25 : w == 16 ? 1.08 : (N & 1) ? 1.12 : 1.22);
        if (cost < best - 1e-9) { best = cost; *tw = w; *th = h; }
    }
}

// Tile of the two-site FP32C kernels (even edges): 32 x 8, or 40 x 6 where it
// pads enough less (rows of 160 bytes start inside lines: 185 against 144 us
// at 128^3 with 0.78 of the threads on sites, 578 against 618 us at 200^3
// with 0.98 against 0.89).
inline void fit_pair_tile(int N, int *tw, int *th) {
    auto pad = [&](int w, int h) { return (double)((N + w - 1) / w) * w * ((N + h - 1) / h) * h; };
    const bool wide = N >= 40 && 1.07 * pad(40, 6) < pad(32, 8);
    *tw = wide ? 40 : 32;
    *th = wide ? 6 : 8;
}

}  // namespace scp
