"""Work plans on the CPU (scp_b200/csrc/plan.cuh and the layouts of the step
kernels and walkers): for every edge up to 700 and some beyond, a tile has no
more sites than the CTA has threads, its staged rows fit the ring field that
the kernel addresses, its halo copies are no more than the threads take, and
the work items cover every plane of every column once.  The walkers' tiles are
checked for other CTA shapes than the compiled one too."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "step2.cuh"
#include "higgs_u1.cuh"
#include "fabrics.cuh"
#include "real6.cuh"
#include "walk_launch.cuh"
using namespace scp;
static int bad = 0;
#define REQUIRE(x, ...) do { if (!(x)) { std::printf("%s: ", #x); std::printf(__VA_ARGS__); std::puts(""); bad++; } } while (0)

static void covers(int N, int tw, int th, int slots) {
    TileGrid g;
    int grid = 0;
    plan_tiles(N, tw, th, slots, &g, &grid);
    REQUIRE(grid >= 1 && grid <= slots && grid <= g.nitems, "N %d grid %d", N, grid);
    REQUIRE(g.ntx * tw >= N && (g.ntx - 1) * tw < N && g.nty * th >= N && (g.nty - 1) * th < N, "N %d %dx%d", N, tw, th);
    std::vector<int> seen(N, 0);
    for (int s = 0; s < g.nseg; s++)
        for (int i = s * g.seg; i < s * g.seg + g.seg && i < N; i++) seen[i]++;
    for (int i = 0; i < N; i++) REQUIRE(seen[i] == 1, "N %d plane %d", N, i);
    REQUIRE(g.nitems == g.ntx * g.nty * g.nseg, "N %d", N);
}
template <class P, int TX, int TY, bool G>
void one_site(int N, bool fp32) {
    using LY = StepLayout<P, TX, TY, G>;
    int w = TX, h = TY;
    fit_tile(N, TX * TY, LY::PX * LY::PY, &w, &h, {}, fp32);
    REQUIRE(w * h <= LY::NT && (w + 2) * (h + 2) <= LY::PX * LY::PY, "N %d %dx%d", N, w, h);
    REQUIRE(2 * w + 2 * h + 2 <= LY::HPT * LY::NT, "N %d %dx%d halo", N, w, h);
    covers(N, w, h, 296);
}
template <bool G>
void pairs(int N) {
    using LY = Step2Layout<32, 8, G>;
    int w = 32, h = 8;
    fit_pair_tile(N, &w, &h);
    REQUIRE(w % 2 == 0 && w / 2 * h <= LY::NT && (w + 4) * (h + 2) <= LY::FS, "N %d %dx%d", N, w, h);
    REQUIRE(w + 2 * h + 2 <= LY::HPT * LY::NT, "N %d %dx%d halo", N, w, h);
    covers(N, w, h, 296);
}
template <class M, int X, int Y>
void walker(int N) {
    using LY = WalkLayout<M, X, Y>;
    int w, h;
    walk_tile<LY>(N, &w, &h);
    REQUIRE(w * h <= LY::NT && (w + 2 * LY::OFF) * (h + 2) <= LY::FS, "N %d %dx%d of %dx%d", N, w, h, X, Y);
    REQUIRE(2 * w + 2 * h + 2 <= LY::NT, "N %d %dx%d halo", N, w, h);
    if (M::WIDE && w % 2 == 0)   // 16-byte chunks of all rows, then the columns and corners
        REQUIRE(w / 2 * (h + 2) + 2 * h + 2 <= LY::NT, "N %d %dx%d chunks", N, w, h);
    covers(N, w, h, 148);
}
template <bool AUX>
void real(int N) {
    using LY = R6Layout<AUX, 32, 12>;
    int w = 32, h = 12;
    fit_tile(N, LY::NT, LY::TFS, &w, &h, {2 * (LY::H - 1), 2 * (LY::H - 1), LY::PFS});
    REQUIRE(w * h <= LY::NT && (w + 2) * (h + 2) <= LY::TFS && (w + 2 * LY::H) * (h + 2 * LY::H) <= LY::PFS, "N %d", N);
    REQUIRE((w + 2 * LY::H) * (h + 2 * LY::H) <= LY::CP * LY::NT && (w + 2) * (h + 2) <= LY::CT * LY::NT, "N %d", N);
    covers(N, w, h, 148);
}
int main() {
    using Mode = StepMode<false, false, false>;
    using Wide = HiggsU1<Mode, true, true>;
    using Narrow = FabricPass<Mode, false, true, true>;
    std::vector<int> edges;
    for (int N = 4; N <= 700; N++) edges.push_back(N);
    for (int N : {799, 1000, 1023, 1024, 1025, 1625, 2047, 2048}) edges.push_back(N);
    for (int N : edges) {
        one_site<F64, 32, 4, true>(N, false);
        one_site<F64, 32, 8, true>(N, false);
        one_site<F64, 32, 4, false>(N, false);
        one_site<F32C, 32, 4, true>(N, true);
        one_site<F32C, 32, 4, false>(N, true);
        if (N % 2 == 0) { pairs<true>(N); pairs<false>(N); }
        walker<Wide, 32, 8>(N);
        walker<Narrow, 32, 8>(N);
        walker<Wide, 32, 12>(N);    // shapes whose fitted tiles would leave a ring sized for rows alone
        walker<Wide, 32, 16>(N);
        walker<Narrow, 32, 12>(N);
        real<true>(N);
        real<false>(N);
    }
    std::puts(bad ? "bad" : "ok");
    return bad != 0;
}
"""


@pytest.mark.skipif(not shutil.which(NVCC), reason="needs nvcc (host compilation of the kernel headers)")
def test_tiles_fit_their_rings(tmp_path):
    src, exe = tmp_path / "plans.cu", tmp_path / "plans"
    src.write_text(PROGRAM)
    subprocess.run([NVCC, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-I",
                    os.path.join(ROOT, "scp_b200", "csrc"), "-I", os.path.join(ROOT, "include"), "-o", str(exe), str(src)],
                   check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout[-2000:]
