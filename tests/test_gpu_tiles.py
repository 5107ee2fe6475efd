"""Edges of the work plans: fitted tiles, site pairs, the plane walkers, the
real mode's fused terms, the packed frames and the diagnostics of compensated
states, at the grid edges where a tile, a row or a launch mode changes."""
import ctypes
import dataclasses
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle
from scp_b200 import PREC_FP32C, native, seeds
from scp_b200.api import DTYPE_F16, DTYPE_F32, DTYPE_F64, Simulation, pinned_empty

pytestmark = pytest.mark.gpu


def rel(a, b):
    nb = np.linalg.norm(b)
    return np.linalg.norm(a - b) / nb if nb > 0 else np.linalg.norm(a - b)


def _frame(params, cols, calls=(1, 3)):
    with Simulation(params, cols) as sim:
        for n in calls:
            sim.step(n)
        return sim.snapshot()


# 16: one 16-site column; 17, 33, 97: odd rows; 48, 80: 16-site rows; 79, 80:
# 128- and 256-site tiles of the gauged step; 112, 113: dependent and ordinary launches
@pytest.mark.parametrize("N", [5, 16, 17, 33, 48, 79, 80, 97, 112, 113])
@pytest.mark.parametrize("gauged", [True, False])
def test_fitted_tiles_give_the_fixed_tile_bits(gpu, N, gauged):
    """Every operation of the FP64 step is explicitly rounded, so a tile shape
    and a launch mode change nothing."""
    st = seeds.small_state(N, gauged, seed=N)
    fixed = dataclasses.replace(st.params, tile_variant=1)
    for a, b in zip(_frame(st.params, st.cols()), _frame(fixed, st.cols())):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("N", [12, 34, 40, 50, 80, 84])   # 40, 80, 84: 40 x 6 tiles
@pytest.mark.parametrize("gauged", [True, False])
def test_pair_tiles_give_the_fixed_tile_bits(gpu, N, gauged):
    st = seeds.small_state(N, gauged, seed=N, precision=PREC_FP32C)
    fixed = dataclasses.replace(st.params, tile_variant=2)
    for a, b in zip(_frame(st.params, st.cols()), _frame(fixed, st.cols())):
        assert np.array_equal(a, b)


BIG_LINKS = {"gauged": {}, "sponge": dict(bc_type=0, damp_width=3.0, damp_rate=0.01),
             "higgs": dict(higgs_v=1.0, higgs_rvoid=2.0)}


@pytest.mark.parametrize("case", sorted(BIG_LINKS))
@pytest.mark.parametrize("N", [17, 34])   # odd rows; an even edge in one 32-site and one 2-site column
def test_large_angles_match_oracle(gpu, case, N):
    """Link angles over the whole of (-pi, pi], where the sines and cosines take
    their range reduction (it is a branch), 6 steps against the checker: within
    the bound the gauged step keeps over 12 steps."""
    st = seeds.small_state(N, True, seed=N + 3, **BIG_LINKS[case])
    rng = np.random.default_rng(N)
    for ax in "xyz":
        st["th_" + ax][:] = rng.uniform(-np.pi, np.pi, st["th_" + ax].shape)
    o = oracle.Oracle(st.params, st.cols())
    o.step(6)
    for c, (a, b) in enumerate(zip(_frame(st.params, st.cols(), (1, 5)), o.cols())):
        assert rel(a, b) <= 1e-11, c


@pytest.mark.parametrize("q", [(0.0, 1.0, -1.0), (0.5, -2.0, 1.0)])
@pytest.mark.parametrize("N,lock", [(17, 1), (34, 1), (34, 0)])
def test_fabrics_match_oracle(gpu, N, lock, q):
    st = seeds.mf_state(N, seed=N, shift=1.0, mf_lock_CQ=lock, q_C=q[0], q_Q=q[1], q_L=q[2])
    o = oracle.Oracle(st.params, st.cols())
    o.step(6)
    for c, (a, b) in enumerate(zip(_frame(st.params, st.cols(), (1, 5)), o.cols())):
        assert rel(a, b) <= 1e-11, c


TERMS = {"strain": dict(alpha_cs=0.2), "hardening": dict(beta_h=0.3), "mode 3": dict(mode=3, kappa_h=0.01),
         "all": dict(mode=1, alpha_cs=0.2, beta_h=0.3, kappa_h=0.01, bc_type=0, damp_width=2.0, damp_rate=0.02)}


@pytest.mark.parametrize("terms", sorted(TERMS))
@pytest.mark.parametrize("N", [5, 13, 33, 40])
def test_real_terms_match_oracle(gpu, terms, N):
    """One, several and partial tiles; the two-site halo wraps on N = 5."""
    st = seeds.real_state(N, seed=N, **TERMS[terms])
    o = oracle.Oracle(st.params, st.cols())
    o.step(8)
    whole = _frame(st.params, st.cols(), (8,))
    for c, (a, b) in enumerate(zip(whole, o.cols())):
        assert rel(a, b) <= 1e-11, c
    for a, b in zip(whole, _frame(st.params, st.cols(), (1, 3, 4))):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("N", [17, 24, 34])
@pytest.mark.parametrize("kw", [dict(gauged=True), dict(gauged=False), dict(gauged=True, g_gauge=0.0),
                                dict(gauged=True, bc_type=0, damp_width=3.0, damp_rate=0.01)])
def test_compensated_diagnostics_match_the_columns(gpu, N, kw):
    """FP32C diagnostics against the allocation-free ones on the state's own
    FP64 columns (hi + lo is exact in a double): the same FP64 terms in another
    order.  Charges and the Gauss residual cancel, so they get a floor."""
    import torch

    kw = dict(kw)
    st = seeds.small_state(N, kw.pop("gauged"), seed=N + 9, precision=PREC_FP32C, **kw)
    with Simulation(st.params, st.cols()) as sim:
        sim.step(5)
        have = sim.diag_vector()
        cols = sim.snapshot()
        g_off = sim.info().G_offset
    dev = [torch.from_numpy(c).to("cuda:0") for c in cols]
    torch.cuda.synchronize()
    p = dataclasses.replace(st.params, precision=0).to_c()
    out = native.DiagOut()
    arr = (ctypes.c_void_p * len(dev))(*[d.data_ptr() for d in dev])
    native.check(native.lib().scp_gpu_diag_noalloc(ctypes.byref(p), arr, g_off, None, ctypes.byref(out)))
    want = np.array(out.v[:31])
    for s in range(31):
        tol = 1e-9 * max(abs(want[s]), 1.0) if s in (7, 13, 14, 15, 19, 24, 25, 27, 28, 29, 30) else 1e-11 * abs(want[s])
        assert abs(have[s] - want[s]) <= tol, (s, have[s], want[s])


@pytest.mark.parametrize("dtype,npd", [(DTYPE_F64, np.float64), (DTYPE_F32, np.float32), (DTYPE_F16, np.uint16)])
@pytest.mark.parametrize("precision", [0, PREC_FP32C])
def test_frames_into_any_columns(gpu, precision, dtype, npd):
    """Synchronous and asynchronous frames into columns of one page-locked
    block (merged copies), of the block in reverse order, of two blocks, and
    of pageable memory are the same."""
    st = seeds.small_state(18, True, seed=4, precision=precision)
    n3, nc = 18 ** 3, st.params.snap_ncols
    block, half = pinned_empty(nc * n3, npd), pinned_empty((nc - 7) * n3, npd)
    rows = [block[c * n3:(c + 1) * n3] for c in range(nc)]
    two = rows[:7] + [half[c * n3:(c + 1) * n3] for c in range(nc - 7)]
    with Simulation(st.params, st.cols()) as sim:
        sim.step(3)
        want = [c.copy() for c in sim.snapshot(dtype)]
        for cols in (rows, rows[::-1], two, [np.empty(n3, npd) for _ in range(nc)]):
            for asynchronous in (False, True):
                for c in cols:
                    c[:] = 0
                if asynchronous:
                    sim.snapshot_async(cols, dtype)
                    sim.snapshot_wait()
                else:
                    sim.snapshot(dtype, out=cols)
                for a, b in zip(cols, want):
                    assert np.array_equal(a, b)


AFTER_RESET = """
import ctypes, glob
from scp_b200 import seeds
from scp_b200.api import Simulation
rt = ctypes.CDLL(glob.glob("/usr/local/cuda/lib64/libcudart.so*")[0])
st = seeds.small_state(24, True, seed=3)
got = []
for _ in range(2):
    with Simulation(st.params, st.cols()) as sim:
        sim.step(3)
        got.append(sim.diag())
    assert rt.cudaDeviceReset() == 0
assert got[0] == got[1]
"""


def test_diagnostics_after_a_device_reset(gpu):
    """Page-locked result slots die with their context: a handle made after a
    reset takes none of the old ones."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", AFTER_RESET], cwd=root, check=True, timeout=120)
