"""Fitted tiles whose last column or row is partial: the tile that a grid edge
gets differs from the fixed shape it is compared with, which the test asserts,
and every site is the same to the last bit."""
import dataclasses

import numpy as np
import pytest

from scp_b200 import PREC_FP32C, seeds
from scp_b200.api import Simulation

pytestmark = pytest.mark.gpu


def _run(params, cols):
    with Simulation(params, cols) as sim:
        info = sim.info()
        sim.step(1)
        sim.step(3)
        return (info.tile_x, info.tile_y), sim.snapshot()


def _compare(st, variant):
    tile, cols = _run(st.params, st.cols())
    fixed_tile, fixed = _run(dataclasses.replace(st.params, tile_variant=variant), st.cols())
    assert tile != fixed_tile, tile
    for a, b in zip(cols, fixed):
        assert np.array_equal(a, b)
    return tile


# 40 x 6 pair tiles whose last column along k holds 26, 30, 34, 36 and 26 sites,
# all but the first with part rows along j too
@pytest.mark.parametrize("N", [66, 70, 74, 76, 106])
@pytest.mark.parametrize("gauged", [True, False])
def test_ragged_pair_tiles(gpu, N, gauged):
    st = seeds.small_state(N, gauged, seed=N, precision=PREC_FP32C)
    assert _compare(st, 2) == (40, 6) and N % 40


# one-site tiles of 128 sites, and of 256 from 80^3 with links (27 x 9 at 81,
# which divides the edge; the others leave part columns or rows)
@pytest.mark.parametrize("precision,N", [(0, 17), (0, 35), (0, 49), (0, 81), (0, 97), (0, 99), (PREC_FP32C, 17),
                                         (PREC_FP32C, 35), (PREC_FP32C, 99)])
@pytest.mark.parametrize("gauged", [True, False])
def test_ragged_fitted_tiles(gpu, precision, N, gauged):
    st = seeds.small_state(N, gauged, seed=N, precision=precision)
    w, h = _compare(st, 1)
    assert N % w or N % h or N == 81
