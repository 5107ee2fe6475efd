"""Handles of different grids made by several threads at once: nothing that a
start-up sets for its own grid may reach another thread's launches."""
import threading

import numpy as np
import pytest

from scp_b200 import seeds
from scp_b200.api import Simulation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edges", [(16, 32, 64, 128), (9, 24, 48, 96)])   # radix-2 lines; direct ones
def test_starts_of_different_grids_at_once(gpu, edges):
    states = [seeds.small_state(N, True, seed=N) for N in edges]
    cols = [st.cols() for st in states]
    want = []
    for st, c in zip(states, cols):
        with Simulation(st.params, c) as sim:
            want.append(sim.diag_vector())
    errors = []

    def start(n, times):
        try:
            for _ in range(times):
                with Simulation(states[n].params, cols[n]) as sim:
                    assert np.array_equal(sim.diag_vector(), want[n])
        except Exception as e:   # reported by the main thread
            errors.append((edges[n], e))

    threads = [threading.Thread(target=start, args=(n, 400 // (n + 1))) for n in range(len(edges)) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[:3]
