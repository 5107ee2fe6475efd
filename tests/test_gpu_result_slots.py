"""More handles at once than one block of page-locked result slots holds: each
keeps its own results, and handles made after them do too."""
import pytest

from scp_b200 import seeds
from scp_b200.api import Simulation

pytestmark = pytest.mark.gpu


def test_many_handles_keep_their_results(gpu):
    states = [seeds.small_state(8, True, seed=s) for s in range(7)]
    want = []
    for st in states:
        with Simulation(st.params, st.cols()) as sim:
            want.append(sim.diag())
    assert len({w["E_total"] for w in want}) == len(states)
    for _ in range(2):
        sims = [Simulation(states[n % 7].params, states[n % 7].cols()) for n in range(270)]
        assert all(sim.diag() == want[n % 7] for n, sim in enumerate(sims))
        assert all(sim.diag() == want[n % 7] for n, sim in reversed(list(enumerate(sims))))
        for sim in sims[::2] + sims[1::2]:
            sim.close()
