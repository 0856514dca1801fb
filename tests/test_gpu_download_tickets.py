"""Tickets of asynchronous downloads: waited for late, out of order, and after
more downloads than the library keeps events for."""
import numpy as np
import pytest

from fluid_step import _abi, scene
from fluid_step.pipelines import Simulation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("downloads", [1, 2, 16, 17, 40])
def test_every_ticket_covers_its_own_copy(downloads):
    w = scene.workload("dam_break_16k")
    sim = Simulation(w.positions()[:3000], w.params)
    tickets, ref = [], []
    for k in range(downloads):
        sim.step(1, want_stats=False)
        out = np.full((3000, 4), np.nan, np.float32)
        field = _abi.FE_FIELD_POSITION_A if k % 2 == 0 else _abi.FE_FIELD_VELOCITY_B
        tickets.append((sim.data.download_async(field, out), out))
        ref.append(sim.data.download(field))
    for k in list(range(1, downloads, 2)) + list(range(0, downloads, 2)):
        t, out = tickets[k]
        sim.data.download_wait(t)
        assert np.array_equal(out.view(np.uint32), ref[k].view(np.uint32)), k
    with pytest.raises(_abi.FluidStepError):
        sim.data.download_wait(tickets[-1][0] + 1)
    sim.close()
