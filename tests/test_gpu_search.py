"""The search by cell counts: the stable sort by cell hash, at the edges of its
tiles and runs, against the oracle."""
import numpy as np
import pytest

from fluid_step import _abi, scene
from fluid_step.pipelines import BatchSimulation, Simulation

pytestmark = pytest.mark.gpu

SEARCH = [_abi.FE_FIELD_ENTRY_HASH, _abi.FE_FIELD_ENTRY_INDEX, _abi.FE_FIELD_GRID_START,
          _abi.FE_FIELD_POSITION_B, _abi.FE_FIELD_VELOCITY_B]


def _params(side=3.0, mode=_abi.FE_MODE_REFERENCE):
    return scene.dam_break_params((0, 0, 0), (side,) * 3, mode=mode)


def _positions(n, kind, side=3.0):
    rng = np.random.default_rng(n)
    if kind == "uniform":          # unordered: every run of equal keys is short
        return rng.uniform(0.03, side - 0.03, (n, 3)).astype(np.float32)
    if kind == "one_cell":         # a single run of the whole warp, one long cell
        return rng.uniform(0.41, 0.49, (n, 3)).astype(np.float32)
    p = rng.uniform(0.03, side - 0.03, (n, 3)).astype(np.float32)
    p[::3] = p[0] * 0 + np.float32(0.75)     # a third at one point, spread over all warps
    return p


@pytest.mark.parametrize("kind", ["uniform", "one_cell", "third"])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 256, 2047, 4097, 8193])
def test_search_is_the_stable_sort(oracle_mod, n, kind):
    """Tables of 1 slot to several scan tiles; twice, since the counters and
    the scan's status carry over from one search to the next."""
    if kind != "uniform":
        n = min(n, 700)
    p, pos = _params(), _positions(n, kind)
    sim = Simulation(pos, p)
    orc = oracle_mod.Oracle(p, pos)
    lib = sim.data._lib
    for k in range(2):
        _abi.check(lib, lib.fe_neighbor_search(sim.data.handle), "fe_neighbor_search")
        orc.run("neighbor_search")
        for f in SEARCH:
            a, b = sim.data.download(f), orc.field(f)
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (k, f)
        moved = _positions(n, "uniform")
        sim.data.upload(_abi.FE_FIELD_POSITION_A, np.c_[moved, np.ones(n)])
        orc.upload(_abi.FE_FIELD_POSITION_A, np.c_[moved, np.ones(n)].astype(np.float32))
    sim.close()


@pytest.mark.parametrize("counts", [(1, 1, 1), (5000, 3, 257, 4096), (64,) * 70])
def test_search_of_a_batch_keeps_scenes_apart(counts):
    """Tables of several scenes back to back, a total that is no multiple of
    the scan's tile or of 8: each scene as it is alone."""
    pos = [_positions(n, "uniform", 2.0) + 0 for n in counts]
    par = [_params(2.0, _abi.FE_MODE_FIXED) for _ in counts]
    batch = BatchSimulation(pos, par)
    batch.step(2)
    for s in sorted({0, len(counts) // 2, len(counts) - 1}):
        one = Simulation(pos[s], par[s])
        one.step(2)
        for f in (_abi.FE_FIELD_POSITION_B, _abi.FE_FIELD_VELOCITY_B, _abi.FE_FIELD_PRESSURE):
            a, b = batch.data.scene(batch.data.download(f), s), one.data.download(f)
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (s, f)
        one.close()
    batch.close()
