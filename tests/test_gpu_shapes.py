"""The shapes of the neighbour passes: every one gives the same bits."""
import ctypes

import numpy as np
import pytest

from fluid_step import _abi, scene
from fluid_step.pipelines import (BatchSimulation, CommandBufferBuilder, ComputePipelines,
                                  GpuPhysicsData, Simulation)

pytestmark = pytest.mark.gpu

FIELDS = [_abi.FE_FIELD_POSITION_A, _abi.FE_FIELD_POSITION_B, _abi.FE_FIELD_VELOCITY_A,
          _abi.FE_FIELD_VELOCITY_B, _abi.FE_FIELD_DENSITY, _abi.FE_FIELD_FACTOR,
          _abi.FE_FIELD_SOURCE_TERM, _abi.FE_FIELD_PRESSURE, _abi.FE_FIELD_PRESSURE_ACCEL]


def _scene(n, mode=_abi.FE_MODE_REFERENCE):
    p = scene.dam_break_params((0, 0, 0), (3.0, 3.0, 2.0), mode=mode)
    pos, _ = scene.lattice((0, 0, 0), (28, 28, 28), 0.025, 1000.0, 0.05, 0.01, 5)
    return p, pos[:n]


def _same(a, b, what):
    for f in FIELDS:
        x, y = a(f).view(np.uint32).reshape(-1), b(f).view(np.uint32).reshape(-1)
        bad = np.nonzero(x != y)[0]
        assert bad.size == 0, (what, f, bad.size, bad[:1])


@pytest.mark.parametrize("mode", [_abi.FE_MODE_REFERENCE, _abi.FE_MODE_FIXED])
@pytest.mark.parametrize("n", [63, 64, 65, 18943, 18944, 18945])
def test_passes_and_frames_around_the_few_particle_line(oracle_mod, n, mode):
    """Both sides of a 64-thread block and of the line between the shapes:
    frames and single passes against the oracle."""
    p, pos = _scene(n, mode)
    orc = oracle_mod.Oracle(p, pos)
    sim = Simulation(pos, p)
    data = GpuPhysicsData(pos, p)
    steps = ComputePipelines()
    steps.prepare_all(data)
    for k in range(2):
        orc.step(1)
        sim.step(1)
        steps.submit_substeps(CommandBufferBuilder(data), 4, 1, k == 0)
    _same(sim.data.download, orc.field, "frames")
    _same(data.download, orc.field, "passes")
    sim.close()
    data.close()


def test_tuned_shapes_above_the_line():
    """The shapes of fe_set_tuning, where they are used."""
    p, pos = _scene(20011, _abi.FE_MODE_FIXED)
    p.solver = _abi.FE_SOLVER_TOLERANCE
    ref = Simulation(pos, p)
    ref.step(2)
    for threads, persistent in ((128, 0), (512, 0), (128, 1), (256, 1), (512, 1)):
        sim = Simulation(pos, p)
        t = sim.data.tuning()
        t.nbr_threads[:] = [min(threads, 256), threads, threads, 256]
        t.nbr_persistent[:] = [persistent] * 4
        sim.data.set_tuning(t)
        sim.step(2)
        _same(sim.data.download, ref.data.download, (threads, persistent))
        sim.close()
    ref.close()


@pytest.mark.parametrize("scenes", [2, 7])
def test_stage_calls_of_a_small_batch(scenes):
    """Every stage call of a batch of few particles, its per-scene statistics
    included, against one context per scene."""
    pos, par = [], []
    for k in range(scenes):
        p, x = _scene(300 + 97 * k, _abi.FE_MODE_FIXED)
        pos.append(x)
        par.append(p)
    batch = BatchSimulation(pos, par)
    singles = [Simulation(x, p) for x, p in zip(pos, par)]
    names = ["neighbor_search", "density_alpha", "viscosity", "density_source",
             "pressure_force", "pressure_update", "pressure_integration", "neighbor_search",
             "density_alpha", "divergence_source", "pressure_force", "pressure_update",
             "divergence_integration", "stats_pass"]
    for sim in [batch] + singles:
        lib, h = sim.data._lib, sim.data.handle
        for _ in range(4):
            for name in names:
                _abi.check(lib, getattr(lib, "fe_" + name)(h), name)
    lib = batch.data._lib
    for k, sim in enumerate(singles):
        a, b = _abi.FeStats(), _abi.FeStats()
        _abi.check(lib, lib.fe_read_scene_stats(batch.data.handle, k, ctypes.byref(a)), "stats")
        _abi.check(lib, lib.fe_read_stats(sim.data.handle, ctypes.byref(b)), "stats")
        assert bytes(a) == bytes(b), k
    x = batch.data.download(_abi.FE_FIELD_POSITION_A).view(np.uint32)
    y = np.concatenate([s.data.download(_abi.FE_FIELD_POSITION_A).view(np.uint32)
                        for s in singles])
    assert np.array_equal(x, y)
    batch.close()
    for sim in singles:
        sim.close()
