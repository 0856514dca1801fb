"""Solver control over the scene table: one block starts, ends and conditions
a solve for every scene, its threads striding over them."""
import numpy as np
import pytest

from fluid_step import _abi, scene
from fluid_step.pipelines import (BatchSimulation, CommandBufferBuilder, ComputePipelines,
                                  GpuPhysicsData, Simulation)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_scenes", [2, 32, 33, 256, 257])
def test_each_scene_keeps_its_own_iteration_counts(n_scenes):
    """Around a warp and a block of scenes: every scene runs its own number of
    iterations (the last one the most), and ends with the fields it has alone."""
    w = scene.batch_workload(n_scenes=n_scenes, seed=4, lo=20, hi=90)
    params = w.params()
    for k, p in enumerate(params):
        p.density_solver_iterations = 3 + k % 3 + (k == n_scenes - 1) * 4
        p.divergence_solver_iterations = 2 + k % 4
    pos = w.positions()
    batch = BatchSimulation(pos, params)
    batch.step(2)
    for s in range(n_scenes):
        st = batch.data.read_scene_stats(s)
        assert (st.density_iterations, st.divergence_iterations) == (
            params[s].density_solver_iterations, params[s].divergence_solver_iterations), s
        assert st.total_density_iterations == 2 * st.density_iterations
    for s in sorted({0, n_scenes // 2, n_scenes - 1}):
        one = Simulation(pos[s], params[s])
        one.step(2)
        for f in (_abi.FE_FIELD_POSITION_A, _abi.FE_FIELD_PRESSURE):
            a, b = batch.data.scene(batch.data.download(f), s), one.data.download(f)
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (s, f)
        one.close()
    batch.close()


FIELDS = [_abi.FE_FIELD_POSITION_A, _abi.FE_FIELD_POSITION_B, _abi.FE_FIELD_VELOCITY_A,
          _abi.FE_FIELD_VELOCITY_B, _abi.FE_FIELD_DENSITY, _abi.FE_FIELD_FACTOR,
          _abi.FE_FIELD_SOURCE_TERM, _abi.FE_FIELD_PRESSURE, _abi.FE_FIELD_PRESSURE_ACCEL]


@pytest.mark.parametrize("non_finite", [False, True])
@pytest.mark.parametrize("n,iters", [(1, 2), (255, 0), (256, 1), (257, 2), (3001, 1), (3001, 5)])
@pytest.mark.parametrize("mode", [_abi.FE_MODE_REFERENCE, _abi.FE_MODE_FIXED])
def test_frame_solve_is_the_solve_pass_by_pass(mode, n, iters, non_finite):
    """The frame's solves (the density solve's first iteration has no
    neighbour loop there) against the general passes called one by one, bit
    for bit: no iteration, the first one alone, several; with an infinite
    velocity, whose source terms are not finite, the gradients' zeros do not
    stay zeros and the frame has to run the loops as well."""
    w = scene.workload("dam_break_16k")
    p = _abi.copy_params(w.params)
    p.mode = mode
    p.density_solver_iterations = p.divergence_solver_iterations = iters
    pos = w.positions()[:n]
    sim = Simulation(pos, p)
    data = GpuPhysicsData(pos, p)
    steps = ComputePipelines()
    steps.prepare_all(data)
    builder = CommandBufferBuilder(data)
    for k in range(2):
        if non_finite and k == 1:
            v = np.zeros((n, 4), np.float32)
            v[n // 2, 1] = np.inf
            for d in (sim.data, data):
                d.upload(_abi.FE_FIELD_VELOCITY_B, v)
        sim.step(1, want_stats=False)
        steps.submit_substeps(builder, iters, 1, k == 0)
        for f in FIELDS:
            a, b = sim.data.download(f), data.download(f)
            bad = np.nonzero(a.view(np.uint32).reshape(-1) != b.view(np.uint32).reshape(-1))[0]
            assert bad.size == 0, (k, f, bad.size, a.reshape(-1)[bad[0]], b.reshape(-1)[bad[0]])
    sim.close()
    data.close()


@pytest.mark.parametrize("n", [9472, 9473, 18945, 28417, 37888, 37889, 56832, 56833])
@pytest.mark.parametrize("cap", [100, 3])
def test_resident_solve_around_its_lines(oracle_mod, n, cap):
    """The solve as one kernel, around the sizes where a particle per thread goes
    over to chunks and chunks to the iterated passes: iterations to a tolerance
    (the FP64 sums over warps and chunks) and to a cap, against the oracle."""
    p = scene.dam_break_params((0, 0, 0), (4.0, 4.0, 4.0), mode=_abi.FE_MODE_FIXED,
                               solver=_abi.FE_SOLVER_TOLERANCE)
    p.max_iterations = cap
    pos, _ = scene.lattice((0, 0, 0), (39, 39, 39), 0.025, 1000.0, 0.05, 0.03, 5)
    pos = pos[:n]
    vel = np.random.default_rng(n).normal(0, 0.3, pos.shape).astype(np.float32)
    sim, orc = Simulation(pos, p, velocities=vel), oracle_mod.Oracle(p, pos, vel)
    for _ in range(2):
        a, b = sim.step(1), orc.step(1)
        for name in ("density_iterations", "divergence_iterations", "density_residual",
                     "divergence_residual", "density_residual_max", "divergence_residual_max"):
            assert getattr(a, name) == getattr(b, name), name
        assert bool(a.flags & _abi.FE_STATS_ITERATION_CAP_HIT) == (
            cap == 3 or bool(b.flags & _abi.FE_STATS_ITERATION_CAP_HIT))
    for f in FIELDS:
        x, y = sim.data.download(f).view(np.uint32), orc.field(f).view(np.uint32)
        assert np.array_equal(x, y), f
    sim.close()


@pytest.mark.parametrize("solvers", ["fixed", "mixed"])
def test_batch_solves_resident_or_iterated(solvers):
    """Scenes that all iterate a fixed number of times are solved in one kernel,
    others iteration by iteration; after a change of parameters too.  Either
    way each as it is alone, one of them with a source that is not finite."""
    w = scene.batch_workload(n_scenes=5, seed=6, lo=300, hi=900)
    params = w.params()
    for k, p in enumerate(params):
        p.density_solver_iterations, p.divergence_solver_iterations = 2 + k, 5 - k
    pos = w.positions()
    batch = BatchSimulation(pos, params)
    singles = [Simulation(a, q) for a, q in zip(pos, params)]
    for frame in range(3):
        if frame == 1 and solvers == "mixed":
            for s in (1, 3):
                params[s].solver = _abi.FE_SOLVER_TOLERANCE
                batch.data.set_scene_params(s, params[s])
                singles[s].data.sync_with_scene(params[s])
        if frame == 2:
            v = batch.data.download(_abi.FE_FIELD_VELOCITY_B)
            first, n = int(batch.data.scene_first[2]), int(batch.data.scene_count[2])
            v[first + n // 2, 1] = np.inf
            batch.data.upload(_abi.FE_FIELD_VELOCITY_B, v)
            singles[2].data.upload(_abi.FE_FIELD_VELOCITY_B, v[first:first + n])
        batch.step(1, want_stats=False)
        for sim in singles:
            sim.step(1, want_stats=False)
        for s, sim in enumerate(singles):
            for f in FIELDS:
                a, b = batch.data.scene(batch.data.download(f), s), sim.data.download(f)
                assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (frame, s, f)
            a, b = None, None
            try:
                a, b = batch.data.read_scene_stats(s), sim.data.read_stats()
            except _abi.FluidStepError:
                pass
            if a and b:
                assert (a.density_iterations, a.divergence_iterations) == (
                    b.density_iterations, b.divergence_iterations), (frame, s)
    batch.close()
    for sim in singles:
        sim.close()


def _with_clumps(n, per_clump, seed):
    """A lattice of n particles and, above it, four clumps whose particles have
    more neighbours than the list holds."""
    pos, _ = scene.lattice((0, 0, 0), (40, 20, 48), 0.025, 1000.0, 0.05, 0.02, seed)
    rng = np.random.default_rng(seed)
    at = np.array([[0.55, 2.0, 0.55], [1.55, 2.0, 0.55], [0.55, 2.0, 1.55], [0.6, 2.0, 0.6]])
    clumps = np.repeat(at, per_clump, 0) + rng.uniform(-0.04, 0.04, (4 * per_clump, 3))
    return np.concatenate([pos[:n], clumps]).astype(np.float32)


@pytest.mark.parametrize("per_clump", [64, 90])
@pytest.mark.parametrize("solver", [_abi.FE_SOLVER_TOLERANCE, _abi.FE_SOLVER_FIXED_ITERS])
@pytest.mark.parametrize("n", [11000, 30011])
def test_strided_resident_solve_past_the_neighbour_list(oracle_mod, n, solver, per_clump):
    """Particles with more neighbours than the list holds walk the buckets in
    every half iteration, between whose barriers other blocks write what the walk
    reads: several iterations over strided chunks against the oracle."""
    p = scene.dam_break_params((0, 0, 0), (4.0, 4.0, 4.0), mode=_abi.FE_MODE_FIXED, solver=solver)
    p.density_solver_iterations, p.divergence_solver_iterations = 9, 7
    p.min_iterations, p.max_iterations = 5, 12
    p.dt = 0.0002
    pos = _with_clumps(n, per_clump, 3)
    sim, orc = Simulation(pos, p), oracle_mod.Oracle(p, pos)
    for _ in range(2):
        a, b = sim.step(1), orc.step(1)
        assert a.flags & _abi.FE_STATS_NEIGHBOR_OVERFLOW
        assert (a.density_iterations, a.divergence_iterations) == (b.density_iterations,
                                                                   b.divergence_iterations)
        for f in FIELDS:
            x, y = sim.data.download(f).view(np.uint32), orc.field(f).view(np.uint32)
            assert np.array_equal(x, y), f
    sim.close()


def test_batch_resident_solve_past_the_neighbour_list(oracle_mod):
    """The same in the scenes of a fixed-iteration batch."""
    pos = [_with_clumps(900, 90, 1), _with_clumps(2500, 70, 2), _with_clumps(700, 0, 3)]
    params = []
    for k in range(3):
        p = scene.dam_break_params((0, 0, 0), (4.0, 4.0, 4.0), mode=_abi.FE_MODE_FIXED)
        p.density_solver_iterations, p.divergence_solver_iterations = 6 + k, 5
        p.dt = 0.0002
        params.append(p)
    batch = BatchSimulation(pos, params)
    oracles = [oracle_mod.Oracle(p, a) for p, a in zip(params, pos)]
    for _ in range(2):
        batch.step(1, want_stats=False)
        for s, orc in enumerate(oracles):
            orc.step(1)
            for f in FIELDS:
                x = batch.data.scene(batch.data.download(f), s)
                assert np.array_equal(x.view(np.uint32), orc.field(f).view(np.uint32)), (s, f)
    batch.close()


@pytest.mark.parametrize("last", [9000, 10000])
def test_batch_solves_around_their_line(last):
    """Fixed-iteration batches below and above the size up to which their solves
    are one kernel: each scene as it is alone."""
    rng = np.random.default_rng(last)
    pos, params = [], []
    for k, n in enumerate((14000, 14400, last)):       # 37400 and 38400 particles
        a, _ = scene.lattice((0, 0, 0), (25, 24, 24), 0.025, 1000.0, 0.05, 0.03, k)
        pos.append(a[:n])
        p = scene.dam_break_params((0, 0, 0), (2.0, 2.0, 2.0), mode=_abi.FE_MODE_FIXED)
        p.density_solver_iterations, p.divergence_solver_iterations = 3 + 2 * k, 4 - k
        params.append(p)
    vel = [rng.normal(0, 0.3, a.shape).astype(np.float32) for a in pos]
    batch = BatchSimulation(pos, params, scene_velocities=vel)
    batch.step(2)
    for s, (a, p, v) in enumerate(zip(pos, params, vel)):
        st = batch.data.read_scene_stats(s)
        assert (st.density_iterations, st.divergence_iterations) == (3 + 2 * s, 4 - s)
        one = Simulation(a, p, velocities=v)
        one.step(2)
        for f in FIELDS:
            x = batch.data.scene(batch.data.download(f), s)
            assert np.array_equal(x.view(np.uint32), one.data.download(f).view(np.uint32)), (s, f)
        one.close()
    batch.close()


@pytest.mark.parametrize("solvers", ["fixed", "mixed"])
def test_batch_scenes_keep_their_counts_beside_a_non_finite_one(solvers):
    """The iteration counts of every scene, resident or iterated; only the scene
    with an infinite velocity may report an error, and only once it has it."""
    w = scene.batch_workload(n_scenes=5, seed=6, lo=300, hi=900)
    params = w.params()
    for k, p in enumerate(params):
        p.density_solver_iterations, p.divergence_solver_iterations = 2 + k, 5 - k
        if solvers == "mixed" and k in (1, 3):
            p.solver = _abi.FE_SOLVER_TOLERANCE
    pos = w.positions()
    batch = BatchSimulation(pos, params)
    singles = [Simulation(a, q) for a, q in zip(pos, params)]
    for frame in range(3):
        if frame == 2:
            v = batch.data.download(_abi.FE_FIELD_VELOCITY_B)
            first, n = int(batch.data.scene_first[2]), int(batch.data.scene_count[2])
            v[first + n // 2, 1] = np.inf
            batch.data.upload(_abi.FE_FIELD_VELOCITY_B, v)
            singles[2].data.upload(_abi.FE_FIELD_VELOCITY_B, v[first:first + n])
        batch.step(1, want_stats=False)
        for s, sim in enumerate(singles):
            sim.step(1, want_stats=False)
            if frame == 2 and s == 2:
                continue
            a, b = batch.data.read_scene_stats(s), sim.data.read_stats()
            counts = (a.density_iterations, a.divergence_iterations)
            assert counts == (b.density_iterations, b.divergence_iterations), (frame, s)
            if params[s].solver == _abi.FE_SOLVER_FIXED_ITERS:
                assert counts == (2 + s, 5 - s), (frame, s)
    batch.close()
    for sim in singles:
        sim.close()


@pytest.mark.parametrize("mode", [_abi.FE_MODE_REFERENCE, _abi.FE_MODE_FIXED])
@pytest.mark.parametrize("side,per_clump", [(0.24, 0), (0.4, 0), (0.4, 100)])
def test_resident_solve_past_the_neighbour_list(oracle_mod, side, per_clump, mode):
    """A particle per thread: particles that walk the buckets in every half
    iteration, all of them, some, and beside ones with lists."""
    rng = np.random.default_rng(int(side * 100))
    pos = (rng.random((900, 3)) * side + 0.12).astype(np.float32)
    if per_clump:
        pos = np.concatenate([pos, _with_clumps(1500, per_clump, 4) + np.float32(0.6)])
    p = scene.dam_break_params((0, 0, 0), (4.0, 4.0, 4.0), mode=mode)
    p.density_solver_iterations, p.divergence_solver_iterations = 5, 6
    p.dt = 0.0001
    sim, orc = Simulation(pos, p), oracle_mod.Oracle(p, pos)
    for k in range(2):
        st = sim.step(1)
        orc.step(1)
        if k == 0:
            assert st.flags & _abi.FE_STATS_NEIGHBOR_OVERFLOW
        for f in FIELDS:
            x, y = sim.data.download(f).view(np.uint32), orc.field(f).view(np.uint32)
            assert np.array_equal(x, y), (k, f)
    sim.close()


@pytest.mark.parametrize("mode", [_abi.FE_MODE_REFERENCE, _abi.FE_MODE_FIXED])
@pytest.mark.parametrize("n", [900, 9000, 12000, 20000])
def test_passes_past_the_neighbour_list(n, mode):
    """Pass by pass, in the shapes for few particles and above them, where some
    particles walk the buckets: the fields of the whole frame."""
    p = scene.dam_break_params((0, 0, 0), (4.0, 4.0, 4.0), mode=mode)
    p.density_solver_iterations = p.divergence_solver_iterations = 3
    p.dt = 0.0002
    pos = _with_clumps(n, 90, 6)
    sim, data = Simulation(pos, p), GpuPhysicsData(pos, p)
    steps = ComputePipelines()
    steps.prepare_all(data)
    builder = CommandBufferBuilder(data)
    for k in range(2):
        sim.step(1, want_stats=False)
        steps.submit_substeps(builder, 3, 1, k == 0)
        for f in FIELDS:
            a, b = sim.data.download(f), data.download(f)
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (k, f)
    assert sim.data.read_stats().flags & _abi.FE_STATS_NEIGHBOR_OVERFLOW
    sim.close()
    data.close()
