"""Solver control over the scene table: one block starts, ends and conditions
a solve for every scene, its threads striding over them."""
import numpy as np
import pytest

from fluid_step import _abi, scene
from fluid_step.pipelines import BatchSimulation, Simulation

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
