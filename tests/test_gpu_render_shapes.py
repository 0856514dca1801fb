"""The splat's and the water pass's tiles at grids that are no multiple of them."""
import numpy as np
import pytest

from fluid_step import _abi, camera, scene
from fluid_step.pipelines import Simulation
from test_gpu_raymarch import _compare

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (31, 7, 8), (33, 9, 17), (32, 8, 8), (65, 40, 24), (5, 3, 70)]


def _sim(res, n=1500):
    p, pos, _ = scene.app_scene()
    p.grid_res[:] = list(res)
    rng = np.random.default_rng(sum(res))
    pos = pos[rng.permutation(len(pos))[:n]].copy()
    pos[:100] = pos[0]                       # many particles in one voxel
    pos[100] = list(p.box_min)
    pos[101] = list(p.box_max)
    return p, pos, Simulation(pos, p)


@pytest.mark.parametrize("res", SHAPES)
def test_splat_of_any_grid(oracle_mod, res):
    p, pos, sim = _sim(res)
    got = sim.data.splat_density()
    ref = oracle_mod.splat_density(np.c_[pos, np.ones(len(pos))].astype(np.float32), p)
    assert np.array_equal(got, ref)
    sim.close()


@pytest.mark.parametrize("eye", [(0.0, 2.0, -4.5), (-0.5, 1.5, 0.0)])
@pytest.mark.parametrize("res", [(31, 7, 8), (33, 9, 17), (65, 40, 24), (128, 128, 128)])
def test_water_pass_of_any_grid(oracle_mod, res, eye):
    """The coarse look at 4^3 blocks: ragged last blocks, borders, an eye
    inside the box."""
    p, pos, sim = _sim(res, n=20000)
    grid = sim.data.splat_density()
    assert (grid > 300).any()
    sky = camera.gradient_sky(64, 32)
    sim.data.set_skybox(sky)
    cam = camera.make_camera(eye, (-0.3, 1.2, 0.0), 120, 90)
    _compare(sim.data.raymarch(cam), oracle_mod.raymarch(grid, sky, cam, p.box_min, p.box_max))
    sim.close()


@pytest.mark.parametrize("res", [(31, 40, 33), (32, 32, 32), (33, 9, 17), (64, 20, 30),
                                 (100, 5, 40)])
def test_water_pass_of_an_uploaded_grid(oracle_mod, res):
    """What the splat keeps for the water pass follows a grid that is uploaded:
    blocks above the surface count, below it, mixed, and its neighbours 300, 301."""
    p, pos, sim = _sim(res)
    sim.data.splat_density()
    rng = np.random.default_rng(sum(res))
    rx, ry, rz = res
    coarse = rng.choice([0, 299, 300, 301, 302, 5000], ((rz + 5) // 6, (ry + 5) // 6, (rx + 5) // 6),
                        p=[0.3, 0.1, 0.1, 0.1, 0.1, 0.3])
    grid = np.ascontiguousarray(
        np.kron(coarse, np.ones((6, 6, 6), int))[:rz, :ry, :rx].astype(np.uint32))
    sim.data.upload(_abi.FE_FIELD_DENSITY_GRID, grid)
    sky = camera.gradient_sky(64, 32)
    sim.data.set_skybox(sky)
    cam = camera.make_camera((0.0, 2.0, -4.5), (-0.3, 1.2, 0.0), 160, 120)
    _compare(sim.data.raymarch(cam), oracle_mod.raymarch(grid, sky, cam, p.box_min, p.box_max))
    # and the next splat's again
    grid = sim.data.splat_density()
    img = sim.data.raymarch(cam)
    ref = oracle_mod.raymarch(grid, sky, cam, p.box_min, p.box_max)
    assert ((img[..., 3] > 0) == (ref[..., 3] > 0)).mean() >= 0.995
    sim.close()
