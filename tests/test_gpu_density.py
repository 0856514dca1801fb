"""density_alpha's two forms and the limits of their tables, against the
oracle: runs of a cell per warp, candidates per row, candidates per lane."""
import numpy as np
import pytest

from fluid_step import _abi, scene
from fluid_step.pipelines import Simulation

pytestmark = pytest.mark.gpu

FIELDS = [_abi.FE_FIELD_POSITION_A, _abi.FE_FIELD_VELOCITY_B, _abi.FE_FIELD_DENSITY,
          _abi.FE_FIELD_FACTOR, _abi.FE_FIELD_SOURCE_TERM, _abi.FE_FIELD_PRESSURE]


def _cells(per_cell, side, h, seed, spread=1.0):
    """`per_cell` particles at random places of each of side^3 cells of size h."""
    rng = np.random.default_rng(seed)
    ijk = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    at = np.repeat(ijk, per_cell, 0) + 1
    u = 0.5 + (rng.random(at.shape) - 0.5) * spread * 0.98
    return ((at + u) * h).astype(np.float32)


@pytest.mark.parametrize("mode", [_abi.FE_MODE_REFERENCE, _abi.FE_MODE_FIXED])
@pytest.mark.parametrize("per_cell,side,spread", [
    (1, 9, 1.0),      # 32 runs a warp: each lane by itself
    (3, 8, 1.0),      # 10 or 11 runs: both forms
    (4, 8, 1.0),      # 8 or 9
    (8, 6, 1.0),      # bulk fluid
    (13, 5, 1.0),     # rows of 351, near the 384 a row may hold; over 44 in range
    (15, 5, 1.0),     # rows of 405: the single-phase walk
    (40, 3, 0.2),     # clumps denser than the neighbour list
    (300, 1, 0.5),    # one cell
])
def test_rows_and_runs_of_every_size(oracle_mod, per_cell, side, spread, mode):
    p = scene.dam_break_params((0, 0, 0), (1.3, 1.3, 1.3), mode=mode)
    p.dt = 0.0002
    pos = _cells(per_cell, side, 0.1, per_cell, spread)
    sim, orc = Simulation(pos, p), oracle_mod.Oracle(p, pos)
    for k in range(2):
        sim.step(1)
        orc.step(1)
        for f in FIELDS:
            a, b = sim.data.download(f).view(np.uint32), orc.field(f).view(np.uint32)
            bad = np.nonzero(a.reshape(-1) != b.reshape(-1))[0]
            assert bad.size == 0, (k, f, bad.size)
    sim.close()


@pytest.mark.parametrize("scale,origin", [(1.0, 0.0), (1e-3, 0.0), (1e3, 0.0), (1.0, 3000.0),
                                          (1e-17, 0.0)])
def test_half_precision_near_test_at_other_scales(oracle_mod, scale, origin):
    """The near test works in units of h relative to the run's first particle:
    other lengths, a far origin, and an h beyond its line (each lane walks)."""
    h = np.float32(0.1 * scale)
    p = scene.dam_break_params((0, 0, 0), (1e9, 1e9, 1e9))
    p.smoothing_radius = float(h)
    p.particle_radius = float(h) / 4
    p.viscosity = 0.0
    pos = (_cells(8, 6, 0.1, 3) * np.float32(scale) + np.float32(origin * scale)).astype(np.float32)
    sim, orc = Simulation(pos, p), oracle_mod.Oracle(p, pos)
    lib = sim.data._lib
    for name in ("neighbor_search", "density_alpha"):
        _abi.check(lib, getattr(lib, "fe_" + name)(sim.data.handle), name)
        orc.run(name)
    for f in (_abi.FE_FIELD_DENSITY, _abi.FE_FIELD_FACTOR):
        a, b = sim.data.download(f), orc.field(f)
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (f, a[:4], b[:4])
    sim.close()


def test_half_precision_near_test_is_a_superset():
    """The arithmetic of the near test (packed half precision, fused) over
    pairs at distances up to h: none is rejected by 1 + 2^-7."""
    rng = np.random.default_rng(1)
    n = 400_000
    a = rng.uniform(0, 1, (n, 3))                     # within the run's cell
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    c = a + d * rng.uniform(0.98, 1.0, (n, 1))        # at nearly h
    o = rng.uniform(0, 1, (n, 3))                     # the run's first particle
    x = (a - o).astype(np.float16).astype(np.float64)
    y = (c - o).astype(np.float16).astype(np.float64)
    f = (x - y).astype(np.float16).astype(np.float64)
    s = (f[:, 2] ** 2).astype(np.float16).astype(np.float64)
    s = (f[:, 1] ** 2 + s).astype(np.float16).astype(np.float64)
    s = (f[:, 0] ** 2 + s).astype(np.float16).astype(np.float64)
    assert s.max() <= 1.0058


@pytest.mark.parametrize("n", [7, 8, 9, 37888, 37889, 56832, 56833])
def test_particles_per_warp(oracle_mod, n):
    """Both sides of 8, 16 and 32 particles per warp, and ragged last warps."""
    p = scene.dam_break_params((0, 0, 0), (4.0, 4.0, 4.0), mode=_abi.FE_MODE_FIXED)
    pos, _ = scene.lattice((0, 0, 0), (39, 39, 39), 0.025, 1000.0, 0.05, 0.04, 5)
    pos = pos[:n]
    sim, orc = Simulation(pos, p), oracle_mod.Oracle(p, pos)
    sim.step(1)
    orc.step(1)
    for f in FIELDS:
        a, b = sim.data.download(f).view(np.uint32), orc.field(f).view(np.uint32)
        assert np.array_equal(a, b), f
    sim.close()


def _row_of(total, h, seed, scattered=0):
    """3^3 cells whose particles make the centre cell's row exactly `total` long,
    and `scattered` particles in the cells around them."""
    rng = np.random.default_rng(seed)
    ijk = np.stack(np.meshgrid(*[np.arange(3)] * 3, indexing="ij"), -1).reshape(-1, 3) + 2
    per = np.full(27, total // 27)
    per[: total - per.sum()] += 1
    rng.shuffle(per)
    at = np.repeat(ijk, per, 0)
    if scattered:
        at = np.concatenate([at, rng.integers(0, 7, (scattered, 3))])
    return ((at + rng.uniform(0.02, 0.98, at.shape)) * h).astype(np.float32)


@pytest.mark.parametrize("mode", [_abi.FE_MODE_REFERENCE, _abi.FE_MODE_FIXED])
@pytest.mark.parametrize("total", [383, 384, 385, 416, 767, 768, 769, 1153, 4000])
def test_rows_of_several_windows(oracle_mod, total, mode):
    """Rows that end at, before and after the 384 candidates of a window, buckets
    that go on from one window to the next, and warps whose runs need different
    numbers of windows."""
    p = scene.dam_break_params((0, 0, 0), (1.3, 1.3, 1.3), mode=mode)
    p.dt = 0.0002
    pos = _row_of(total, 0.1, total, scattered=200)
    sim, orc = Simulation(pos, p), oracle_mod.Oracle(p, pos)
    for k in range(2):
        sim.step(1)
        orc.step(1)
        for f in FIELDS:
            a, b = sim.data.download(f).view(np.uint32), orc.field(f).view(np.uint32)
            assert np.array_equal(a, b), (k, f)
    sim.close()


def test_rows_of_several_windows_with_32_particles_per_warp(oracle_mod):
    """The same in a context large enough for whole warps."""
    p = scene.dam_break_params((0, 0, 0), (4.0, 4.0, 4.0), mode=_abi.FE_MODE_FIXED)
    p.dt = 0.0002
    rest, _ = scene.lattice((1.2, 0, 1.2), (40, 39, 39), 0.025, 1000.0, 0.05, 0.04, 5)
    pos = np.concatenate([_row_of(1000, 0.1, 7, scattered=300), rest])
    sim, orc = Simulation(pos, p), oracle_mod.Oracle(p, pos)
    sim.step(1)
    orc.step(1)
    for f in FIELDS:
        a, b = sim.data.download(f).view(np.uint32), orc.field(f).view(np.uint32)
        assert np.array_equal(a, b), f
    sim.close()


@pytest.mark.parametrize("mode", [_abi.FE_MODE_REFERENCE, _abi.FE_MODE_FIXED])
def test_many_runs_beside_crowded_cells(oracle_mod, mode):
    """Warps with a cell per particle, some of whose particles have one, two or
    more stages of candidates in a crowded cell beside theirs."""
    p = scene.dam_break_params((0, 0, 0), (4.0, 4.0, 4.0), mode=mode)
    p.dt = 0.0002
    pos = [_cells(1, 38, 0.1, 11)]
    rng = np.random.default_rng(12)
    for m in (30, 44, 45, 60, 90, 150, 400):
        for at in rng.integers(2, 38, (5, 3)):
            pos.append((at + rng.uniform(0.02, 0.98, (m, 3))) * 0.1)
    pos = np.concatenate(pos).astype(np.float32)
    assert len(pos) > 56832          # 32 particles per warp
    sim, orc = Simulation(pos, p), oracle_mod.Oracle(p, pos)
    sim.step(1)
    orc.step(1)
    for f in FIELDS:
        a, b = sim.data.download(f).view(np.uint32), orc.field(f).view(np.uint32)
        assert np.array_equal(a, b), f
    sim.close()


@pytest.mark.parametrize("n", [23680, 23681, 23700])
def test_particles_per_warp_around_the_first_line(oracle_mod, n):
    test_particles_per_warp(oracle_mod, n)
