"""The full-shell brick kernels (6 and 8) where their neighbour walk can go wrong: rows of more
candidates than one walk segment holds, segments that do not fit and are evaluated early, odd
rows and their fillers, boxes smaller than a halo (cells staged at several images), halo rows
longer than a warp.  Each must equal the thread-per-bead kernel (1), which tests and adds
the same pairs one by one from global memory, bit for bit."""

import numpy as np
import pytest

import pdpd_engine as E
import pdpd_world as W

pytestmark = pytest.mark.gpu


def _run(world, steps, **cfg):
    w = world.copy()
    eng = E.GB300DPDEngine("fp32")
    for k, v in cfg.items():
        eng.SetConfigEntry(k, v)
    eng.Attach(w)
    eng.Run(steps)
    return w


CASES = {
    # box, density, kernel and brick shape
    "dense_rows": ((6, 5, 7), 13, {"force_kernel": 8, "brick_x": 2, "brick_y": 2, "brick_z": 2}),
    "denser_rows": ((4, 4, 5), 24, {"force_kernel": 6, "brick_x": 1, "brick_y": 1, "brick_z": 2}),
    "early_evaluation": ((7, 6, 9), 9, {"force_kernel": 8, "list_capacity": 3}),
    "sparse": ((9, 8, 7), 0.4, {"force_kernel": 8}),
    "side_2": ((2, 2, 2), 3, {"force_kernel": 6}),
    "side_3_by_2": ((3, 2, 5), 5, {"force_kernel": 8, "brick_x": 8, "brick_y": 8, "brick_z": 8}),
    "halo_row_of_33": ((3, 2, 31), 3, {"force_kernel": 8, "brick_x": 1, "brick_y": 1, "brick_z": 32}),
    "halo_row_of_34": ((2, 3, 64), 3, {"force_kernel": 6, "brick_x": 1, "brick_y": 2, "brick_z": 32}),
    "uneven_bricks": ((13, 11, 17), 3, {"force_kernel": 8, "brick_x": 5, "brick_y": 8, "brick_z": 8}),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_walk_edges_equal_the_bead_kernel(name):
    box, density, cfg = CASES[name]
    world = W.make_water(box, seed=51, dt=0.002, density=density)
    ref = _run(world, 4, force_kernel=1)
    w = _run(world, 4, **cfg)
    assert np.array_equal(w.x, ref.x) and np.array_equal(w.v, ref.v) and np.array_equal(w.f, ref.f)


@pytest.mark.parametrize("force_kernel", [6, 8])
def test_walk_of_coincident_and_barely_separated_beads(force_kernel):
    """Beads at one place (the pair test leaves them out) and pairs at separations around 1
    (the walk's test keeps candidates up to 1.0001, the exact one decides)."""
    world = W.make_water(6, seed=52, dt=0.002)
    rng = np.random.default_rng(53)
    n = world.n_beads // 2
    d = rng.standard_normal((n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    r = 1.0 + rng.uniform(-2e-4, 2e-4, n)
    r[:5] = 0.0
    world.x[n:2 * n] = np.mod(world.x[:n] + r[:, None] * d, 6.0)
    world.v[:] = 0.0
    ref = _run(world, 2, force_kernel=1)
    w = _run(world, 2, force_kernel=force_kernel)
    assert np.array_equal(w.x, ref.x) and np.array_equal(w.f, ref.f)


@pytest.mark.parametrize("cfg", [{}, {"list_capacity": 3}, {"grid_blocks": 7}])
@pytest.mark.parametrize("box", [(2, 2, 2), (4, 3, 5), (9, 9, 9), (12, 12, 12), (14, 13, 14), (16, 16, 16),
                                 (17, 17, 16), (18, 18, 18)])
def test_three_lanes_per_bead_equal_the_bead_kernel(box, cfg):
    """The smallest boxes run three lanes per bead (18^3 the largest): with chains, and a clump whose
    beads have more candidates than a bead's pool holds."""
    world = W.make_polymer_box(box, chain_fraction=0.2, seed=54, dt=0.0005)
    free = np.flatnonzero(world.is_monomer)[:60 if world.n_beads > 100 else 0]
    world.x[free] = 1.0 + 0.8 * np.random.default_rng(55).random((len(free), 3))
    ref = _run(world, 3, force_kernel=1)
    w = _run(world, 3, **cfg)
    assert np.array_equal(w.x, ref.x) and np.array_equal(w.v, ref.v) and np.array_equal(w.f, ref.f)


@pytest.mark.parametrize("list_capacity", [0, 10, 40])
@pytest.mark.parametrize("force_kernel", [6, 8])
@pytest.mark.parametrize("density", [4.5, 11, 30])
def test_dense_boxes_equal_the_bead_kernel(density, force_kernel, list_capacity):
    """Boxes dense enough for the lanes to keep more segments and flush them together: room for all
    of a bead's, for a plane of rows, for less; bricks that are staged, and a clump that is not.
    A list_capacity set later applies from the next attach."""
    world = W.make_water((7, 9, 8), seed=56, dt=0.0005, density=density, a=0.5)
    n = world.n_beads // 8
    world.x[:n] = 2.0 + 2.5 * np.random.default_rng(57).random((n, 3))
    ref = _run(world, 3, force_kernel=1)
    w = world.copy()
    eng = E.GB300DPDEngine("fp32")
    eng.SetConfigEntry("force_kernel", force_kernel)
    eng.SetConfigEntry("list_capacity", list_capacity)
    eng.Attach(w)
    eng.Run(1)
    eng.SetConfigEntry("list_capacity", 3)
    eng.SetConfigEntry("grid_blocks", 50)
    eng.Run(2)
    assert np.array_equal(w.x, ref.x) and np.array_equal(w.v, ref.v) and np.array_equal(w.f, ref.f)
