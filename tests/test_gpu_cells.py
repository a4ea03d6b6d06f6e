"""The cell-list rebuild where it changes path: cells that hold as many beads as their bucket has
room for, one more, and many more (the overflow lists), and cell counts at the edges of the
one-kernel prefix sum (16 chunks of 2,048 cells)."""

import numpy as np
import pytest

import oracle as O
import pdpd_engine as E
import pdpd_world as W

pytestmark = pytest.mark.gpu


def _clumps(counts, seed):
    """A 6^3 box of density about 3 whose first cells hold the given numbers of beads."""
    w = W.make_water(6, seed=seed, a=0.5, gamma=0.5, dt=0.001)
    rng = np.random.default_rng(seed)
    at = 0
    for k, n in enumerate(counts):
        cell = np.array([k // 6, k % 6, (3 * k) % 6], float)
        w.x[at:at + n] = cell + 0.01 + 0.98 * rng.random((n, 3))
        at += n
    assert at <= w.n_beads
    return w


COUNTS = [15, 16, 17, 18, 33, 64, 65, 130]


def _run(worlds, prec, steps):
    eng = E.GB300DPDEngine(prec)
    eng.AttachBatch(worlds)
    eng.Run(steps)


def test_full_and_overflowing_cells_fp64():
    w = _clumps(COUNTS, 71)
    o = O.OracleWorld(w)
    o.run(3)
    _run([w], "fp64", 3)
    assert np.array_equal(w.x, o.x) and np.array_equal(w.v, o.v) and np.array_equal(w.f, o.f)


def test_full_and_overflowing_cells_fp32():
    """Alone the clumped cells overflow their buckets; beside a dense world, which gives the
    batch larger buckets, fewer do: the same state to the bit."""
    a = _clumps(COUNTS, 72)
    b, dense = a.copy(), W.make_water((3, 4, 3), seed=73, a=0.5, density=24, dt=0.001)
    _run([a], "fp32", 3)
    _run([dense, b], "fp32", 3)
    assert np.array_equal(a.x, b.x) and np.array_equal(a.v, b.v) and np.array_equal(a.f, b.f)


@pytest.mark.parametrize("box", [(2, 2, 512), (32, 32, 32), (31, 33, 32), (32, 32, 33), (2, 5, 3277), (64, 64, 9)])
def test_prefix_sum_edges(box):
    w = W.make_water(box, seed=74, density=0.5)
    o = O.OracleWorld(w)
    o.run(2, nthreads=8)
    _run([w], "fp64", 2)
    assert np.array_equal(w.x, o.x) and np.array_equal(w.f, o.f)


@pytest.mark.parametrize("copies", [4, 12])
def test_bond_lanes_per_bead(copies):
    """6,144 polymer beads alone (eight lanes each), four and twelve times that in one batch (two
    lanes, one): the same state to the bit."""
    a = W.make_polymer_box(16, chain_fraction=0.5, seed=75, dt=0.001, theta0=0.3)
    batch = [a.copy() for _ in range(copies)]
    _run([a], "fp32", 3)
    _run(batch, "fp32", 3)
    for b in batch:
        assert np.array_equal(a.x, b.x) and np.array_equal(a.v, b.v) and np.array_equal(a.f, b.f)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("box,density", [
    ((3, 3, 3), 3), ((8, 16, 32), 1), ((8, 16, 32), 4097.5 / 4096), ((16, 16, 16), 3), ((16, 16, 16), 12289.5 / 4096),
    ((2, 5, 409), 0.5), ((2, 5, 410), 0.5), ((2, 3, 2), 60)])
def test_one_kernel_rebuild_edges(prec, box, density):
    """The one-kernel rebuild's limits (4,096 cells; 4,096 beads in FP64, 12,288 in FP32) and buckets
    that overflow, against the same box in a batch too large for it: the same state to the bit."""
    w = W.make_water(box, seed=76, a=0.5, gamma=0.5, density=density, dt=0.001)
    a, b, big = w.copy(), w.copy(), W.make_water((16, 16, 17), seed=77, density=0.1)
    _run([a], prec, 3)
    _run([b, big], prec, 3)
    assert np.array_equal(a.x, b.x) and np.array_equal(a.v, b.v) and np.array_equal(a.f, b.f)
    if prec == "fp64":
        o = O.OracleWorld(w)
        o.run(3, nthreads=8)
        assert np.array_equal(a.x, o.x) and np.array_equal(a.v, o.v) and np.array_equal(a.f, o.f)
