"""Batches of worlds of very different densities, whose bricks have different shapes: each world as
it is alone."""

import numpy as np
import pytest

import oracle as O
import pdpd_engine as E
import pdpd_world as W

pytestmark = pytest.mark.gpu

BATCHES = {
    "dense_beside_sparse": [((6, 6, 6), 30), ((40, 41, 39), 0.1)],
    "dense_among_many": [((20, 21, 19), 3), ((9, 8, 10), 14), ((22, 20, 24), 3), ((5, 4, 5), 45), ((20, 20, 20), 3)],
    "sparse_among_dense": [((12, 11, 12), 12), ((30, 30, 31), 0.02), ((12, 12, 13), 12)],
    "empty_and_dense": [((5, 6, 5), 20), ((16, 16, 16), 1.0 / 4096), ((2, 2, 2), 60)],
}


@pytest.mark.parametrize("config", [{}, {"force_kernel": 8}, {"brick_x": 3, "brick_y": 4, "brick_z": 5}, {"autotune": 1}])
@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("name", sorted(BATCHES))
def test_batches_of_mixed_density(name, prec, config):
    worlds = [W.make_water(box, seed=90 + k, density=rho, a=0.5, dt=0.001) for k, (box, rho) in enumerate(BATCHES[name])]
    ref = [w.copy() for w in worlds]
    steps = 40 if "autotune" in config else 3  # (the trials are steps of the run)
    if prec == "fp64":
        ref = [O.OracleWorld(w) for w in ref]
        for o in ref:
            o.run(steps, nthreads=8)
    else:
        for w in ref:
            eng = E.GB300DPDEngine("fp32")
            eng.SetConfigEntry("force_kernel", 1)
            eng.Attach(w)
            eng.Run(steps)
    eng = E.GB300DPDEngine(prec)
    for k, v in config.items():
        eng.SetConfigEntry(k, v)
    eng.AttachBatch(worlds)
    eng.Run(steps)
    for w, o in zip(worlds, ref):
        assert np.array_equal(w.x, o.x) and np.array_equal(w.v, o.v) and np.array_equal(w.f, o.f)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_a_dense_world_does_not_enlarge_the_others(prec):
    """Device memory of a small dense world and a large sparse one in a batch: what the two take one by
    one (the buckets of all cells were as large as the densest world's: 200 MB more here)."""
    torch = pytest.importorskip("torch")

    def taken(worlds):
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        eng = E.GB300DPDEngine(prec)
        eng.AttachBatch(worlds)
        eng.Run(1)
        return free - torch.cuda.mem_get_info()[0]

    dense, sparse = W.make_water(6, seed=95, density=30, a=0.5, dt=0.001), W.make_water(100, seed=96, density=0.1, dt=0.001)
    taken([dense.copy()])  # (the context's own allocations)
    apart = taken([dense.copy()]) + taken([sparse.copy()])
    assert taken([dense, sparse]) <= apart + (24 << 20)


def test_an_uneven_box_gets_other_bricks_between_runs():
    """A box whose density varies over it (its beads overflow their cells' buckets): the same state to the
    bit as by the thread-per-bead kernel, from the first run on and after the bricks have changed."""
    a = W.make_water(40, seed=97, a=1.0, dt=0.001)
    a.x[:, 2] = a.x[:, 2] ** 3 / 1600
    b = a.copy()
    eng, ref = E.GB300DPDEngine("fp32"), E.GB300DPDEngine("fp32")
    ref.SetConfigEntry("force_kernel", 1)
    eng.Attach(a)
    ref.Attach(b)
    shapes = set()
    for steps in (1, 3, 2):
        eng.Run(steps)
        ref.Run(steps)
        shapes.add(tuple(v for n, _, v in eng.GetConfigEntries() if n.startswith("brick_")))
        assert np.array_equal(a.x, b.x) and np.array_equal(a.v, b.v) and np.array_equal(a.f, b.f)
    assert ("4", "4", "6") in shapes


def test_an_uneven_world_gets_other_bricks_among_even_ones():
    """The same as the thread-per-bead kernel's to the bit, before and after the host has seen which world
    is uneven."""
    boxes = [(20, 21, 19), (41, 40, 39), (3, 4, 3), (26, 25, 27), (40, 38, 41)]
    a = [W.make_water(box, seed=60 + k, a=1.0, dt=0.001) for k, box in enumerate(boxes)]
    a[3].x[:, 2] = a[3].x[:, 2] ** 3 / 27**2
    b = [w.copy() for w in a]
    eng, ref = E.GB300DPDEngine("fp32"), E.GB300DPDEngine("fp32")
    ref.SetConfigEntry("force_kernel", 1)
    eng.AttachBatch(a)
    ref.AttachBatch(b)
    for steps in (1, 3, 2):
        eng.Run(steps)
        ref.Run(steps)
        for w, o in zip(a, b):
            assert np.array_equal(w.x, o.x) and np.array_equal(w.v, o.v) and np.array_equal(w.f, o.f)


def test_an_uneven_batch_leaves_no_mark_on_the_next():
    """An even box attached after an uneven one has the bricks of an even box."""
    def shape(eng):
        return tuple(v for n, _, v in eng.GetConfigEntries() if n.startswith("brick_"))

    even = [W.make_water(40, seed=k, a=1.0, dt=0.001) for k in range(2)]
    uneven = even[0].copy()
    uneven.x[:, 2] = uneven.x[:, 2] ** 3 / 1600
    fresh, eng = E.GB300DPDEngine("fp32"), E.GB300DPDEngine("fp32")
    fresh.Attach(even[0])
    fresh.Run(1)
    fresh.Run(1)
    for w in (uneven, even[1]):
        eng.Attach(w)
        eng.Run(1)
        eng.Run(1)
    assert shape(eng) == shape(fresh)
