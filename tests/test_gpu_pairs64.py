"""The FP64 engine's pair lists, bit for bit against the oracle where they can go wrong: boxes so
small that a pair is met at several images or every pair lies across a face, unsymmetric
strengths (evaluated from both sides), beads of bricks too full to stage or with more candidates
than their walk segments hold, batches whose lists do not fit in the room reserved for them (a
clustered world), sparse and dense boxes, and mixed batches."""

import numpy as np
import pytest

import oracle as O
import pdpd_engine as E
import pdpd_world as W

pytestmark = pytest.mark.gpu


def _water(box, seed, density=3, a=25.0, dt=0.01):
    return W.make_water(box, seed=seed, density=density, a=a, dt=dt)


def _clustered(side, seed):
    w = _water(side, seed, dt=0.002)
    rng = np.random.default_rng(seed)
    n = w.n_beads * 2 // 3
    w.x[:n] = 0.3 + 1.6 * rng.random((n, 3))
    return w


def _unsymmetric(seed):
    w = W.make_polymer_box((5, 6, 4), chain_fraction=0.3, seed=seed)
    w.conservative[0, 2] = 40.0
    w.dissipative[1, 0] = 5.5
    return w


WORLDS = {
    "side_2": lambda: _water((2, 2, 2), 61),
    "side_2_by_3_by_9": lambda: _water((2, 3, 9), 62),
    "sparse": lambda: _water((9, 8, 10), 63, density=0.3),
    "dense": lambda: _water((5, 4, 6), 64, density=14, a=4.0, dt=0.002),
    "clustered": lambda: _clustered(9, 65),
    "unsymmetric": lambda: _unsymmetric(66),
    "polymer_uneven": lambda: W.make_polymer_box((13, 7, 10), chain_fraction=0.3, seed=67, theta0=0.2),
    "large_bricks": lambda: W.make_polymer_box((62, 59, 57), chain_fraction=0.05, seed=68),
}


@pytest.mark.parametrize("list_capacity", [0, 3])
@pytest.mark.parametrize("name", sorted(WORLDS))
def test_pair_lists_bit_exact(name, list_capacity):
    world = WORLDS[name]()
    steps = 2 if world.n_beads > 100000 else 4
    ow = O.OracleWorld(world)
    ow.run(steps, nthreads=8)
    eng = E.GB300DPDEngine("fp64")
    eng.SetConfigEntry("list_capacity", list_capacity)  # 3: many beads' segments do not fit
    eng.Attach(world)
    eng.Run(steps)
    assert np.array_equal(world.x, ow.x) and np.array_equal(world.v, ow.v) and np.array_equal(world.f, ow.f)


def test_pair_lists_of_a_mixed_batch():
    names = [n for n in sorted(WORLDS) if n != "large_bricks"]
    worlds = [WORLDS[n]() for n in names]
    oracles = [O.OracleWorld(w) for w in worlds]
    eng = E.GB300DPDEngine("fp64")
    eng.AttachBatch(worlds)
    eng.Run(3)
    for n, w, o in zip(names, worlds, oracles):
        o.run(3)
        assert np.array_equal(w.x, o.x) and np.array_equal(w.v, o.v) and np.array_equal(w.f, o.f), n


@pytest.mark.parametrize("side", [14, 20, 24, 27])
def test_lanes_per_bead_of_small_and_larger_boxes(side):
    """Three lanes per bead up to 24^3, each shape of brick; one above.  The small worlds beside a
    larger box, one lane per bead for all of them."""
    names = [n for n in sorted(WORLDS) if n not in ("large_bricks", "dense")] if side == 27 else []
    worlds = [WORLDS[n]() for n in names] + [W.make_polymer_box(side, chain_fraction=0.1, seed=69, dt=0.005)]
    oracles = [O.OracleWorld(w) for w in worlds]
    eng = E.GB300DPDEngine("fp64")
    eng.AttachBatch(worlds)
    eng.Run(2)
    for w, o in zip(worlds, oracles):
        o.run(2, nthreads=8)
        assert np.array_equal(w.x, o.x) and np.array_equal(w.v, o.v) and np.array_equal(w.f, o.f)
