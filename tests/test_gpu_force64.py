"""The FP64 force pass without pair lists (config ``pair_lists`` 0, and batches there is no room for
the lists of), bit for bit against the oracle: boxes of side 2, polymers (bonds beside the prefix
sum, one launch of it and two), dense and clustered beads (full candidate lists), unsymmetric
strengths, stationary types, per-cell strengths, mixed batches, and against the lists."""

import numpy as np
import pytest

import oracle as O
import pdpd_engine as E
import pdpd_world as W
from _helpers import load_world_fixture, merge_fixture_names, world_fixture_names
from test_gpu_pairs64 import WORLDS

pytestmark = pytest.mark.gpu


def _engine(worlds, list_capacity=0, pair_lists=0):
    eng = E.GB300DPDEngine("fp64")
    eng.SetConfigEntry("pair_lists", pair_lists)
    eng.SetConfigEntry("list_capacity", list_capacity)
    eng.AttachBatch(worlds)
    return eng


def _same(a, b):
    return all(np.array_equal(getattr(a, k), getattr(b, k)) for k in "xvf")


@pytest.mark.parametrize("list_capacity", [0, 3])
@pytest.mark.parametrize("name", sorted(WORLDS))
def test_bit_exact(name, list_capacity):
    w = WORLDS[name]()
    steps = 2 if w.n_beads > 100000 else 4
    o = O.OracleWorld(w)
    o.run(steps, nthreads=8)
    _engine([w], list_capacity).Run(steps)
    assert _same(w, o)


@pytest.mark.parametrize("name", world_fixture_names() + merge_fixture_names())
def test_fixtures(name):
    w, ref = load_world_fixture(name)
    steps = min(5, int(ref["checkpoints"][-1]))
    o = O.OracleWorld(w)
    o.run(steps, nthreads=8)
    _engine([w]).Run(steps)
    assert _same(w, o)


def test_mixed_batch_and_the_lists():
    names = [n for n in sorted(WORLDS) if n != "large_bricks"]
    a = [WORLDS[n]() for n in names]
    b = [w.copy() for w in a]
    oracles = [O.OracleWorld(w) for w in a]
    _engine(a).Run(3)
    _engine(b, pair_lists=1).Run(3)
    for n, x, y, o in zip(names, a, b, oracles):
        o.run(3)
        assert _same(x, o) and _same(y, o), n
