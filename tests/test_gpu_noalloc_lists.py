"""pdpd_step_noalloc's force kernel at its edges, bit for bit against the oracle: beads that do not
fill the last block, boxes whose neighbour rows wrap onto themselves, rows longer than a list holds
(a dense box: those beads are evaluated one by one), long boxes (positions far from 0 in FP32),
and several bead types with unsymmetric strengths."""

import numpy as np
import pytest

import oracle as O
import pdpd_engine as E
import pdpd_world as W

pytestmark = pytest.mark.gpu


def _types(w, seed):
    rng = np.random.default_rng(seed)
    n = w.n_beads
    w.conservative = rng.uniform(5, 60, (3, 3))
    w.dissipative = rng.uniform(1, 6, (3, 3))
    w.stationary = np.zeros(3, bool)
    w.polymer_types = [W.PolymerType([k]) for k in range(3)]
    t = rng.integers(0, 3, n).astype(np.uint8)
    w.poly_type, w.bead_type, w.polymer_type_of_bead = t.astype(np.uint32), t, t
    return w


WORLDS = {
    "one_bead": lambda: W.make_water((2, 2, 2), seed=81, density=0.125),
    "partial_block": lambda: W.make_water((5, 3, 4), seed=82),
    "side_2": lambda: W.make_water((2, 2, 3), seed=83),
    "long_rows": lambda: W.make_water((4, 3, 4), seed=84, density=40, a=1.0, dt=0.001),
    "long_box": lambda: W.make_water((2, 4, 4000), seed=85, density=2),
    "three_types": lambda: _types(W.make_water((6, 7, 5), seed=86), 87),
}


@pytest.mark.parametrize("name", sorted(WORLDS))
def test_noalloc_lists_bit_exact(name):
    torch = pytest.importorskip("torch")
    w = WORLDS[name]()
    o = O.OracleWorld(w)
    o.run(4, nthreads=8)
    dev = torch.device("cuda", 0)
    x, v, f = (torch.from_numpy(a.copy()).to(dev) for a in (w.x, w.v, w.f))
    h = torch.from_numpy(w.hashes().view(np.int32).copy()).to(dev)
    for k in range(2):
        E.step_noalloc(w, x.data_ptr(), v.data_ptr(), f.data_ptr(), h.data_ptr(), 2, t=2 * k)
    for a, b in ((x, o.x), (v, o.v), (f, o.f)):
        assert np.array_equal(a.cpu().numpy(), b)


def _clump(seed, n_in, edge):
    w = W.make_water((6, 5, 7), seed=seed, density=4, a=0.3, gamma=0.5, dt=0.0005)
    w.x[:n_in] = 1.3 + edge * np.random.default_rng(seed).random((n_in, 3))
    return w


# (26 candidates in a row; more than the list holds at once; a whole box of such beads)
CLUMPS = {"few_long": (88, 60, 1.0), "many_refills": (89, 700, 0.9), "spread": (90, 800, 2.5)}


@pytest.mark.parametrize("name", sorted(CLUMPS))
def test_noalloc_long_beads_beside_others(name):
    torch = pytest.importorskip("torch")
    w = _clump(*CLUMPS[name])
    o = O.OracleWorld(w)
    o.run(3, nthreads=8)
    x, v, f = (torch.from_numpy(a.copy()).to("cuda:0") for a in (w.x, w.v, w.f))
    h = torch.from_numpy(w.hashes().view(np.int32).copy()).to("cuda:0")
    E.step_noalloc(w, x.data_ptr(), v.data_ptr(), f.data_ptr(), h.data_ptr(), 3, t=0)
    for a, b in ((x, o.x), (v, o.v), (f, o.f)):
        assert np.array_equal(a.cpu().numpy(), b)
