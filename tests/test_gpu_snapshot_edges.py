"""v2binary snapshots at the encoder's edges, byte for byte against the codec's restatement: worlds
of one record, of a tile's 64 records and one more, boxes whose positions round up to the box
side, vectors at the format's limits in FP32 (exponents at both ends, mantissas that round up to
256, subnormals), and polymers that put their headers between the records."""

import numpy as np
import pytest

import pdpd_engine as E
import pdpd_world as W
import v2binary as V

pytestmark = pytest.mark.gpu


def _edge_vectors(w, rng):
    n = w.n_beads
    e = rng.integers(-20, 14, n)
    m = rng.choice([1.0, 0.5, 255.5 / 256, 255.4999 / 256, 0.75, 511.0 / 512], (n, 3)) * rng.choice([-1, 1], (n, 3))
    v = (m * 2.0 ** e[:, None]).astype(np.float32).astype(np.float64)
    v[rng.random((n, 3)) < 0.2] = 0.0
    v[::17] = np.float32(1e-42)
    return v


def _world(kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "polymers":
        w = W.make_polymer_box((7, 5, 9), chain_fraction=0.4, seed=seed)
    else:
        n = {"one": 1, "tile": 64, "tile_and_one": 65, "many": 4000}[kind]
        w = W.make_water((11, 13, 4), seed=seed, density=n / (11 * 13 * 4.0) + 1e-9)
        assert w.n_beads == n
    w.v, w.f = _edge_vectors(w, rng), _edge_vectors(w, rng)
    L = np.asarray(w.box, float)
    at = rng.random((w.n_beads, 3)) < 0.1
    # just below a cell face: rounds up to the face, and at the box side to 0
    w.x = np.where(at, np.minimum(np.floor(w.x) + 1.0, L) - 2.0 ** -20, w.x)
    return w


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("kind", ["one", "tile", "tile_and_one", "many", "polymers"])
def test_snapshot_edges(kind, prec):
    w = _world(kind, 91)
    eng = E.GB300DPDEngine(prec)
    eng.Attach(w)
    eng.v2binary_prepare()
    got = eng.v2binary_encode()
    x, v, f, _ = eng.read_state(0)  # (what the engine holds: FP32 offsets in the FP32 engine)
    ref = w.copy()
    ref.x, ref.v, ref.f = x, v, f
    assert got.tobytes() == V.encode_section(ref)
