"""Kinds of batches that the default kernels once ran slower than another path of this engine does:
the default is timed against that path, with room for noise (the best of several runs of each)."""

import time

import pytest

import pdpd_engine as E
import pdpd_world as W

pytestmark = pytest.mark.gpu


def _water(box, density, seed=1):
    return W.make_water(box, seed=seed, density=density, a=1.0, gamma=4.5, dt=0.002)


def _step_us(prec, worlds, steps=6, **config):
    eng = E.GB300DPDEngine(prec)
    for k, v in config.items():
        eng.SetConfigEntry(k, v)
    eng.AttachBatch([w.copy() for w in worlds])
    best = 1e9
    for _ in range(6):
        t0 = time.perf_counter()
        eng.run_async(steps)
        eng.sync()
        best = min(best, time.perf_counter() - t0)
    return best / steps * 1e6


@pytest.mark.parametrize("box,density", [(24, 10), (24, 14), (20, 20)])
def test_dense_boxes_fp32(box, density):
    """Against the thread-per-bead kernel: 0.15-0.25 of its time; 0.65-0.75 when each lane of a warp
    flushed its walk segments on its own."""
    w = [_water(box, density)]
    assert _step_us("fp32", w) < 0.45 * _step_us("fp32", w, force_kernel=1)


@pytest.mark.parametrize("box,density", [(64, 0.05), (128, 0.05), (200, 0.01), (128, 0.5), (20, 0.3), (24, 6)])
def test_sparse_and_dense_boxes_fp64(box, density):
    """With pair lists and without, whichever is the faster; with lists at any density, 128^3 of
    density 0.05 took 3 times as long as without."""
    w = [_water(box, density)]
    best = min(_step_us("fp64", w, pair_lists=0), _step_us("fp64", w, pair_lists=2))
    assert _step_us("fp64", w) < 1.25 * best


def test_many_tiny_sparse_worlds_fp64():
    """Without pair lists, which took 1.3 times as long."""
    worlds = [_water(2, 0.125, k) for k in range(4000)]
    assert _step_us("fp64", worlds) < 1.12 * _step_us("fp64", worlds, pair_lists=0)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_a_dense_world_beside_a_large_sparse_one(prec):
    """Against the two one after the other: about as long; FP32 took 5 times as long when the densest
    world's brick shape was that of all."""
    dense, sparse = _water(6, 30, 1), _water(100, 0.1, 2)
    apart = _step_us(prec, [dense]) + _step_us(prec, [sparse])
    assert _step_us(prec, [dense, sparse]) < 1.4 * apart


def test_default_shape_of_the_narrow_kernel():
    """force_kernel 6 against itself on the bricks that suit it; 4.5 times as long on the largest, whose
    halo does not fit its blocks."""
    w = [_water(64, 3)]
    assert _step_us("fp32", w, force_kernel=6) < 1.3 * _step_us("fp32", w, force_kernel=6, brick_x=3, brick_y=4, brick_z=6)


@pytest.mark.parametrize("side,copies,config", [(2, 2000, {}), (3, 2000, {}), (32, 1, {"brick_x": 3, "brick_y": 3, "brick_z": 3})])
def test_many_bricks_of_few_beads(side, copies, config):
    """Against force_kernel 6, whose blocks have 128 threads; 1.3 to 1.9 times as long with 512."""
    worlds = [_water(side, 3, k) for k in range(copies)]
    assert _step_us("fp32", worlds, **config) < 1.15 * _step_us("fp32", worlds, force_kernel=6, **config)


@pytest.mark.parametrize("box,density", [(10, 20), (8, 60)])
def test_dense_boxes_noalloc(box, density):
    """pdpd_step_noalloc against the FP64 engine without pair lists, a thread per bead: 0.05-0.15 of its
    time; 0.4-0.5 when one lane evaluated all pairs of a bead whose candidates did not fit."""
    torch = pytest.importorskip("torch")
    w = _water(box, density)
    x, v, f = (torch.from_numpy(a.copy()).to("cuda:0") for a in (w.x, w.v, w.f))
    h = torch.from_numpy(w.hashes().view("int32").copy()).to("cuda:0")
    best = 1e9
    for k in range(4):
        t0 = time.perf_counter()
        E.step_noalloc(w, x.data_ptr(), v.data_ptr(), f.data_ptr(), h.data_ptr(), 4, t=4 * k)
        best = min(best, (time.perf_counter() - t0) / 4 * 1e6)
    none = _step_us("fp64", [w], pair_lists=0)
    assert best < 0.3 * none


@pytest.mark.parametrize("side,density", [(24, 3), (16, 8)])
def test_fp64_force_pass_without_lists_of_few_tiles(side, density):
    """Per bead, against a box of many more tiles than SMs: 2.7 and 3.1 times as long when the blocks of
    the small box crowded on a few SMs, 1.8 and 1.4 spread evenly."""
    small, large = _water(side, density), _water(2 * side, density)
    per_bead = [_step_us("fp64", [w], pair_lists=0, steps=4) / w.n_beads for w in (small, large)]
    assert per_bead[0] < 2.25 * per_bead[1]


def test_bricks_of_a_small_batch_spread_over_the_sms():
    """A brick per SM, against force_kernel 6 on smaller ones: 0.82 of its time, 1.05 with two bricks on
    some SMs and none on others."""
    w = [_water(25, 3)]
    assert _step_us("fp32", w, steps=20) < 0.93 * _step_us("fp32", w, steps=20, force_kernel=6)


def test_attach_of_many_worlds():
    """FP64 against FP32, whose host work is nearly the same: 1.0; 1.3 when the brick shape's estimate
    ran over every world for every shape."""
    def attach_us(eng, worlds):
        t0 = time.perf_counter()
        eng.AttachBatch(worlds)
        return (time.perf_counter() - t0) * 1e6

    worlds = [_water((5 + k % 5, 6 + k % 3, 7 + k % 4), 3, k) for k in range(300)]
    engines = [E.GB300DPDEngine(prec) for prec in ("fp64", "fp32")]
    us = [[attach_us(eng, worlds) for eng in engines] for _ in range(25)]  # in turn
    fp64, fp32 = map(min, zip(*us))
    assert fp64 < 1.17 * fp32


def test_an_uneven_large_box():
    """80% of the beads in a fifth of the box, against smaller bricks: 1.9 times as long in the default
    ones of its mean density."""
    import numpy as np

    w = _water(64, 3)
    n, rng = w.n_beads * 4 // 5, np.random.default_rng(1)
    w.x[:n, 2], w.x[n:, 2] = 12.8 * rng.random(n), 12.8 + 51.2 * rng.random(w.n_beads - n)
    assert _step_us("fp32", [w]) < 1.35 * _step_us("fp32", [w], brick_x=4, brick_y=4, brick_z=6)


def test_most_beads_in_full_bricks():
    """A box beside a sparse one whose bricks outnumber its own, against force_kernel 8: 1.33 times as long
    when the bricks' mean, not the beads', chose the blocks."""
    worlds = [_water((15, 16, 22), 3), _water((32, 49, 26), 0.07, 2)]
    assert _step_us("fp32", worlds, steps=20) < 1.15 * _step_us("fp32", worlds, steps=20, force_kernel=8)


@pytest.mark.parametrize("box,copies,shape", [((37, 25, 19), 56, (5, 8, 8)), ((41, 33, 27), 8, (4, 4, 6))])
def test_batches_of_uneven_boxes(box, copies, shape):
    """Density falling as 1/sqrt(z), against the bricks that suit the batch; the small boxes took 1.2 times
    as long in 4x4x6, the others in the default ones of their mean density."""
    worlds = [_water(box, 3, k) for k in range(copies)]
    for w in worlds:
        w.x[:, 2] = w.x[:, 2] ** 2 / box[2]
    best = _step_us("fp32", worlds, steps=4, **dict(zip(("brick_x", "brick_y", "brick_z"), shape)))
    assert _step_us("fp32", worlds, steps=4) < 1.1 * best


def test_a_dense_uneven_world_beside_others_fp64():
    """Against the two one after the other: as long; 1.5 times when the dense world had the bricks of the
    batch's size, and the last of them were waited for."""
    dense, others = _water((30, 24, 24), 6.28), [_water(24, 1, k) for k in range(8)]
    dense.x[:, 2] = dense.x[:, 2] ** 2 / 24
    apart = _step_us("fp64", [dense], steps=3) + _step_us("fp64", others, steps=3)
    assert _step_us("fp64", [dense] + others, steps=3) < 1.25 * apart


def test_a_dense_world_behind_others_fp64():
    """Against the dense world in front: the same time; 1.11 times when its bricks were the pass's last."""
    dense, others = _water(22, 10), [_water(20, 0.7, k) for k in range(50)]
    assert _step_us("fp64", others + [dense]) < 1.06 * _step_us("fp64", [dense] + others)


@pytest.mark.parametrize("box,copies,density", [((11, 9, 14), 100, 0.05), ((11, 9, 14), 100, 0.15), ((6, 6, 6), 1000, 0.25)])
def test_sparse_worlds_that_fill_their_bricks_badly_fp64(box, copies, density):
    """Without pair lists, which took 1.46, 1.34 and 1.24 times as long."""
    worlds = [_water(box, density, k) for k in range(copies)]
    assert _step_us("fp64", worlds) < 1.12 * _step_us("fp64", worlds, pair_lists=0)


@pytest.mark.parametrize("boxes", [[((41, 67, 65), 0.16), ((11, 11, 13), 3)], [((64, 75, 100), 0.45)]])
def test_a_few_full_bricks_among_many(boxes):
    """A box of density 3 beside a sparse one, and a sparse box whose density falls as 1/sqrt(z), against
    force_kernel 8: 1.6 times as long in blocks of 128 threads."""
    worlds = [_water(box, density, k) for k, (box, density) in enumerate(boxes)]
    if len(worlds) == 1:
        worlds[0].x[:, 2] = worlds[0].x[:, 2] ** 2 / worlds[0].box[2]
    assert _step_us("fp32", worlds, steps=20) < 1.15 * _step_us("fp32", worlds, steps=20, force_kernel=8)


def test_an_uneven_box_of_low_density():
    """Density 1 falling as 1/sqrt(z), against the default bricks for even boxes; 1.12 times as long in
    smaller ones."""
    w = _water((64, 75, 100), 1)
    w.x[:, 2] = w.x[:, 2] ** 2 / 100
    assert _step_us("fp32", [w]) < 1.06 * _step_us("fp32", [w], brick_x=5, brick_y=8, brick_z=8)


def test_a_small_dense_world_beside_a_sparse_one_fp64():
    """With pair lists; 1.37 times as long without, for the few beads of the dense world."""
    worlds = [_water((63, 53, 91), 0.11), _water((10, 9, 8), 3, 2)]
    assert _step_us("fp64", worlds) < 1.15 * _step_us("fp64", worlds, pair_lists=2)


def test_an_uneven_box_of_high_density():
    """Density 5 falling as 1/sqrt(z), against 3x4x4 bricks; 1.3 times as long in 4x4x6."""
    w = _water(60, 5)
    w.x[:, 2] = w.x[:, 2] ** 2 / 60
    assert _step_us("fp32", [w]) < 1.12 * _step_us("fp32", [w], brick_x=3, brick_y=4, brick_z=4)


def test_an_uneven_world_among_even_ones():
    """Against 4x4x6 bricks for the whole batch; 2 times as long when the uneven world's crowded cells were
    too few of the batch to count."""
    worlds = [_water(box, 3, k) for k, box in enumerate([(43, 44, 40), (34, 46, 31), (26, 34, 41), (31, 16, 29)])]
    worlds[3].x[:, 2] = worlds[3].x[:, 2] ** 2 / 29
    assert _step_us("fp32", worlds) < 1.2 * _step_us("fp32", worlds, brick_x=4, brick_y=4, brick_z=6)


@pytest.mark.parametrize("uneven,even,copies", [((37, 28, 33), (58, 35, 46), 1), ((30, 30, 30), (36, 36, 36), 2), ((24, 24, 24), (40, 40, 40), 1)])
def test_a_batch_of_a_few_boxes_with_an_uneven_one(uneven, even, copies):
    """Against 4x5x8 bricks; the first two 1.15 to 1.25 times as long when the uneven box had smaller ones."""
    worlds = [_water(uneven, 3)] + [_water(even, 3, 2 + k) for k in range(copies)]
    worlds[0].x[:, 2] = worlds[0].x[:, 2] ** 2 / uneven[2]
    assert _step_us("fp32", worlds) < 1.1 * _step_us("fp32", worlds, brick_x=4, brick_y=5, brick_z=8)
