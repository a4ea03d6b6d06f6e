"""Engines of one process beside each other: what one engine sets up for its batch leaves the
others' kernels as they were."""

import numpy as np
import pytest

import pdpd_engine as E
import pdpd_world as W

pytestmark = pytest.mark.gpu

# A larger box, then a smaller one of the same kernel whose blocks take less shared memory.
PAIRS = {
    "fp32": ("fp32", {}, 48, 30),
    "fp32_three_lanes": ("fp32", {}, 16, 5),
    "fp32_variant_6": ("fp32", {"force_kernel": 6}, 30, 6),
    "fp32_half_shell": ("fp32", {"force_kernel": 9}, 30, (4, 4, 2)),
    "fp64": ("fp64", {}, 48, 30),
    "fp64_three_lanes": ("fp64", {}, 16, 5),
}


@pytest.mark.parametrize("graphs", [0, 1])
@pytest.mark.parametrize("name", sorted(PAIRS))
def test_a_smaller_batch_of_another_engine_leaves_an_attached_one_runnable(name, graphs):
    prec, config, large, small = PAIRS[name]

    def engine(world):
        e = E.GB300DPDEngine(prec)
        e.SetConfigEntry("use_graphs", graphs)
        for k, v in config.items():
            e.SetConfigEntry(k, v)
        e.Attach(world)
        return e

    w = W.make_water(large, seed=81, dt=0.005)
    alone, beside = w.copy(), w.copy()
    engine(alone).Run(4)
    a = engine(beside)
    b = engine(W.make_water(small, seed=82, dt=0.005))
    b.Run(2)
    a.Run(4)
    for k in "xvf":
        assert np.array_equal(getattr(alone, k), getattr(beside, k)), k
