"""A GPU with little memory left: the FP64 pair lists are optional and take none of what the engine
needs later."""

import numpy as np
import pytest

import pdpd_engine as E
import pdpd_world as W

pytestmark = pytest.mark.gpu

MB = 1 << 20


class _Filled:
    """Leaves `mb` MB of device memory free."""

    def __init__(self, torch, mb):
        torch.cuda.empty_cache()
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        self.torch, self.t = torch, torch.empty(max(0, free - mb * MB), dtype=torch.uint8, device="cuda:0")

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        del self.t
        self.torch.cuda.empty_cache()


def _everything(world, pair_lists):
    """Attach, runs, snapshot, read-backs through every later buffer; None if the attach finds no memory."""
    w = world.copy()
    eng = E.GB300DPDEngine("fp64")
    eng.SetConfigEntry("host_direct", 0)  # (a second staging buffer)
    eng.SetConfigEntry("pair_lists", pair_lists)
    try:
        eng.Attach(w)
    except RuntimeError as ex:
        assert "allocation" in str(ex), ex
        eng.close()
        return None
    try:
        eng.Run(3, 2, lambda: True)
        eng.v2binary_prepare()
        section = eng.v2binary_encode()
        eng.v2binary_decode(section)
        eng.log_pair_terms(np.arange(4, dtype=np.uint32))
    finally:
        eng.close()
    return w.x.copy()


def test_pair_lists_leave_room_for_the_other_buffers():
    torch = pytest.importorskip("torch")
    world = W.make_water(40, seed=99, dt=0.005)  # lists of about 100 MB
    ref = _everything(world, 0)
    least = None
    for mb in range(24, 400, 8):  # the least that a run without lists needs
        with _Filled(torch, mb):
            try:
                ok = _everything(world, 0) is not None
            except RuntimeError:
                ok = False
        if ok:
            least = mb
            break
    assert least is not None
    for mb in range(least + 8, least + 140, 12):
        with _Filled(torch, mb):
            x = _everything(world, 1)
        assert x is not None and np.array_equal(x, ref), mb
