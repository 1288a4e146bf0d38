"""A grid build whose look-backs do not wait at all (a tile whose predecessors have
not answered counts their elements itself): the same order, positions and lists."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
RECOUNTS = 16  # the handle's counter of tiles that counted for themselves


@pytest.mark.parametrize("n", [1025, 40000, 300000, 1000000])
def test_expired_look_back_counts_for_itself(capi, n):
    import torch

    lib = capi.lib()
    lib.egt_internal_set_polls.argtypes = [C.c_void_p, C.c_int, C.c_int]
    lib.egt_internal_counter.restype = C.c_int64
    lib.egt_internal_counter.argtypes = [C.c_void_p, C.c_int]
    g = np.random.Generator(np.random.PCG64(n))
    x = g.uniform(0, 1, (n, 3)).astype(np.float32)
    x[: n // 3] = 0.4 + 0.01 * x[: n // 3]
    t = torch.from_numpy(x).cuda()
    h = capi.GridStructure(x)
    h.GRIDCUDAKNNSELF_COMPACT(6)
    want = (h.GetOriginalRefIndexes(), h.sorted_positions(), h.sorted_lists())
    assert lib.egt_internal_counter(h.handle, RECOUNTS) == 0
    recounts = 0
    for polls in (0, 1, -1):
        lib.egt_internal_set_polls(h.handle, 0, polls)
        before = lib.egt_internal_counter(h.handle, RECOUNTS)
        for _ in range(3):
            h.UpdatePointsDevice(t.data_ptr())
            h.GRIDCUDAKNNSELF_COMPACT(6)
            for a, b in zip((h.GetOriginalRefIndexes(), h.sorted_positions(), h.sorted_lists()), want):
                assert np.array_equal(a, b)
        if polls == 0:
            recounts = lib.egt_internal_counter(h.handle, RECOUNTS) - before
        if polls < 0:
            assert lib.egt_internal_counter(h.handle, RECOUNTS) == before
    assert recounts > 0 or n < 40000
    h.close()
