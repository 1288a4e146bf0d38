"""A resident Taubin loop whose waits expire (the limit set to one poll) still
ends with the loop's result: the half-steps are computed again without waits,
the same positions bit for bit, and the handle works on."""
import ctypes as C

import numpy as np
import pytest

from multigpuegtsmoothing_b200 import datagen

pytestmark = pytest.mark.gpu
REDONE = 31  # the handle's counter of loops computed again


def _counter(lib, handle, word):
    lib.egt_internal_counter.restype = C.c_int64
    lib.egt_internal_counter.argtypes = [C.c_void_p, C.c_int]
    return lib.egt_internal_counter(handle, word)


@pytest.mark.parametrize("n,iters", [(2500, 7), (36001, 5)])
def test_expired_wait_is_computed_again(capi, n, iters):
    lib = capi.lib()
    lib.egt_internal_set_polls.argtypes = [C.c_void_p, C.c_int, C.c_int]
    xyz = datagen.sphere_cloud(n, 0.005, n)
    out = []
    for polls in (0, 1):
        g = capi.GridStructure(xyz)
        g.GRIDCUDAKNNSELF_COMPACT(24)
        egt = capi.EGT_CUDA(g)
        egt.Filter(0.65)
        lib.egt_internal_set_polls(g.handle, polls, -1)
        egt.Taubin(iters, 0.63, -0.64)
        first = g.sorted_positions()
        redone = _counter(lib, g.handle, REDONE)
        assert redone == 0 if polls == 0 else redone == 1
        lib.egt_internal_set_polls(g.handle, 0, -1)
        egt.Taubin(iters, 0.63, -0.64)  # the next loop is not touched by the expired one
        g.timings()
        assert _counter(lib, g.handle, REDONE) == redone
        out.append((first, g.sorted_positions(), np.stack(capi.getOutputPoints(g))))
        g.close()
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.array_equal(a, b)
