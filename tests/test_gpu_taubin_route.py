"""Which loop a small cloud's smoothing takes: one resident launch where every
tile's neighbours are staged, a launch per half-step where some tile gathers
from global memory (rows that poll each neighbour through L2 are slower)."""
import numpy as np
import pytest

from multigpuegtsmoothing_b200 import datagen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,alpha", [(5000, 24, None), (5000, 24, 0.65), (5000, 12, None), (20000, 40, 0.1)])
def test_spilled_tiles_take_launches(capi, n, k, alpha):
    iters = 20
    g = capi.GridStructure(datagen.sphere_cloud(n, 0.005, n))
    g.GRIDCUDAKNNSELF_COMPACT(k)
    egt = capi.EGT_CUDA(g)
    if alpha:
        egt.Filter(alpha)
    for _ in range(2):  # the tables are built in the first call and kept in the second
        before = capi.kernel_launches()
        egt.Taubin(iters)
        launches = capi.kernel_launches() - before
        t = g.timings()
        assert t["taubin_tiles"] == (n + 255) // 256
        if t["taubin_spill_tiles"]:
            assert launches >= 2 * iters
        else:
            assert launches < 2 * iters
    assert np.isfinite(g.sorted_positions()).all()
    assert (t["taubin_spill_tiles"] > 0) == (alpha != 0.65 and k > 18)
    g.close()
