"""The cell-tile search at the ends of its forms (k up to 22, 40, 64, and the
smallest k it takes) and of its cloud sizes, on surfaces, in a volume and on a
curve (most candidates below the bucket range), against the ring search taken
step by step (EGT_KNN_PLAIN): identical lists, invalid rows and deepest level."""
import numpy as np
import pytest

from multigpuegtsmoothing_b200 import datagen

pytestmark = pytest.mark.gpu


def _cloud(shape, n):
    g = np.random.Generator(np.random.PCG64(n))
    if shape == "volume":
        return g.uniform(0, 1, (n, 3)).astype(np.float32)
    if shape == "curve":
        t = g.uniform(0, 6, n)
        x = np.stack([np.cos(t), np.sin(t), 0.1 * t], 1)
        x[n // 2:] = g.uniform(-1, 1, (n - n // 2, 3))
        return (x + 1e-4 * g.standard_normal((n, 3))).astype(np.float32)
    if shape == "copies":  # every point three times: equal distances in every row
        return np.repeat(g.uniform(0, 1, (n // 3 + 1, 3)), 3, axis=0)[:n].astype(np.float32)
    return datagen.sphere_cloud(n, 0.004, n)


@pytest.mark.parametrize("shape,n,k", [("sphere", 65536, 8), ("sphere", 65535, 8), ("volume", 66000, 15),
                                       ("curve", 70000, 12), ("volume", 50000, 16), ("sphere", 49999, 16),
                                       ("sphere", 50001, 22), ("volume", 51000, 23), ("curve", 52000, 40),
                                       ("volume", 53000, 41), ("sphere", 54001, 64), ("curve", 55000, 64),
                                       ("copies", 60000, 20), ("copies", 70000, 9)])
def test_tile_forms_match_ring_search(capi, shape, n, k):
    xyz = _cloud(shape, n)
    g = capi.GridStructure(xyz)
    r = capi.GridStructure(xyz, config=capi.default_config(knn_mode=0))
    for p in (g, r):
        p.GRIDCUDAKNNSELF_COMPACT(k)
    assert np.array_equal(g.sorted_lists(), r.sorted_lists())
    t, tr = g.timings(), r.timings()
    assert t["invalid_queries"] == tr["invalid_queries"]
    assert t["levels_used"] == tr["levels_used"]
    g.close()
    r.close()
