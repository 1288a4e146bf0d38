"""Paths of the searches that other tests' sizes no longer reach: the chunked host
search (several chunks on two streams), the tiles' rejection of equal distances,
and their certificates off the surfaces; knn_fallback's one meaning."""
import numpy as np
import pytest

from multigpuegtsmoothing_b200 import datagen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,k", [(0, 40), (3, 5), (3, 65), (3, 97), (2, 100)])
def test_chunked_host_lists(capi, mode, k):
    """262,144 points or more run as nine chunks where the default does not take the tiles."""
    xyz = datagen.superquadrics(300_000, seed=11)
    g = capi.GridStructure(xyz, config=capi.default_config(knn_mode=mode))
    g.GRIDCUDAKNNSELF_COMPACT(k)
    want, lists, t = g.GetKNNIndexes(), g.sorted_lists(), g.timings()
    g.close()
    g = capi.GridStructure(xyz, config=capi.default_config(knn_mode=mode))
    for _ in range(2):  # the second call reuses the handle's buffers
        assert np.array_equal(g.knn_host(k), want)
        assert np.array_equal(g.sorted_lists(), lists)
        t2 = g.timings()
        for key in ("invalid_queries", "levels_used", "knn_fallback", "exact_reruns"):
            assert t2[key] == t[key], key
    g.close()


def _shape(shape, n):
    g = np.random.Generator(np.random.PCG64(n))
    if shape == "lattice":
        m = round(n ** (1 / 3))
        return (np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3) / 8.0).astype(np.float32)
    if shape == "copies":
        return np.repeat(g.uniform(0, 1, (n // 3 + 1, 3)), 3, axis=0)[:n].astype(np.float32)
    if shape == "volume":
        return g.uniform(0, 1, (n, 3)).astype(np.float32)
    t = g.uniform(0, 6, n)  # a curve in a sparse cube
    x = np.stack([np.cos(t), np.sin(t), 0.1 * t], 1)
    x[n // 2:] = g.uniform(-1, 1, (n - n // 2, 3))
    return (x + 1e-4 * g.standard_normal((n, 3))).astype(np.float32)


@pytest.mark.parametrize("shape,n,k", [("lattice", 64000, 26), ("copies", 60000, 20), ("copies", 120000, 9),
                                       ("volume", 66000, 16), ("volume", 120000, 15), ("curve", 55000, 64),
                                       ("curve", 52000, 40)])
def test_tiles_certify_or_reject(capi, shape, n, k):
    xyz = _shape(shape, n)
    assert xyz.shape[0] == n
    g = capi.GridStructure(xyz)
    r = capi.GridStructure(xyz, config=capi.default_config(knn_mode=0))
    for p in (g, r):
        p.GRIDCUDAKNNSELF_COMPACT(k)
    assert np.array_equal(g.sorted_lists(), r.sorted_lists())
    t, tr = g.timings(), r.timings()
    assert t["invalid_queries"] == tr["invalid_queries"] and t["levels_used"] == tr["levels_used"]
    if shape in ("lattice", "copies"):
        assert t["knn_fallback"] == n and t["exact_reruns"] == n  # every row has equal distances
    else:
        assert t["knn_fallback"] < n  # some rows are the tiles' own
    g.close()
    r.close()


@pytest.mark.parametrize("n,k", [(5000, 20), (5000, 10), (5000, 70), (60000, 20)])
def test_fallback_means_the_same_through_both_calls(capi, n, k):
    g = capi.GridStructure(datagen.sphere_cloud(n, 0.004, n))
    g.GRIDCUDAKNNSELF_COMPACT(k)
    a = g.timings()["knn_fallback"]
    g.knn_host(k)
    assert g.timings()["knn_fallback"] == a
    if n < 40000:
        assert a == (n if 16 <= k <= 64 else 0)
    g.close()
