"""Which searches the default mode takes (cell tiles from 40,000 points, for k
below 16 from 100,000, and there not where many queries are left to the ring
search), and that every route gives the ring search's lists."""
import numpy as np
import pytest

from multigpuegtsmoothing_b200 import datagen

pytestmark = pytest.mark.gpu


def _clusters(n):
    """Eight clusters of very different widths: many blocks too dense or too sparse for the tiles."""
    g = np.random.Generator(np.random.PCG64(n))
    at = g.integers(0, 8, n)
    width = np.minimum(0.002 * 3.0 ** np.arange(8), 0.3)
    return (g.random((8, 3))[at] + width[at, None] * g.standard_normal((n, 3))).astype(np.float32)


# left: rows the ring search ran (none counted where k below 16 never met the tiles)
@pytest.mark.parametrize("shape,n,k,left", [("sphere", 39999, 16, "all"), ("sphere", 40000, 16, "few"),
                                            ("sphere", 40001, 64, "few"), ("sphere", 99999, 15, "none"),
                                            ("sphere", 100000, 8, "few"), ("sphere", 100001, 15, "few"),
                                            ("clusters", 120000, 10, "all"), ("clusters", 120000, 20, "some")])
def test_route_and_lists(capi, shape, n, k, left):
    xyz = _clusters(n) if shape == "clusters" else datagen.sphere_cloud(n, 0.004, n)
    g = capi.GridStructure(xyz)
    r = capi.GridStructure(xyz, config=capi.default_config(knn_mode=0))
    for p in (g, r):
        p.GRIDCUDAKNNSELF_COMPACT(k)
    assert np.array_equal(g.sorted_lists(), r.sorted_lists())
    t, tr = g.timings(), r.timings()
    assert t["invalid_queries"] == tr["invalid_queries"]
    assert t["levels_used"] == tr["levels_used"]
    ring = t["knn_fallback"]
    assert {"all": ring == n, "none": ring == 0, "few": 0 <= ring < 0.1 * n, "some": 0 < ring < n}[left], ring
    assert t["knn_evaluations"] > n * k
    g.close()
    r.close()


@pytest.mark.parametrize("count,n", [(12, 10000), (120, 1000)])  # tiles; too few points a cloud for k below 16
def test_batch_routes(capi, count, n):
    clouds = [(datagen.sphere_cloud(n, 0.01, c), 10) for c in range(count)]
    b = capi.Batch(clouds)
    b.set_tuning(4, 0)
    for _ in range(12):  # the lists of unselected queries start empty in every call
        b.knn()
    for c in (0, count // 2, count - 1):
        with capi.GridStructure(clouds[c][0], config=capi.default_config(knn_mode=0)) as g:
            g.GRIDCUDAKNNSELF_COMPACT(10)
            assert np.array_equal(b.knn_host(c), g.GetKNNIndexes())
    b.close()


def test_batch_repeated_calls(capi):
    """Clouds with many queries left to the ring search, searched again and again."""
    clouds = [(_clusters(500), 30) for _ in range(100)]
    b = capi.Batch(clouds)
    b.set_tuning(4, 0)
    for _ in range(40):
        b.knn()
    with capi.GridStructure(clouds[0][0], config=capi.default_config(knn_mode=0)) as g:
        g.GRIDCUDAKNNSELF_COMPACT(30)
        want = g.GetKNNIndexes()
    for c in (0, 57, 99):
        assert np.array_equal(b.knn_host(c), want)
    b.close()
