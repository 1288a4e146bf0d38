"""Batched clouds with oversized cells: rows, invalid counts and lists equal each
cloud's own handle, at the limit (a cell of exactly max_points_in_cell points) and
around it, with tiles and without."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cloud(n, heap, seed):
    """n points, `heap` of them in one cell of every level."""
    g = np.random.Generator(np.random.PCG64(seed))
    x = g.random((n, 3))
    x[:heap] = 0.5004 + 1e-5 * g.random((heap, 3))
    return x.astype(np.float32)


@pytest.mark.parametrize("n,k,cap", [(3000, 10, 64), (20000, 20, 64), (20000, 20, 63), (20000, 20, 65), (400, 5, 1)])
def test_oversized_cells(capi, n, k, cap):
    clouds = [(_cloud(n, 64, 1), k), (_cloud(n, 0, 2), k), (_cloud(n, 200, 3), k)]
    cfg = capi.default_config(max_points_in_cell=cap)
    b = capi.Batch(clouds, config=cfg)
    b.set_tuning(4, 0)
    invalid = 0
    for _ in range(2):
        b.knn()
    for c, (x, _) in enumerate(clouds):
        with capi.GridStructure(x, config=capi.default_config(max_points_in_cell=cap, knn_mode=0)) as g:
            g.GRIDCUDAKNNSELF_COMPACT(k)
            assert np.array_equal(b.knn_host(c), g.GetKNNIndexes())
            invalid += g.timings()["invalid_queries"]
    assert b.timings()["invalid_queries"] == invalid
    b.close()
