"""The ring search where its form changes (a jump to the first level that can
fill the list, or the walk level by level; list registers), in the default mode
against the walk (EGT_KNN_PLAIN): identical lists, invalid rows and deepest level."""
import numpy as np
import pytest

from multigpuegtsmoothing_b200 import datagen

pytestmark = pytest.mark.gpu


# three registers a lane (k 64..95): the jump up to 2^23 list entries, n (k + 1)
@pytest.mark.parametrize("n,k", [(127100, 65), (127101, 65), (3000, 63), (3000, 64), (20000, 95), (20000, 96),
                                 (2500, 127), (2500, 128), (1500, 255), (1500, 256), (90, 95), (7, 80)])
def test_default_matches_walk(capi, n, k):
    xyz = datagen.sphere_cloud(n, 0.005, n)
    xyz[: n // 4] *= np.float32(0.1)  # a dense part
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


@pytest.mark.parametrize("nq", [2, 777, 30000])
def test_query_forms_agree(capi, nq):
    """k below 3, to 31 and above take different forms: a shorter row is the start of a longer one."""
    xyz = datagen.superquadrics(60000, seed=3)
    g = np.random.Generator(np.random.PCG64(nq))
    q = xyz[g.integers(0, xyz.shape[0], nq)] + g.normal(0, 0.01, (nq, 3)).astype(np.float32)
    q[:1] = 3.0  # outside the cloud's cube
    with capi.GridStructure(xyz) as h:
        want, bad = h.GRIDCUDAKNNCompact(q, 96)
        ok = want[:, -1] >= 0
        assert ok.any()
        for k in (1, 2, 3, 31, 32, 63, 64):
            got, _ = h.GRIDCUDAKNNCompact(q, k)
            assert np.array_equal(got[ok], want[ok, :k])
