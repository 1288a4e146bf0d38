"""Orientation where many rows list the same points (equal points of a scan
all list the same few; here the lists are written so): edge buckets longer than
are ordered by counting, with repeated entries, around the limit of 1,024.  The
signs are the oracle's, as in test_gpu_orient_buckets.py."""
import numpy as np
import pytest

from multigpuegtsmoothing_b200 import datagen

pytestmark = pytest.mark.gpu


class _Lists:
    def __init__(self, v):
        self.__cuda_array_interface__ = {"shape": (int(v.n), int(v.k)), "typestr": "<i4", "data": (v.lists, False),
                                         "version": 2}


@pytest.mark.parametrize("n,hub,rows", [(3000, 5, 1020), (3000, 5, 1040), (5000, 0, 5000), (70000, 33000, 70000),
                                        (70000, 3, 70000)])
def test_hub_signs_match_oracle(capi, oracle, n, hub, rows):
    import torch

    xyz = datagen.sphere_cloud(n, 0.01, n)
    g = capi.GridStructure(xyz, config=capi.default_config(normals_gap_tol=0.0))
    g.GRIDCUDAKNNSELF_COMPACT(9)
    v = g.views()
    t = torch.as_tensor(_Lists(v), device="cuda")
    t[:rows, 8] = hub      # many rows list one point
    t[: rows // 2, 7] = hub  # half of them twice
    t[hub, 7:] = (hub + 1) % n
    torch.cuda.synchronize()
    capi._check(capi.lib().egt_commit_views(g.handle, v.x, v.y, v.z, None))
    capi.Normal_CUDA(g).GetNormals()
    got, lists = g.sorted_normals(), g.sorted_lists()
    assert (lists[:rows, 8] == hub).sum() >= rows - 1
    ok = np.isfinite(got).all(0)
    assert ok.mean() > 0.99
    want, parent, nc = oracle.orient(got, lists)
    assert np.array_equal(want[:, ok], got[:, ok])
    assert g.timings()["components"] == nc
    g.close()


def test_equal_points_cost_no_square(capi):
    """50,000 equal points: 1.4 ms, against 54 when buckets of any length are counted."""
    xyz = datagen.sphere_cloud(200000, 0.01, 9)
    xyz[:50000] = 0.0
    g = capi.GridStructure(xyz)
    g.GRIDCUDAKNNSELF_COMPACT(40)
    for _ in range(2):
        capi.Normal_CUDA(g).GetNormals()
    assert g.timings()["orient_ms"] < 20.0
    g.close()
