"""The orientation's edge buckets and forest rounds at their edges: one-way
list entries (k = 1), rows longer than a row's 16 lanes, block remainders,
and a curve whose weights grow along it, so that a round's links form one chain
of all its points.  The signs are the oracle's: its forest and walk leave them
unchanged, the trees are as many, and every root keeps its unoriented sign."""
import numpy as np
import pytest

from multigpuegtsmoothing_b200 import datagen

pytestmark = pytest.mark.gpu


def _spiral(n):
    t = np.linspace(0.0, 1.0, n) ** 1.5 * 6.0 + 0.2
    return np.stack([t * np.cos(3 * t), t * np.sin(3 * t), 0.3 * t * t], 1).astype(np.float32)


@pytest.mark.parametrize("n,k,shape", [(2, 1, "ball"), (17, 3, "ball"), (256, 1, "ball"), (257, 17, "ball"),
                                       (2049, 40, "ball"), (6000, 4, "spiral"), (70000, 9, "ball")])
def test_signs_match_oracle(capi, oracle, n, k, shape):
    xyz = _spiral(n) if shape == "spiral" else datagen.sphere_cloud(n, 0.01, n)
    g = capi.GridStructure(xyz, config=capi.default_config(normals_gap_tol=0.0))
    g.GRIDCUDAKNNSELF_COMPACT(k)
    capi.Normal_CUDA(g).GetNormals()
    got, lists = g.sorted_normals(), g.sorted_lists()
    ok = np.isfinite(got).all(0)
    raw = oracle.normals(g.sorted_positions(), lists, False)
    want, parent, nc = oracle.orient(got, lists)
    assert np.array_equal(want[:, ok], got[:, ok])
    assert g.timings()["components"] == nc
    roots = np.where(parent < 0)[0]
    has_child = np.zeros(n, bool)
    has_child[parent[parent >= 0]] = True
    roots = roots[has_child[roots] & ok[roots]]
    # (k below 3 leaves the smallest eigenvalue's direction open)
    if k >= 3:
        assert ((got[:, roots] * raw[:, roots]).sum(0) > 0).all()
