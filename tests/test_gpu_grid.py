"""Grid build at the edges of its tiles: the radix passes take 1,024 elements a
block up to 262,144 points and 3,072 above, the table kernel 4,096.  Order,
positions and the lists found through every level's tables against the oracle,
all exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(n):
    """Half a uniform cube, half a tight cluster with duplicates: crowded and empty cells on every level."""
    g = np.random.Generator(np.random.PCG64(n))
    x = g.uniform(-1.0, 2.0, (n, 3))
    m = n // 2
    x[:m] = 0.3 + 0.01 * g.standard_normal((m, 3))
    if m > 8:
        x[: m // 8] = x[m // 8: 2 * (m // 8)]
    return g.permutation(x.astype(np.float32))


@pytest.mark.parametrize("n", [1, 2, 1023, 1024, 1025, 3073, 4096, 4097, 262144, 262145])
def test_grid_build_matches_oracle(capi, oracle, n):
    xyz = _points(n)
    want = oracle.knn(xyz, 3)
    g = capi.GridStructure(xyz)
    for _ in range(2):  # the second time over the first one's tables
        assert np.array_equal(g.GetOriginalRefIndexes(), want["perm"])
        assert np.array_equal(g.sorted_positions(), want["pos"])
        g.GRIDCUDAKNNSELF_COMPACT(3)
        assert np.array_equal(g.sorted_lists(), want["lists"])
        import torch
        t = torch.from_numpy(xyz).cuda()
        flat = torch.empty(t.numel() + 1, device="cuda")
        flat[1:] = t.reshape(-1)  # 4-byte aligned only
        g.UpdatePointsDevice(flat.data_ptr() + 4)
    g.close()
