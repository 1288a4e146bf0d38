"""The grid build above the size from which the library sorts (24 * 2^20 points):
order, positions and every level's tables are those of a stable sort by cell."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [24 << 20, (24 << 20) + 1])
def test_large_grid(capi, n):
    import torch

    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    x = torch.rand(n, 3, generator=gen, device="cuda")
    x[: n // 2] = 0.3 + 0.05 * x[: n // 2]
    with capi.GridStructure(None, device_ptr=x.data_ptr(), n=n) as g:
        v = g.views()
        lo, hi = np.float32(v.min_extent), np.float32(v.max_extent)
        # the library's arithmetic, one rounding an operation (on the host: a GPU tensor
        # divided by a scalar is multiplied by its reciprocal)
        p = (x.cpu().numpy() - lo) / (hi - lo)
        eps = np.float32(1e-6)
        a, b = -eps, np.float32(1.0 + float(eps))
        c = torch.from_numpy(((p - a) / (b - a) * np.float32(1024.0)).astype(np.int64)).cuda()
        want = torch.argsort(c[:, 0] + (c[:, 1] << 10) + (c[:, 2] << 20), stable=True).cpu().numpy()
        assert np.array_equal(g.GetOriginalRefIndexes(), want)
        assert np.array_equal(g.sorted_positions(), p[want].T)
        # the upper levels' tables: lists of a sample against the search of the same points as queries
        g.GRIDCUDAKNNSELF_COMPACT(4)
        lists = g.GetKNNIndexes()
        at = np.arange(0, n, n // 5000)
        near, bad = g.GRIDCUDAKNNCompact(x[torch.from_numpy(at).cuda()].cpu().numpy(), 5)
        assert bad == 0
        same = np.array([set(r) == set(l) | {i} for r, l, i in zip(near, lists[at], at)])
        assert same.mean() > 0.999  # (equal distances aside)
