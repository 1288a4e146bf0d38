"""egt_update_points_device and the calls after it on other streams: when it
returns the grid is complete, whatever stream reads it next."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_update_then_search_on_another_stream(capi):
    import torch

    n, k = 2_000_000, 10
    g = np.random.Generator(np.random.PCG64(5))
    clouds = [torch.from_numpy(g.uniform(0, 1, (n, 3)).astype(np.float32)).cuda() for _ in range(3)]
    want = []
    for x in clouds:
        with capi.GridStructure(None, device_ptr=x.data_ptr(), n=n) as h:
            h.GRIDCUDAKNNSELF_COMPACT(k)
            want.append((h.GetOriginalRefIndexes(), h.sorted_lists()))
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    lib = capi.lib()
    with capi.GridStructure(None, device_ptr=clouds[0].data_ptr(), n=n) as h:
        views = h.views()
        out = torch.empty(n, dtype=torch.int32, pin_memory=True)
        for x, (perm, lists) in list(zip(clouds, want))[1:]:
            capi._check(lib.egt_update_points_device(h.handle, C.c_void_p(x.data_ptr()), C.c_void_p(a.cuda_stream)))
            class Perm:  # the view's pointer, read on another stream without a wait
                __cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (views.perm, False), "version": 2}
            with torch.cuda.stream(b):
                out.copy_(torch.as_tensor(Perm(), device="cuda"), non_blocking=True)
            b.synchronize()
            capi._check(lib.egt_knn(h.handle, k, C.c_void_p(b.cuda_stream)))
            b.synchronize()
            assert np.array_equal(out.numpy(), perm)
            assert np.array_equal(h.sorted_lists(), lists)
