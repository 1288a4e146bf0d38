"""The resident Taubin loop (clouds of up to one tile per resident block) and
the launch-per-half-step loop above it, against the general half-step kernel
(egt_taubin_halfstep) applied one by one: the same arithmetic in the same
order, so the positions are equal bit for bit."""
import ctypes as C

import numpy as np
import pytest

from multigpuegtsmoothing_b200 import datagen

pytestmark = pytest.mark.gpu


# tiles of 256 rows; one B200 keeps 592 tiles resident (151,552 rows)
@pytest.mark.parametrize("n,iters,filtered", [(1, 2, True), (255, 5, True), (257, 5, True), (5000, 40, True),
                                              (4001, 6, False),  # unfiltered: every tile gathers from global memory
                                              (151552, 9, True), (151553, 9, True)])
def test_loop_matches_single_half_steps(capi, n, iters, filtered):
    import torch

    lam, mu, k = 0.63, -0.64, 24
    xyz = datagen.sphere_cloud(n, 0.005, 7 + n)
    xyz[: n // 3] *= np.float32(0.2)  # two densities: tiles with few and with many distinct neighbours
    g = capi.GridStructure(xyz)
    g.GRIDCUDAKNNSELF_COMPACT(k)
    egt = capi.EGT_CUDA(g)
    if filtered:
        egt.Filter(0.65)
    off, col, nnz = C.c_void_p(), C.c_void_p(), C.c_int64()
    capi._check(capi.lib().egt_get_csr(g.handle, C.byref(off), C.byref(col), C.byref(nnz)))
    a = torch.zeros((n, 4), device="cuda")
    a[:, :3] = torch.from_numpy(g.sorted_positions().T.copy()).cuda()
    b = torch.zeros_like(a)
    for it in range(2 * iters):
        src, dst = (a, b) if it % 2 == 0 else (b, a)
        capi._check(capi.lib().egt_taubin_halfstep(C.c_void_p(src.data_ptr()), C.c_void_p(dst.data_ptr()), off, col, n,
                                                   lam if it % 2 == 0 else mu, 0, None))
    want = a[:, :3].cpu().numpy().T
    egt.Taubin(iters - 1, lam, mu)  # in two calls: the second starts from the first's positions
    egt.Taubin(1, lam, mu)
    assert np.array_equal(g.sorted_positions(), want)
    g.timings()  # no wait expired
