"""Performance cases: the calls a program makes on a point cloud or a mesh,
through the library's public entry points (include/egt_b200.h and its Python
mirror), over the sizes it makes them for.

Shapes and parameters are those of the repository's workloads (datagen.py):
noisy spheres, clustered superquadrics, thickened sheets, torus meshes; k up
to 64; 150-300 Taubin iterations; lambda 0.63, mu -0.64; alpha 0.65 for
clouds and 1e-8 for meshes.  Inputs are generated on the GPU from the seed.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

from multigpuegtsmoothing_b200 import capi

LAMBDA, MU = 0.63, -0.64
L2_BYTES = 126e6
KEPT = 16  # neighbours the elliptic-Gabriel filter keeps of a row at alpha 0.65, on surfaces


def listed():
    return [
        # A live preview: new positions of a small cloud every frame, grid and
        # lists rebuilt on the device.  Launches and latency count.
        {"name": "search_2k_k10", "kind": "search", "shape": "sphere", "n": 2000, "k": 10},
        # The same for a single scan (the 35,947 points of the reference's bunny).
        {"name": "search_scan_k40", "kind": "search", "shape": "sphere", "n": 35947, "k": 40},
        # The benchmark's headline: grid and lists of a large cloud of very uneven density.
        {"name": "search_4m_k40", "kind": "search", "shape": "superquadrics", "n": 4000000, "k": 40},
        # The largest cloud, with the longest lists.
        {"name": "search_sheets_20m_k64", "kind": "search", "shape": "sheets", "n": 20000000, "k": 64},
        # Host to host: points from pinned memory, lists back in original order
        # (the benchmark's end-to-end figure, on a cloud of ordinary size).
        {"name": "host_lists_1m_k40", "kind": "host_lists", "shape": "superquadrics", "n": 1000000, "k": 40},
        # Registration (ICP): the points of one scan looked up in another cloud.
        {"name": "query_100k_in_1m_k8", "kind": "query", "shape": "superquadrics", "n": 1000000, "nq": 100000, "k": 8},
        # Host to host on a small scan of odd size: everything the CLI does
        # between reading and writing a file, set-up of the provider included.
        {"name": "whole_2503_k16", "kind": "whole", "shape": "sphere", "n": 2503, "k": 16, "iters": 150},
        # Smoothing a scan at the reference CLI's settings.
        {"name": "smooth_scan_k40", "kind": "smooth", "shape": "sphere", "n": 35947, "k": 40, "iters": 150},
        # Smoothing a mesh (1-ring neighbours), from host arrays.
        {"name": "mesh_131k_k40", "kind": "mesh", "nu": 512, "nv": 256, "k": 40, "iters": 150},
        # The large cloud: lists, filter and 300 iterations.
        {"name": "smooth_4m_k40", "kind": "smooth", "shape": "superquadrics", "n": 4000000, "k": 40, "iters": 300},
        # Oriented normals of a filtered cloud.
        {"name": "normals_1m_k40", "kind": "normals", "shape": "superquadrics", "n": 1000000, "k": 40},
        # Many clouds of uneven size and k in one batch.
        {"name": "batch_32", "kind": "batch", "count": 32, "nmin": 2000, "nmax": 500000, "mix": 4, "iters": 150},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["search", "search", "host_lists", "query", "whole", "smooth", "smooth", "mesh", "normals",
                       "batch"])
    c = {"kind": kind}
    if kind == "mesh":
        c.update(nu=rng.randint(40, 512), nv=rng.randint(24, 256), k=rng.choice([12, 20, 40]),
                 iters=rng.randint(10, 150))
        return c
    if kind == "batch":
        c.update(count=rng.randint(3, 32), nmin=2000, nmax=_log_int(rng, 8000, 500000), mix=rng.randint(0, 1 << 20),
                 iters=rng.randint(10, 150))
        return c
    hi = {"search": 4000000, "host_lists": 2000000, "query": 1000000, "whole": 100000, "smooth": 2000000,
          "normals": 1000000}[kind]
    c.update(shape=rng.choice(["sphere", "superquadrics", "sheets"]), n=_log_int(rng, 2000, hi),
             k=rng.choice([8, 10, 16, 20, 24, 30, 40, 40, 64]))
    if kind == "query":
        c.update(nq=_log_int(rng, 500, 200000), k=rng.choice([1, 4, 8, 16, 32]))
    if kind in ("whole", "smooth"):
        c.update(iters=rng.randint(10, 300))
    return c


# ---- inputs -------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 12345)
    return g


def _sphere(n, g):
    """Unit sphere, radial noise 0.005."""
    d = torch.randn(n, 3, generator=g, device="cuda")
    d /= d.norm(dim=1, keepdim=True)
    return d * (1.0 + 0.005 * torch.randn(n, 1, generator=g, device="cuda"))


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda")


def _superquadrics(n, g):
    """Three overlapping superellipsoids, 50:1 clustered density, noise 0.2 % of the diagonal."""
    shapes = [((0.3, 0.3), (1.0, 0.8, 0.6), (-0.35, 0.0, 0.0)), ((1.0, 1.0), (0.7, 0.7, 0.7), (0.35, 0.1, 0.05)),
              ((2.0, 0.5), (0.6, 0.9, 0.5), (0.0, -0.3, 0.2))]
    par = torch.tensor([[*e, *s, *c] for e, s, c in shapes], device="cuda")
    centres = _rand(g, 12, 3) * 1.8 - 0.9
    out, have = [], 0
    while have < n:
        m = max(1 << 16, min(1 << 23, 4 * (n - have)))
        p = par[torch.randint(0, 3, (m,), generator=g, device="cuda")]
        eta, om = (_rand(g, m) - 0.5) * math.pi, (_rand(g, m) - 0.5) * 2 * math.pi
        ce, se, co, so = eta.cos(), eta.sin(), om.cos(), om.sin()
        spow = lambda b, e: b.sign() * b.abs().pow(e)  # noqa: E731
        x = torch.stack([spow(ce, p[:, 0]) * spow(co, p[:, 1]), spow(ce, p[:, 0]) * spow(so, p[:, 1]),
                         spow(se, p[:, 0])], 1) * p[:, 2:5] + p[:, 5:8]
        near = torch.cdist(x, centres).amin(1)
        rho = 1.0 + 49.0 * torch.exp(-near * near / (2.0 * 0.18 ** 2))
        x = x[_rand(g, m) * 50.0 < rho][:n - have]
        out.append(x)
        have += x.shape[0]
    p = torch.cat(out)
    diag = (p.amax(0) - p.amin(0)).norm()
    return p + 0.002 * diag * torch.randn(n, 3, generator=g, device="cuda")


def _sheets(n, g):
    """Thickened planes and spheres, 1000:1 density."""
    planes = [((0.0, 0.0, 0.0), (1.0, 0.0, 0.0), (0.0, 1.0, 0.0)), ((0.0, 0.0, 0.3), (1.0, 0.0, 0.0), (0.0, 0.6, 0.8)),
              ((0.2, -0.1, -0.2), (0.0, 0.0, 1.0), (0.8, 0.6, 0.0)), ((-0.3, 0.3, 0.0), (0.6, -0.8, 0.0), (0.0, 0.0, 1.0))]
    spheres = [((0.3, 0.3, 0.3), 0.35), ((-0.4, -0.2, 0.1), 0.25), ((0.1, -0.4, -0.3), 0.2)]
    po = torch.tensor([o for o, _, _ in planes] + [c for c, _ in spheres], device="cuda")
    pa = torch.tensor([a for _, a, _ in planes] + [(0.0,) * 3] * 3, device="cuda")
    pb = torch.tensor([b for _, _, b in planes] + [(0.0,) * 3] * 3, device="cuda")
    rad = torch.tensor([0.0] * 4 + [r for _, r in spheres], device="cuda")
    out, have = [], 0
    while have < n:
        m = max(1 << 16, min(1 << 24, 8 * (n - have)))
        s = torch.randint(0, 7, (m,), generator=g, device="cuda")
        uv = _rand(g, m, 2) * 1.6 - 0.8
        d = torch.randn(m, 3, generator=g, device="cuda")
        d /= d.norm(dim=1, keepdim=True)
        x = po[s] + uv[:, :1] * pa[s] + uv[:, 1:] * pb[s] + rad[s][:, None] * d
        f = 0.5 + 0.5 * torch.sin(3.0 * x[:, 0] + 1.0) * torch.cos(2.0 * x[:, 1] - 0.5)
        x = x[_rand(g, m) < torch.exp(math.log(1000.0) * (f - 1.0))][:n - have]
        out.append(x)
        have += x.shape[0]
    return torch.cat(out) + 0.002 * torch.randn(n, 3, generator=g, device="cuda")


def _cloud(case, seed):
    make = {"sphere": _sphere, "superquadrics": _superquadrics, "sheets": _sheets}[case["shape"]]
    return make(case["n"], _gen(seed)).float().contiguous()


def _mesh(case, seed):
    """Torus R=1, r=0.3 on an nu x nv grid, noise 0.5 % of r: host arrays, as read from a file."""
    nu, nv = case["nu"], case["nv"]
    g = np.random.Generator(np.random.PCG64(seed))
    u = 2.0 * np.pi * np.arange(nu)[:, None] / nu
    v = 2.0 * np.pi * np.arange(nv)[None, :] / nv
    w = 1.0 + 0.3 * np.cos(v)
    xyz = np.stack([w * np.cos(u), w * np.sin(u), np.broadcast_to(0.3 * np.sin(v), (nu, nv))], -1).reshape(-1, 3)
    xyz = (xyz + 0.0015 * g.standard_normal(xyz.shape)).astype(np.float32)
    ii, jj = np.meshgrid(np.arange(nu), np.arange(nv), indexing="ij")
    at = lambda i, j: (i % nu) * nv + j % nv  # noqa: E731
    a, b, c, d = at(ii, jj), at(ii + 1, jj), at(ii + 1, jj + 1), at(ii, jj + 1)
    tris = np.stack([np.stack([a, b, c], -1), np.stack([a, c, d], -1)], 2).reshape(-1, 3).astype(np.uint32)
    return xyz, tris


def _batch_sizes(case):
    """(points, k, is a sphere) of each cloud: the same for every seed."""
    r = random.Random(case["mix"])
    return [(_log_int(r, case["nmin"], case["nmax"]), r.choice([10, 20, 40]), r.random() < 0.5)
            for _ in range(case["count"])]


def _batch_clouds(case, seed):
    g = _gen(seed)
    out = []
    for n, k, ball in _batch_sizes(case):
        if ball:
            x = _sphere(n, g)
        else:
            u, v = _rand(g, n) * 2 * math.pi, _rand(g, n) * 2 * math.pi
            w = 1.0 + 0.3 * v.cos()
            x = torch.stack([w * u.cos(), w * u.sin(), 0.3 * v.sin()], 1)
            x = x + 0.0015 * torch.randn(n, 3, generator=g, device="cuda")
        x = x * (0.5 + 3.5 * _rand(g, 1)) + (_rand(g, 3) * 20 - 10)
        out.append((x.float().cpu().numpy(), k))
    return out


class _Device:
    """A device buffer of a provider as a tensor; keeps the provider alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 2}


def _lists(g):
    v = g.views()
    return torch.as_tensor(_Device(g, v.lists, (int(v.n), int(v.k)), "<i4"), device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "mesh":
        s["xyz"], s["tris"] = _mesh(case, seed)
        return s
    if kind == "batch":
        s["batch"] = capi.Batch(_batch_clouds(case, seed))
        return s
    xyz = _cloud(case, seed)
    if kind == "whole":
        s["xyz"] = xyz.cpu().numpy()
        return s
    if kind == "host_lists":
        pin = lambda t: t.pin_memory().numpy()  # noqa: E731
        s["xyz"] = pin(xyz.cpu())
        s["lists"] = torch.empty((case["n"], case["k"]), dtype=torch.int32, pin_memory=True).numpy()
        return s
    s["g"] = capi.GridStructure(None, device_ptr=xyz.data_ptr(), n=case["n"])
    if kind == "query":
        # another scan of the same object: a subset, jittered by the noise of a scanner
        gen = _gen(seed + 1000003)
        at = torch.randint(0, case["n"], (case["nq"],), generator=gen, device="cuda")
        s["q"] = (xyz[at] + 0.002 * torch.randn(case["nq"], 3, generator=gen, device="cuda")).cpu().numpy()
        return s
    if kind == "normals":
        s["g"].GRIDCUDAKNNSELF_COMPACT(case["k"])
        capi.EGT_CUDA(s["g"]).Filter(0.65)
        return s
    s["xyz"] = xyz
    if kind == "smooth":
        s["out"] = [torch.empty(case["n"], device="cuda") for _ in range(3)]
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "search":
        g = state["g"]
        g.UpdatePointsDevice(state["xyz"].data_ptr())
        g.GRIDCUDAKNNSELF_COMPACT(case["k"])
        return _lists(g)
    if kind == "host_lists":
        with capi.GridStructure(state["xyz"]) as g:
            return g.knn_host(case["k"], state["lists"])
    if kind == "query":
        return state["g"].GRIDCUDAKNNCompact(state["q"], case["k"])
    if kind == "whole":
        with capi.GridStructure(state["xyz"]) as g:
            g.GRIDCUDAKNNSELF_COMPACT(case["k"])
            capi.EGT_CUDA(g).PerformSmoothing(case["iters"], LAMBDA, MU, 0.65)
            return {"normals": capi.Normal_CUDA(g).GetNormals(), "points": capi.getOutputPoints(g)}
    if kind == "mesh":
        with capi.GridMeshCuda(state["xyz"], state["tris"]) as g:
            g.GetNeighborsFromTriangles(case["k"])
            capi.EGT_CUDA(g).PerformSmoothing(case["iters"], LAMBDA, MU, 1e-8)
            return capi.getOutputPoints(g)
    if kind == "smooth":
        g = state["g"]
        g.UpdatePointsDevice(state["xyz"].data_ptr())
        g.GRIDCUDAKNNSELF_COMPACT(case["k"])
        capi.EGT_CUDA(g).PerformSmoothing(case["iters"], LAMBDA, MU, 0.65)
        p = [C.c_void_p(t.data_ptr()) for t in state["out"]]
        capi._check(capi.lib().egt_output_device(g.handle, *p, g.stream))
        return state["out"]
    if kind == "normals":
        g = state["g"]  # the normals stay on the device
        capi._check(capi.lib().egt_normals(g.handle, None, None, None, g.stream))
        return torch.as_tensor(_Device(g, g.views().normals, (3, case["n"]), "<f4"), device="cuda")
    if kind == "batch":
        state["batch"].run(case["iters"], LAMBDA, MU, 0.65)
        return state["batch"].output()
    raise ValueError(kind)


def work(case):
    """Bytes and operations of one pass: inputs once, outputs once, and for the
    smoothing the 2 * iters half-steps, each of which needs all of the last
    one's positions: their arithmetic, and their traffic where positions and
    neighbourhoods do not fit the cache."""
    kind = case["kind"]
    if kind == "batch":
        parts = [(n, k) for n, k, _ in _batch_sizes(case)]
    elif kind == "mesh":
        parts = [(case["nu"] * case["nv"], 6)]
    else:
        parts = [(case["n"], case["k"])]
    n = sum(p[0] for p in parts)
    nk = sum(p[0] * p[1] for p in parts)
    search = 0.0 if kind == "mesh" else 8.0 * nk  # a distance for each entry of a list
    if kind in ("search", "host_lists"):
        return {"bytes": 12.0 * n + 4.0 * nk, "flops": search}
    if kind == "query":
        return {"bytes": 12.0 * (n + case["nq"]) + 4.0 * case["nq"] * case["k"], "flops": 8.0 * case["nq"] * case["k"]}
    kept = sum(p[0] * min(p[1], KEPT) for p in parts)
    if kind == "normals":
        return {"bytes": 24.0 * n + 4.0 * kept, "flops": 30.0 * kept + 200.0 * n}
    step = 28.0 * n + 4.0 * kept
    steps = 2 * case["iters"]
    moved = 24.0 * n + (steps * step if step > L2_BYTES else 0.0)
    if kind == "whole":
        moved += 12.0 * n
    if kind == "mesh":
        moved += 24.0 * n  # two triangles a vertex
    tests = 24.0 * nk  # at least one ellipsoid test for each entry
    return {"bytes": moved, "flops": search + tests + steps * (24.0 * kept + 12.0 * n)}


# ---- the same in 64 bits ------------------------------------------------------------

def _unit(x):
    """The library's normalised coordinates: one scalar range for all axes."""
    lo, hi = x.min() - 1e-6, x.max() + 1e-6
    return (x - lo) / (hi - lo), lo, hi - lo


def _nearest(p, k):
    out = []
    for a in range(0, p.shape[0], 2048):
        d = (p[a:a + 2048, None, 0] - p[None, :, 0]) ** 2
        d += (p[a:a + 2048, None, 1] - p[None, :, 1]) ** 2
        d += (p[a:a + 2048, None, 2] - p[None, :, 2]) ** 2
        r = torch.arange(d.shape[0], device=d.device)
        d[r, r + a] = math.inf
        out.append(d.topk(k, dim=1, largest=False, sorted=True).indices)
    return torch.cat(out)


def _filtered(p, idx, alpha):
    """Entries of the lists that no closer entry's ellipsoid test drops (-1: none)."""
    keep = idx >= 0
    for a in range(0, p.shape[0], 4096):
        i = idx[a:a + 4096].clamp(min=0)
        c = p[a:a + 4096, None, :]
        q = p[i]
        axis = q - c
        full = axis.norm(dim=2, keepdim=True)
        axis = axis / full.clamp(min=1e-300)
        rel = q[:, None, :, :] - (0.5 * (q + c))[:, :, None, :]  # [row, tested j, closer u]
        along = (rel * axis[:, :, None, :]).sum(3)
        across = (rel * rel).sum(3) - along * along
        d = 0.5 * full[:, :, 0]
        inside = along * along + across / (alpha * alpha) < (d * d)[:, :, None]
        j = torch.arange(i.shape[1], device=i.device)
        inside &= (j[None, :] < j[:, None])[None] & (idx[a:a + 4096] >= 0)[:, None, :]
        inside &= ((d >= 1e-6) & (full[:, :, 0] >= 1e-6))[:, :, None]
        keep[a:a + 4096] &= ~inside.any(2)
    return keep


def _taubin(p, idx, keep, iters):
    i = idx.clamp(min=0)
    w0 = keep.double()
    for step in range(2 * iters):
        d = p[i] - p[:, None, :]
        w = torch.exp(-(d * d).sum(2)) * w0
        total = w.sum(1, keepdim=True)
        total = torch.where(total == 0, torch.full_like(total, 1e-8), total)
        p = p + (LAMBDA if step % 2 == 0 else MU) * (w[:, :, None] * d).sum(1) / total
    return p


def _smoothed(xyz, k, iters, alpha, idx=None):
    """[n, 3] smoothed positions."""
    p, lo, span = _unit(xyz.double())
    if idx is None:
        idx = _nearest(p, k)
    keep = _filtered(p, idx, alpha)
    return _taubin(p, idx, keep, iters) * span + lo


def _one_ring(xyz, tris, k):
    """Neighbours over triangle edges, nearest first, -1 padded."""
    t = torch.from_numpy(tris.astype(np.int64)).cuda()
    n = xyz.shape[0]
    e = torch.cat([t[:, [0, 1]], t[:, [1, 0]], t[:, [1, 2]], t[:, [2, 1]], t[:, [0, 2]], t[:, [2, 0]]])
    key = torch.unique(e[:, 0] * n + e[:, 1])
    u, v = key // n, key % n
    p = _unit(xyz.double())[0]
    order = torch.argsort((p[u] - p[v]).norm(dim=1), stable=True)
    u, v = u[order], v[order]
    order = torch.argsort(u, stable=True)
    u, v = u[order], v[order]
    start = torch.searchsorted(u, torch.arange(n, device=u.device))
    at = torch.arange(u.shape[0], device=u.device) - start[u]
    idx = torch.full((n, k), -1, dtype=torch.int64, device=u.device)
    ok = at < k
    idx[u[ok], at[ok]] = v[ok]
    return idx


def exact(case, seed):
    """run()'s smoothed positions in 64 bits, for the clouds whose neighbours a
    brute-force search finds in time.  Lists are whole numbers, and the sign of
    a normal is a choice of the spanning tree: no value for those."""
    kind = case["kind"]
    if kind in ("smooth", "whole"):
        if float(case["n"]) ** 2 > 4e9 or case["n"] * case["k"] * case["iters"] > 1e9:
            return None
        p = _smoothed(_cloud(case, seed), case["k"], case["iters"], 0.65)
        p = [p[:, c] for c in range(3)]
        return {"normals": (None, None, None), "points": p} if kind == "whole" else p
    if kind == "mesh":
        xyz, tris = _mesh(case, seed)
        x = torch.from_numpy(xyz).cuda()
        p = _smoothed(x, case["k"], case["iters"], 1e-8, _one_ring(x, tris, min(case["k"], 12)))
        return tuple(p[:, c] for c in range(3))
    if kind == "batch":
        if sum(float(n) ** 2 for n, _, _ in _batch_sizes(case)) > 2e10:
            return None
        return [_smoothed(torch.from_numpy(x).cuda(), k, case["iters"], 0.65) for x, k in _batch_clouds(case, seed)]
    return None
