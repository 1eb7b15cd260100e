"""The work that users of dwg_b200 have it do, as cases that can be timed.

Kinds of case:

* ``reconstruct`` -- ``dwg_reconstruct_host``: points in, point normals and the
  final mesh out, in host memory, with the flags of the DWG_CUDA command;
* ``knn``         -- the neighbour index (``KnnIndex``): built and queried once,
  or kept and queried;
* ``winding``     -- the winding-number sums at points (``TurboLibiGWN``): tree
  built and used once, or kept while the normals change;
* ``grid``        -- the plain sums on a sampling grid, far field of order 0-2;
* ``gradient``    -- sums and their gradients at points;
* ``mc``          -- marching cubes of a sampled field (``TurboMC``);
* ``mlp``         -- loss and gradients of one training batch of the learned
  normal initialiser (``LearnedNormalInit``).
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from dwg_b200 import capi, turbo

DEV = "cuda"
AREA = 2e-6  # the pipeline's area per leaf
TERMS_PER_QUERY = 19.0  # Barnes-Hut terms of one query per log2(points) at beta 2.3


def listed():
    return [
        # a quick neighbour lookup in a small scan: latency and launches
        dict(name="knn_once_2k", kind="knn", n=2000, nq=2000, k=10, queries="self", kept=False),
        # the triangles of a mesh against the leaves of a large cloud, one diffusion step's search
        dict(name="knn_kept_1m", kind="knn", n=1000000, nq=1000000, k=15, queries="near", kept=True),
        # the winding number of a few thousand points, tree included: inside/outside tests of a small object
        dict(name="winding_once_5k", kind="winding", n=5003, nq=5003, screened=False, precision=1, kept=False),
        # one diffusion step's sums at its own points after new normals
        dict(name="winding_kept_300k", kind="winding", n=300000, nq=300000, screened=True, precision=1, kept=True),
        # libigl's fast winding number with its default expansion on a sampling grid
        dict(name="grid_order2_100k", kind="grid", n=100000, res=160, order=2, beta=2.0),
        # field and gradient at surface samples (normals of the implicit surface, projection steps)
        dict(name="gradient_100k", kind="gradient", n=100000, nq=200001, screened=True),
        # meshing: a preview grid with odd sides, and a fine one
        dict(name="mc_97", kind="mc", rx=97, ry=83, rz=61),
        dict(name="mc_384", kind="mc", rx=384, ry=384, rz=384),
        # a training batch of the learned initialiser, forward and backward
        dict(name="mlp_65k", kind="mlp", batch=65536),
        # whole reconstructions: the small noisy sphere, the non-uniform torus, the union of thin superquadrics
        dict(name="reconstruct_10k", kind="reconstruct", shape="sphere", n=10000, grid=128, iters=30, com_as=0,
             precision=1),
        dict(name="reconstruct_100k", kind="reconstruct", shape="torus", n=100000, grid=256, iters=30, com_as=0,
             precision=1),
        dict(name="reconstruct_1m", kind="reconstruct", shape="union", n=1010000, grid=256, iters=30, com_as=0,
             precision=1),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["knn", "winding", "grid", "gradient", "mc", "mlp", "reconstruct", "reconstruct"])
    if kind == "knn":
        n = _logint(rng, 2000, 1000000)
        return dict(kind=kind, n=n, nq=_logint(rng, 2000, 1000000), k=rng.choice([8, 10, 15, 16, 32]),
                    queries=rng.choice(["self", "near"]), kept=rng.random() < 0.5)
    if kind == "winding":
        return dict(kind=kind, n=_logint(rng, 2000, 500000), nq=_logint(rng, 2000, 500000),
                    screened=rng.random() < 0.6, precision=rng.choice([0, 1, 3]), kept=rng.random() < 0.5)
    if kind == "grid":
        return dict(kind=kind, n=_logint(rng, 2000, 300000), res=rng.randint(48, 200), order=rng.choice([0, 1, 2]),
                    beta=rng.choice([2.0, 2.3]))
    if kind == "gradient":
        return dict(kind=kind, n=_logint(rng, 2000, 300000), nq=_logint(rng, 2000, 300000),
                    screened=rng.random() < 0.5)
    if kind == "mc":
        s = _logint(rng, 33, 400)
        return dict(kind=kind, rx=s, ry=max(17, int(s * rng.uniform(0.4, 1.0))),
                    rz=max(17, int(s * rng.uniform(0.4, 1.0))))
    if kind == "mlp":
        return dict(kind=kind, batch=_logint(rng, 500, 130000))
    n = _logint(rng, 2000, 300000)
    return dict(kind=kind, shape=rng.choice(["sphere", "torus", "union"]), n=n,
                grid=min(256, max(128, round(128 * (n / 2000.0) ** (1 / 3)))), iters=rng.choice([20, 30, 40]),
                com_as=rng.choice([0, 0, 0, 1]), precision=rng.choice([0, 1, 1, 3]))


# ------------------------------------------------------------------ clouds --
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _uniform(g, lo, hi, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64) * (hi - lo) + lo


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float64)


def _sphere(n, g):
    d = _normal(g, n, 3)
    d = d / d.norm(dim=1, keepdim=True)
    return d + 0.002 * _normal(g, n, 3), d


def _torus(n, g, R=1.0, r=0.35):
    """Area-uniform times 1 + 0.8 sin(3 theta), noise along the normal."""
    th, ph = _uniform(g, 0, 2 * math.pi, 8 * n), _uniform(g, 0, 2 * math.pi, 8 * n)
    w = (R + r * ph.cos()) * (1 + 0.8 * (3 * th).sin())
    keep = (_uniform(g, 0, 1.8 * (R + r), 8 * n) < w).nonzero()[:n, 0]
    th, ph = th[keep], ph[keep]
    nrm = torch.stack([ph.cos() * th.cos(), ph.cos() * th.sin(), ph.sin()], 1)
    ctr = torch.stack([R * th.cos(), R * th.sin(), torch.zeros_like(th)], 1)
    return ctr + (r + 0.003 * _normal(g, len(th), 1)) * nrm, nrm


def _rotation(g):
    q, r = torch.linalg.qr(_normal(g, 3, 3))
    return q * r.diagonal().sign()


def _inside(x, s):
    """The superquadric's inside-outside function (below 1 inside)."""
    y = ((x - s["c"]) @ s["R"]).abs() / s["a"]
    return (y[:, 0] ** (2 / s["e2"]) + y[:, 1] ** (2 / s["e2"])) ** (s["e2"] / s["e1"]) + y[:, 2] ** (2 / s["e1"])


def _union(n, g, k=12, outliers=0.01):
    """Surface samples of a union of superquadrics, about area-uniform, with
    sheets thinner than the sampling, and uniform outliers in the box."""
    solids = [dict(e1=float(_uniform(g, 0.3, 3.0, 1)), e2=float(_uniform(g, 0.3, 3.0, 1)),
                   a=_uniform(g, 0.05, 1.0, 3), R=_rotation(g), c=_uniform(g, -1.0, 1.0, 3)) for _ in range(k)]
    m = n - round(n * outliers / (1 + outliers))
    areas = [float(((s["a"][0] * s["a"][1]) ** 1.6 + (s["a"][0] * s["a"][2]) ** 1.6
                    + (s["a"][1] * s["a"][2]) ** 1.6) ** (1 / 1.6)) for s in solids]
    got, have = [], 0
    while have < m:
        for i, s in enumerate(solids):
            cnt = int(6 * m * areas[i] / sum(areas)) + 64

            def at(eta, om):
                def fp(x, e):
                    return x.sign() * x.abs() ** e
                return torch.stack([fp(eta.cos(), s["e1"]) * fp(om.cos(), s["e2"]),
                                    fp(eta.cos(), s["e1"]) * fp(om.sin(), s["e2"]), fp(eta.sin(), s["e1"])], 1) * s["a"]
            eta, om = _uniform(g, -math.pi / 2, math.pi / 2, cnt), _uniform(g, -math.pi, math.pi, cnt)
            x = at(eta, om)
            dA = torch.linalg.cross(at(eta + 1e-4, om) - x, at(eta, om + 1e-4) - x).norm(dim=1).nan_to_num(0, 0, 0)
            cap = dA.sort().values[int(0.99 * cnt)] + 1e-20
            x = x[_uniform(g, 0, 1, cnt) * cap < dA] @ s["R"].T + s["c"]
            keep = torch.ones(len(x), dtype=torch.bool, device=DEV)
            for j, t in enumerate(solids):
                if j != i:
                    keep &= _inside(x, t) >= 1
            got.append(x[keep])
            have += len(got[-1])
    P = torch.cat(got)
    P = P[torch.randperm(len(P), generator=g, device=DEV)[:m]]
    lo, hi = P.amin(0), P.amax(0)
    return torch.cat([P, lo + (hi - lo) * _uniform(g, 0, 1, n - m, 3)]), None


def _normalised(P):
    """Centred on the mean, divided by twice the largest coordinate, as the reader does."""
    P = P - P.mean(0)
    return P / (2 * P.abs().max())


def _torus_cloud(n, g):
    P, N = _torus(n, g)
    return _normalised(P).float().contiguous(), N.float().contiguous()


def _near(P, nq, g):
    """Queries as triangle centroids of an early iteration lie: most close to
    the surface, a quarter off it, some far."""
    x = P[torch.randint(len(P), (nq,), generator=g, device=DEV)].double()
    far = _uniform(g, 0, 1, nq, 1)
    s = torch.where(far < 0.75, 0.003, torch.where(far < 0.95, 0.03, 0.15))
    return (x + s * _normal(g, nq, 3)).float().contiguous()


# ------------------------------------------------------------------- cases --
def _areas(n):
    return torch.full((n,), AREA, device=DEV)


def _grid_of(P, res):
    """Samples per axis, origin and spacing of a grid around the points, ``res`` along the longest side."""
    lo, hi = P.amin(0).double() - 0.05, P.amax(0).double() + 0.05
    h = float((hi - lo).max()) / (res - 1)
    return np.ceil(((hi - lo) / h).cpu().numpy() - 1e-9).astype(np.int32) + 1, lo.float().cpu().numpy(), np.float32(h)


def _field(rx, ry, rz, g):
    """A smooth indicator of blobs and tubes with sampling noise near the iso value, x fastest."""
    ax = [torch.arange(r, device=DEV, dtype=torch.float32) / max(rx, ry, rz) for r in (rx, ry, rz)]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    d = torch.full_like(x, 1e3)
    ext = [r / max(rx, ry, rz) for r in (rx, ry, rz)]
    for _ in range(12):
        c, r = _uniform(g, 0.15, 0.85, 3).tolist(), float(_uniform(g, 0.03, 0.22, 1))
        q = ((x - c[0] * ext[0]) ** 2 + (y - c[1] * ext[1]) ** 2 + (z - c[2] * ext[2]) ** 2).sqrt()
        d = torch.minimum(d, (q - r).abs() - 0.15 * r)
    v = torch.sigmoid(-40 * d) - 0.02 * torch.rand(d.shape, generator=g, device=DEV)
    return v.reshape(-1).contiguous()


def _mlp_params(g):
    out = []
    for din, dout in ((16, 128), (128, 128), (128, 128), (128, 8)):
        w = _uniform(g, -1, 1, din, dout) / math.sqrt(din)
        if din == 16:
            w[12:] = 0
        if dout == 8:
            w[:, 3:] = 0
        b = 0.1 * _uniform(g, -1, 1, dout)
        if dout == 8:
            b[3:] = 0
        out += [w.reshape(-1), b]
    return torch.cat(out).float().cpu().numpy()


def prepare(case, seed):
    g, kind = _gen(seed), case["kind"]
    if kind == "reconstruct":
        P = {"sphere": _sphere, "torus": _torus, "union": _union}[case["shape"]](case["n"], g)[0]
        params = capi.default_params(grid_reso=case["grid"], final_reso=case["grid"], total_iter=case["iters"],
                                     com_as=case["com_as"], precision=case["precision"])
        return dict(kind=kind, points=_normalised(P).float().cpu().pin_memory(), params=params,
                    normals=torch.zeros((case["n"], 3)).pin_memory(),
                    tris=torch.zeros((24 * case["grid"] ** 2, 9)).pin_memory())
    if kind == "knn":
        P, _ = _torus_cloud(case["n"], g)
        Q = P if case["queries"] == "self" and case["nq"] >= case["n"] else \
            P[:case["nq"]].contiguous() if case["queries"] == "self" else _near(P, case["nq"], g)
        return dict(kind=kind, points=P, queries=Q, k=case["k"], index=turbo.KnnIndex(P) if case["kept"] else None)
    if kind in ("winding", "gradient", "grid"):
        P, N = _torus_cloud(case["n"], g)
        st = dict(kind=kind, points=P, normals=N, areas=_areas(len(P)), case=case)
        if kind == "grid":
            st["grid"] = _grid_of(P, case["res"])
        else:
            st["queries"] = P if case["nq"] == case["n"] else _near(P, case["nq"], g)
        if case.get("kept", True):
            st["tree"] = turbo.TurboLibiGWN(P, max_depth=10, areas=st["areas"])
            st["tree"].UpdateMassNormals(N, st["areas"])
        return st
    if kind == "mc":
        res = (case["rx"], case["ry"], case["rz"])
        buf = [torch.zeros((24 * max(res) ** 2, c), device=DEV) for c in (9, 3, 3)]
        return dict(kind=kind, field=_field(*res, g), res=res, buf=buf, iso=0.5,
                    origin=np.array([-0.5, -0.4, -0.3], np.float32), spacing=float(np.float32(1.0 / max(res))))
    m = turbo.LearnedNormalInit()
    flat = _mlp_params(g)
    m.set_params(flat)
    # features as the feature pass gives them: eigenvalue fractions, two unit vectors, a centroid offset
    n = case["batch"]
    ev = _uniform(g, 0, 1, n, 3).sort(dim=1, descending=True).values
    vec = [v / v.norm(dim=1, keepdim=True) for v in (_normal(g, n, 3), _normal(g, n, 3), _normal(g, n, 3))]
    x = torch.cat([ev / ev.sum(1, keepdim=True), vec[0], vec[1], 0.4 * _normal(g, n, 3)], 1).float().contiguous()
    return dict(kind=kind, mlp=m, flat=flat, features=x, targets=vec[2].float().contiguous())


def run(st):
    kind = st["kind"]
    if kind == "reconstruct":
        count = ctypes.c_longlong()
        capi.check(capi.load().dwg_reconstruct_host(
            capi.ptr(st["points"]), None, len(st["points"]), ctypes.byref(st["params"]), capi.ptr(st["normals"]),
            capi.ptr(st["tris"]), len(st["tris"]), ctypes.byref(count), capi.stream_ptr()))
        return dict(count=count.value, normals=st["normals"], tris=st["tris"])
    if kind == "knn":
        if st["index"] is not None:
            return st["index"].query(st["queries"], st["k"])
        out = torch.empty((len(st["queries"]), st["k"]), dtype=torch.int32, device=DEV)
        return turbo.CudaKNNWithKDTreeforDWG(st["points"], len(st["points"]), st["queries"], len(st["queries"]), None,
                                             None, out, st["k"])
    if kind == "mc":
        T = turbo.TurboMC().TurboMarchingCubes(
            st["field"], None, *st["res"], st["iso"], origin=st["origin"], spacing=st["spacing"], tris=st["buf"][0],
            mid_points=st["buf"][1], mid_normals=st["buf"][2], capacity=len(st["buf"][0]))
        return dict(count=T, tris=st["buf"][0], centroids=st["buf"][1], normals=st["buf"][2])
    if kind == "mlp":
        loss, grads = st["mlp"].gradients(st["features"], st["targets"])
        return dict(loss=loss, grads=grads)
    case, tree = st["case"], st.get("tree")
    if kind == "grid":
        return tree.grid(*st["grid"], beta=case["beta"], sigma=0.0, screened=False, order=case["order"])
    if kind == "gradient":
        return tree.value_and_gradient(st["queries"], sigma=10.0 if case["screened"] else 0.0,
                                       screened=case["screened"])
    if tree is None:
        tree = turbo.TurboLibiGWN(st["points"], max_depth=10, areas=st["areas"])
    tree.UpdateMassNormals(st["normals"], st["areas"])
    if case["screened"]:
        return tree.TurboLibiScreenedGWNLaunch(st["queries"], sigma=10.0, precision=case["precision"])
    return tree.TurboLibiGWNLaunch(st["queries"], precision=case["precision"])


def work(case):
    kind = case["kind"]
    if kind == "reconstruct":
        # points in; mesh and normals out; every iteration sums the field at the grid and the leaves and meshes it
        n, samples = case["n"], 0.35 * case["grid"] ** 3
        tris = 2.5 * case["grid"] ** 2
        terms = (samples + n) * TERMS_PER_QUERY * math.log2(n)
        return dict(bytes=24.0 * n + 36 * tris + case["iters"] * (8 * samples + 24 * n + 84 * tris),
                    flops=(case["iters"] + 1) * 20.0 * terms)
    if kind == "knn":
        return dict(bytes=12.0 * case["n"] + (12.0 + 4 * case["k"]) * case["nq"], flops=0.0)
    if kind == "mc":
        cells = case["rx"] * case["ry"] * case["rz"]
        return dict(bytes=4.0 * cells + 60.0 * 6 * cells ** (2 / 3), flops=0.0)
    if kind == "mlp":
        net = 12 * 128 + 2 * 128 * 128 + 128 * 3
        return dict(bytes=60.0 * case["batch"] + 8.0 * net, flops=6.0 * net * case["batch"])
    n = case["n"]
    nq = 0.12 * case["res"] ** 3 if kind == "grid" else case["nq"]
    per = {0: 20, 1: 50, 2: 95}[case["order"]] if kind == "grid" else 45 if kind == "gradient" else 20
    out = 4 if kind != "gradient" else 16
    return dict(bytes=28.0 * n + (out + (0 if kind == "grid" else 12)) * nq,
                flops=per * nq * TERMS_PER_QUERY * math.log2(n))


# ---------------------------------------------------------- values in FP64 --
def exact(case, seed):
    """Sums, vertices and gradients in 64 bits by plain torch.  None for the
    reconstructions (minutes of sums) and the neighbour lists (indices)."""
    kind = case["kind"]
    if kind in ("reconstruct", "knn"):
        return None
    st = prepare(case, seed)
    if kind == "mlp":
        return _exact_mlp(st)
    if kind == "mc":
        return _exact_mc(st)
    if kind == "grid":
        res, org, h = st["grid"]
        ax = [np.float32(org[d]) + np.arange(res[d], dtype=np.float32) * h for d in range(3)]
        z, y, x = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
        Q = torch.from_numpy(np.stack([x.ravel(), y.ravel(), z.ravel()], 1)).to(DEV)
        return _sums(st, Q, case["beta"], 0.0, False, case["order"], False)
    screened = case["screened"]
    return _sums(st, st["queries"], 2.3, 10.0 if screened else 0.0, screened, 0, kind == "gradient")


def _octree(P, A, N, D, order):
    """Levels of the Barnes-Hut octree: cells split while they hold more than
    one point, centres of mass, radii and moments in FP64."""
    n = len(P)
    lo, hi = P.amin(0), P.amax(0)
    c, w = ((lo + hi) / 2).repeat(n, 1), float((hi - lo).max())
    key = torch.zeros(n, dtype=torch.int64, device=DEV)
    for _ in range(D):
        bit = P >= c
        key = key * 8 + (bit * torch.tensor([1, 2, 4], device=DEV)).sum(1)
        c = c + torch.where(bit, w / 4, -w / 4)
        w = w / 2
    key, perm = torch.sort(key, stable=True)
    P, A, N = P[perm], A[perm], N[perm]
    at = torch.arange(n, device=DEV)  # the points whose cell was split
    levels = []
    for d in range(D + 1):
        pre = key[at] >> (3 * (D - d))
        _, own, cnt = torch.unique_consecutive(pre, return_inverse=True, return_counts=True)
        m = len(cnt)

        def total(v):
            return torch.zeros((m,) + v.shape[1:], dtype=torch.float64, device=DEV).index_add_(0, own, v)
        mass = total(A[at])
        cm = total(A[at, None] * P[at]) / mass[:, None]
        rel = P[at] - cm[own]
        rad = torch.zeros(m, dtype=torch.float64, device=DEV).scatter_reduce_(0, own, rel.norm(dim=1), "amax")
        an = A[at, None] * N[at]
        lv = dict(start=at[torch.cumsum(cnt, 0) - cnt], count=cnt, cm=cm, rad=rad, ec=total(an),
                  leaf=(cnt == 1) | (d == D))
        if order >= 1:
            lv["m1"] = total(rel[:, :, None] * an[:, None, :])
        if order >= 2:
            lv["m2"] = total(0.5 * rel[:, :, None, None] * rel[:, None, :, None] * an[:, None, None, :])
        if levels:  # the split cells of the level above, in order, own these runs
            up = levels[-1]
            _, kids = torch.unique_consecutive(pre >> 3, return_inverse=True)
            first = torch.full((int((~up["leaf"]).sum()),), m, dtype=torch.int64, device=DEV)
            first.scatter_reduce_(0, kids, own, "amin")
            up["first"] = torch.zeros(len(up["count"]), dtype=torch.int64, device=DEV)
            up["kids"] = torch.zeros_like(up["first"])
            up["first"][~up["leaf"]] = first
            up["kids"][~up["leaf"]] = torch.diff(first, append=torch.tensor([m], device=DEV))
        levels.append(lv)
        at = at[~lv["leaf"][own]]
        if not len(at):
            break
    return P, A, N, levels


def _spread(first, count):
    """For runs [first, first + count): the owner and the element of every member."""
    own = torch.repeat_interleave(torch.arange(len(count), device=DEV), count)
    off = torch.arange(len(own), device=DEV) - (torch.cumsum(count, 0) - count)[own]
    return own, first[own] + off


def _terms(d, e, sigma, screened, grad):
    """Value (and gradient) of the terms with offset d = p - q and moment e = A n."""
    r2, dot = (d * d).sum(1), (d * e).sum(1)
    r = r2.sqrt()
    if screened:
        ok = r > 1e-10
        rho = r.clamp(min=float(np.float32(0.0015)))
        ex = (sigma * rho).exp()
        den, up = ex * 4 * math.pi * rho ** 3 + 1e-7, sigma * rho + 1
        G = up / den
        dG = (sigma * den - up * ex * (sigma * 4 * math.pi * rho ** 3 + 12 * math.pi * rho ** 2)) / den ** 2
        k = torch.where(r > float(np.float32(0.0015)), -dot * dG / r, 0.0)
    else:
        ok = r > 0
        den = 4 * math.pi * r * r2 + 1e-8
        G, k = 1 / den, dot * 12 * math.pi * r / den ** 2
    v = torch.where(ok, G * dot, 0.0)
    return v, torch.where(ok[:, None], k[:, None] * d - G[:, None] * e, 0.0) if grad else None


def _expansion(loc, m1, m2):
    """igl::fast_winding_number's far-field terms of orders 1 and 2."""
    r = loc.norm(dim=1)
    p3, p5, p7 = (4 * math.pi * r ** q for q in (3, 5, 7))
    v = m1.diagonal(dim1=1, dim2=2).sum(1) / p3 - 3 * torch.einsum("pu,pv,puv->p", loc, loc, m1) / p5
    if m2 is not None:
        tr = torch.einsum("piuu->pi", m2) + torch.einsum("piiv->pv", m2) + torch.einsum("piui->pu", m2)
        v += 15 * torch.einsum("pi,pu,pv,piuv->p", loc, loc, loc, m2) / p7 - 3 * (loc * tr).sum(1) / p5
    return v


def _sums(st, Q, beta, sigma, screened, order, grad):
    P, A, N, levels = _octree(st["points"].double(), st["areas"].double(), st["normals"].double(), 10, order)
    w = torch.zeros(len(Q), dtype=torch.float64, device=DEV)
    gr = torch.zeros((len(Q), 3), dtype=torch.float64, device=DEV)

    def add(qi, d, e, extra=None):
        v, t = _terms(d, e, sigma, screened, grad)
        w.index_add_(0, qi, v if extra is None else v + extra)
        if grad:
            gr.index_add_(0, qi, t)
    for b in range(0, len(Q), 30000):
        qi = torch.arange(b, min(b + 30000, len(Q)), device=DEV)
        node = torch.zeros_like(qi)
        for lv in levels:
            leaf = lv["leaf"][node]
            own, j = _spread(lv["start"][node[leaf]], lv["count"][node[leaf]])
            ql = qi[leaf][own]
            add(ql, P[j] - Q[ql].double(), A[j, None] * N[j])
            qi, node = qi[~leaf], node[~leaf]
            d = lv["cm"][node] - Q[qi].double()
            far = d.norm(dim=1) > beta * lv["rad"][node]
            f = node[far]
            extra = _expansion(d[far], lv["m1"][f], lv["m2"][f] if order > 1 else None) if order else None
            add(qi[far], d[far], lv["ec"][f], extra)
            qi, node = qi[~far], node[~far]
            if not len(qi):
                break
            own, node = _spread(lv["first"][node], lv["kids"][node])
            qi = qi[own]
    return (w, gr) if grad else w


def _exact_mlp(st):
    flat = torch.from_numpy(st["flat"]).to(DEV).double().requires_grad_(True)
    h = torch.nn.functional.pad(st["features"].double(), (0, 4))
    o = 0
    for layer, (din, dout) in enumerate(((16, 128), (128, 128), (128, 128), (128, 8))):
        h = h @ flat[o:o + din * dout].view(din, dout) + flat[o + din * dout:o + din * dout + dout]
        o += din * dout + dout
        if layer < 3:
            h = torch.nn.functional.gelu(h)
    y = h[:, :3]
    loss = (1 - ((y / (y.norm(dim=1, keepdim=True) + 1e-12)) * st["targets"].double()).sum(1)).mean()
    loss.backward()
    return dict(loss=loss.detach(), grads=flat.grad)


# The triangles of the 256 marching-cubes cases, three edges each ("-": none).
# Bit c of a case is set where corner c is above the iso value; the corners go
# round the cell's top (0-3), then its bottom (4-7); edges 0-3 go round the
# top, 4-7 round the bottom, 8-11 join the two.
CASES = (
    "- 083 019 183981 12a 08312a 92a029 2832a8a98 3b2 0b28b0 19023b 1b219b98b 3a1ba3 0a108a8ba 3903b9ba9 "
    "98aa8b 478 430734 019847 419471731 12a847 34730412a 92a902847 2a9297273794 8473b2 b47b24204 "
    "90184723b 47b94b9b2921 3a13ba784 1ba14b1047b4 47890b9bab03 47b4b99ba 954 954083 054150 854835315 "
    "12a954 30812a495 52a542402 2a5325354348 95423b 0b208b495 05401523b 21525828b485 a3ba13954 "
    "4950818a18ba 54050b5bab03 54858aa8b 978579 930953573 078017157 153357 978957a12 a12950530573 "
    "802825857a52 2a5253357 7957893b2 95797292027b 23b018178157 b21b17715 958857a13a3b 5705097b010aba0 "
    "ba0b03a50807570 ba57b5 a65 0835a6 9015a6 1831985a6 165261 165126308 965906026 598582526328 23ba65 "
    "b08b20a65 01923b5a6 5a61929b298b 63b653513 08b0b50515b6 3b6036065059 65969bb98 5a6478 43047365a "
    "1905a6847 a65197173794 612651478 125526304347 847905065026 739794329596269 3b2784a65 5a647242027b "
    "01947823b5a6 9219b294b7b45a6 8473b53515b6 51b5b610b7b404b 059065036b63847 65969b4797b9 a4964a "
    "4a649a083 a01a60640 83181686461a 149124264 308129249264 024426 832824426 a49a64b23 08228b49a4a6 "
    "3b201606461a 64161a48121b8b1 964936913b63 8b1810b61914641 3b6360064 648b68 7a678a89a 0730a709a67a "
    "a671a7178180 a67a71173 126168189867 269291679093739 780706602 732672 23ba68a89867 20727b09767a9a7 "
    "1801781a767a23b b21b17a61671 896867916b63136 091b67 7807063b0b60 7b6 76b 308b76 019b76 819831b76 "
    "a126b7 12a3086b7 2902a96b7 6b72a3a83a98 723627 708760620 276237019 162186198876 a76a17137 "
    "a7617a187108 03707a0a96a7 76a7a88a9 684b86 36b306046 86b846901 946963931b36 6846b82a1 12a30b06b046 "
    "4b846b0292a9 a93a32943b36463 823842462 042462 190234246438 194142246 8138618466a1 a10a06604 "
    "4634386a3039a93 a946a4 49576b 083495b76 50154076b b76834354315 954a1276b 6b712a083495 76b54a42a402 "
    "348354325a52b76 723762549 954086062687 362376150540 628687218485158 954a16176137 16a176107870954 "
    "40a4a503a6a737a 76a7a854a48a 6956b9b89 36b063056095 0b805b01556b 6b3635531 12a95b9b8b56 "
    "0b306b09656912a b85b56805a52025 6b36352a3a53 589528562382 956960062 158180568382628 156216 "
    "13616a386569896 a10a06950560 03856a a56 b5a75b b5ab75830 5b75ab190 a75ab7981831 b12b71751 "
    "08312717572b 9759279022b7 75272b592328982 25a235375 820852875a25 9015a35373a2 982921872a25752 135375 "
    "087071175 903935537 987597 5845a8ab8 5045b05abb30 01984a8aba45 ab4a45b34941314 2512852b8458 "
    "04b0b345b2b151b 0250592b5458b85 9452b3 25a352345384 5a2524420 3a235a385458019 5a2524192942 845853351 "
    "045105 845853905035 945 4b749b9ab 0834979b79ab 1ab1b414074b 3143481a474bab4 4b79b492b912 "
    "9749b791b2b1083 b74b42240 b74b42834324 29a279237749 9a7974a27870207 37a3a274a1a040a 1a2874 491417713 "
    "491417081871 403743 487 9a8ab8 30939bb9a 01a0a88ab 31ab3a 12b1b99b8 30939b1292b9 02b80b 32b "
    "23828aa89 9a2092 23828a0181a8 1a2 138918 091 038 - "
).split()
CORNERS = ((0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1), (0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0))
EDGES = ((0, 1), (1, 2), (2, 3), (3, 0), (4, 5), (5, 6), (6, 7), (7, 4), (0, 4), (1, 5), (2, 6), (3, 7))


def _exact_mc(st):
    rx, ry, rz = st["res"]
    v = st["field"].view(rz, ry, rx)
    corner = [v[z:rz - 1 + z, y:ry - 1 + y, x:rx - 1 + x].reshape(-1) for x, y, z in CORNERS]
    case = sum((c > st["iso"]).long() << i for i, c in enumerate(corner))
    most = max(len(t) for t in CASES) // 3
    table = torch.full((256, most, 3), -1, dtype=torch.int64)
    for i, t in enumerate(CASES):
        for j in range(len(t) // 3):
            table[i, j] = torch.tensor([int(e, 16) for e in t[3 * j:3 * j + 3]])
    table = table.to(DEV)
    cell, k = (table[:, :, 0] >= 0)[case].nonzero(as_tuple=True)  # in cell order, then case order
    edge = table[case[cell], k]
    at = torch.stack([cell % (rx - 1), cell // (rx - 1) % (ry - 1), cell // ((rx - 1) * (ry - 1))], 1)
    org = torch.tensor(st["origin"], device=DEV).double()
    corners, edges = torch.tensor(CORNERS, device=DEV), torch.tensor(EDGES, device=DEV)
    values = torch.stack([c[cell] for c in corner], 1).double()
    verts = []
    for t in range(3):
        a, b = edges[edge[:, t], 0], edges[edge[:, t], 1]
        p, q = (org + (at + corners[i]) * st["spacing"] for i in (a, b))
        va, vb = (values.gather(1, i[:, None])[:, 0] for i in (a, b))
        verts.append(p - ((va - st["iso"]) / (vb - va + 1e-10))[:, None] * (q - p))
    cross = torch.linalg.cross(verts[1] - verts[0], verts[2] - verts[0])

    def filled(x):  # the rest of the output buffer holds zeros
        return torch.nn.functional.pad(x, (0, 0, 0, len(st["buf"][0]) - len(x)))
    return dict(count=None, tris=filled(torch.cat(verts, 1)), centroids=filled(sum(verts) / 3),
                normals=filled(-cross / (cross.norm(dim=1, keepdim=True) + 1e-8)))
