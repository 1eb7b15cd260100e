"""Gradients of the winding-number sums and the FP64 sums on the GPU
(dwg_gwn_points_grad / _grid_grad / _points_fp64 / _grid_fp64) against the
FP64 oracle with the same opening decisions.  The oracle's gradient itself is
checked against central differences in tests/test_oracle.py."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from dwg_b200 import datasets as D, turbo  # noqa: E402

pytestmark = pytest.mark.gpu


def cu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.fixture(scope="module")
def case(oracle_lib):
    P, N = D.torus(20000, seed=21)
    Pn, _, _ = D.normalize(P)
    rng = np.random.default_rng(3)
    A = rng.uniform(1e-6, 3e-6, len(Pn)).astype(np.float32)
    R = rng.uniform(0.001, 0.004, len(Pn)).astype(np.float32)
    Q = np.concatenate([Pn[:4000] + rng.normal(0, 0.01, (4000, 3)),
                        rng.uniform(-0.55, 0.55, (6000, 3))]).astype(np.float32)
    return Pn, N.astype(np.float32), A, R, Q


@pytest.mark.parametrize("screened,sigma,radii", [(True, 20.0, False), (True, 10.0, True), (False, 0.0, False)])
def test_fp64_sums_and_gradients_match_oracle(oracle_lib, case, screened, sigma, radii):
    Pn, N, A, R, Q = case
    tree = turbo.TurboLibiGWN(cu(Pn), max_depth=8, areas=cu(A))
    Rd = cu(R) if radii else None
    tree.UpdateMassNormals(cu(N), cu(A))
    w64, g64 = tree.value_and_gradient(cu(Q), i_Normals=cu(N), i_As=cu(A), i_radii=Rd, beta=2.3, sigma=sigma,
                                       screened=screened, fp64=True)
    w32, g32 = tree.value_and_gradient(cu(Q), i_Normals=cu(N), i_As=cu(A), i_radii=Rd, beta=2.3, sigma=sigma,
                                       screened=screened)
    assert tree.status() == 0
    ot = oracle_lib.Octree(Pn, 8)
    wo, go = ot.gwn_grad(Pn, N, A, Q, beta=2.3, sigma=sigma, screened=screened, radii=R if radii else None)
    w64, g64 = w64.cpu().numpy(), g64.cpu().numpy()
    w32, g32 = w32.cpu().numpy().astype(np.float64), g32.cpu().numpy().astype(np.float64)
    sw, sg = np.abs(wo).max(), np.abs(go).max()
    # FP64 on the GPU = the oracle's FP64 sums up to the order of the additions
    assert np.abs(w64 - wo).max() <= 1e-11 * sw, np.abs(w64 - wo).max() / sw
    assert np.abs(g64 - go).max() <= 1e-11 * sg, np.abs(g64 - go).max() / sg
    # FP32 terms summed in FP64: FP32 rounding of each term
    ew, eg = np.abs(w32 - wo), np.abs(g32 - go)
    assert ew.max() <= 1e-5 * sw and np.sqrt(np.mean(ew ** 2)) <= 1e-6 * sw, (ew.max() / sw)
    assert eg.max() <= 1e-4 * sg and np.sqrt(np.mean(eg ** 2)) <= 1e-5 * sg, (eg.max() / sg)
    # the values equal the warp kernels' sums to FP32 rounding
    if not radii:
        out = torch.empty(len(Q), dtype=torch.float32, device="cuda")
        if screened:
            tree.TurboLibiScreenedGWNLaunch(cu(Q), None, len(Q), None, None, None, 2.3, sigma, out)
        else:
            tree.TurboLibiGWNLaunch(cu(Q), None, len(Q), None, None, 2.3, out)
        wk = out.cpu().numpy().astype(np.float64)
        assert np.abs(wk - wo).max() <= 1e-5 * sw


def test_grid_fp64_and_gradient_match_points(oracle_lib, case):
    Pn, N, A, R, Q = case
    tree = turbo.TurboLibiGWN(cu(Pn), max_depth=8, areas=cu(A))
    tree.UpdateMassNormals(cu(N), cu(A))
    res, org, h = np.array([23, 19, 11], np.int32), np.array([-0.55, -0.5, -0.2], np.float32), np.float32(0.045)
    wg, gg = tree.value_and_gradient(grid=(res, org, h), beta=2.3, sigma=20.0, fp64=True)
    z, y, x = np.meshgrid(np.arange(res[2]), np.arange(res[1]), np.arange(res[0]), indexing="ij")
    G = np.stack([org[0] + x.astype(np.float32) * h, org[1] + y.astype(np.float32) * h,
                  org[2] + z.astype(np.float32) * h], -1).reshape(-1, 3).astype(np.float32)
    wp, gp = tree.value_and_gradient(cu(G), beta=2.3, sigma=20.0, fp64=True)
    assert np.array_equal(wg.cpu().numpy(), wp.cpu().numpy())
    assert np.array_equal(gg.cpu().numpy(), gp.cpu().numpy())
    # and the FP32 grid sums of the warp kernels sit within FP32 rounding of them
    w32 = tree.grid(res, org, h, sigma=20.0).cpu().numpy().astype(np.float64)
    w64 = wg.cpu().numpy()
    assert np.abs(w32 - w64).max() <= 1e-5 * np.abs(w64).max()


@pytest.mark.parametrize("screened", [True, False])
def test_sums_do_not_depend_on_the_call(case, screened):
    # a query's value and gradient are the same bits alone and in any call:
    # groups of 1, 2, 4, 8, 16 and 32 queries and their last, partial groups
    # (3,552 warps fill the GPU: up to 3,552, 7,104, ... queries)
    Pn, N, A, R, Q = case
    tree = turbo.TurboLibiGWN(cu(Pn), max_depth=8, areas=cu(A))
    tree.UpdateMassNormals(cu(N), cu(A))
    rng = np.random.default_rng(8)
    q = np.concatenate([Q, Pn[rng.integers(0, len(Pn), 115000)] + rng.normal(0, 0.02, (115000, 3))])
    q = cu(q[rng.permutation(len(q))].astype(np.float32))
    kw = dict(sigma=20.0 if screened else 0.0, screened=screened)

    def values(x, precision):
        if screened:
            return tree.TurboLibiScreenedGWNLaunch(x, sigma=20.0, precision=precision)
        return tree.TurboLibiGWNLaunch(x, precision=precision)
    full = [values(q, p) for p in (0, 1, 2, 3)]
    w, g = tree.value_and_gradient(q, **kw)
    for m in (1, 2, 33, 3552, 3553, 10000, 20001, 50000, 60001):
        x = q[:m].contiguous()
        for p in (0, 1, 2, 3):
            assert torch.equal(values(x, p), full[p][:m]), (m, p)
        w2, g2 = tree.value_and_gradient(x, **kw)
        assert torch.equal(w2, w[:m]) and torch.equal(g2, g[:m]), m
    assert tree.status() == 0


def test_gradients_and_fp64_sums_of_two_streams(case):
    # calls of one octree that overlap: each has its own order of the queries
    Pn, N, A, R, Q = case
    tree = turbo.TurboLibiGWN(cu(Pn), max_depth=8, areas=cu(A))
    tree.UpdateMassNormals(cu(N), cu(A))
    rng = np.random.default_rng(9)
    near = (Pn[rng.integers(0, len(Pn), 31000)] + rng.normal(0, 0.02, (31000, 3))).astype(np.float32)
    sets = [cu(Q[:7001]), cu(near)]
    ref = [(*tree.value_and_gradient(x, sigma=20.0), *tree.value_and_gradient(x, sigma=20.0, fp64=True)) for x in sets]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in sets]
    got = [[], []]
    for _ in range(6):
        for i in (0, 1):
            with torch.cuda.stream(streams[i]):
                got[i].append((*tree.value_and_gradient(sets[i], sigma=20.0),
                               *tree.value_and_gradient(sets[i], sigma=20.0, fp64=True)))
    torch.cuda.synchronize()
    for i in (0, 1):
        for out in got[i]:
            assert all(torch.equal(a, b) for a, b in zip(out, ref[i]))
    assert tree.status() == 0


@pytest.mark.parametrize("res", [(1, 1, 1), (5, 3, 2), (23, 19, 11), (33, 40, 30), (70, 61, 54)])
@pytest.mark.parametrize("screened", [True, False])
def test_grid_gradients_match_fp64(case, res, screened):
    # FP32 gradients at a grid: bricks cut at its ends, parts of a brick of 1
    # to 32 samples; tolerances as at points, relative to the sums at points
    Pn, N, A, R, Q = case
    tree = turbo.TurboLibiGWN(cu(Pn), max_depth=8, areas=cu(A))
    tree.UpdateMassNormals(cu(N), cu(A))
    kw = dict(beta=2.3, sigma=20.0 if screened else 0.0, screened=screened)
    sw, sg = (float(t.abs().max()) for t in tree.value_and_gradient(cu(Q), fp64=True, **kw))
    res = np.array(res, np.int32)
    grid = (res, np.array([-0.52, -0.5, -0.2], np.float32), np.float32(1.0 / max(res.max(), 2)))
    w64, g64 = tree.value_and_gradient(grid=grid, fp64=True, **kw)
    w32, g32 = tree.value_and_gradient(grid=grid, **kw)
    ew, eg = (w32.double() - w64).abs(), (g32.double() - g64).abs()
    assert float(ew.max()) <= 1e-5 * sw and float((ew ** 2).mean()) ** 0.5 <= 1e-6 * sw
    assert float(eg.max()) <= 1e-4 * sg and float((eg ** 2).mean()) ** 0.5 <= 1e-5 * sg
    assert tree.status() == 0


def test_fp64_sums_do_not_depend_on_the_call(case):
    # with and without a spatial order
    Pn, N, A, R, Q = case
    tree = turbo.TurboLibiGWN(cu(Pn), max_depth=8, areas=cu(A))
    tree.UpdateMassNormals(cu(N), cu(A))
    w, g = tree.value_and_gradient(cu(Q), sigma=20.0, fp64=True)
    for m in (1, 256, 257):
        w2, g2 = tree.value_and_gradient(cu(Q[:m]), sigma=20.0, fp64=True)
        assert torch.equal(w2, w[:m]) and torch.equal(g2, g[:m])
