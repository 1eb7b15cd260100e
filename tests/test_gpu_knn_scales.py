"""Exact neighbours whatever the cloud's place and size: clouds far from the
origin, and clouds far smaller and far larger than 1, against brute force over all keys on the GPU."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from dwg_b200 import turbo  # noqa: E402

pytestmark = pytest.mark.gpu


def brute(P, Q, k):
    """The k smallest keys (bits of the squared distance, rounded operation by
    operation in FP32, then the index) of every query."""
    idx = torch.arange(len(P), device=P.device, dtype=torch.int64)
    out = []
    for q in Q.split(max(1, 200_000_000 // len(P))):
        d = [P[None, :, c] - q[:, c, None] for c in range(3)]
        d2 = (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2]
        key = (d2.contiguous().view(torch.int32).to(torch.int64) << 32) | idx[None, :]
        out.append((key.topk(k, dim=1, largest=False, sorted=True).values & 0xffffffff).to(torch.int32))
    return torch.cat(out)


def torus(n, seed):
    """About 1 wide."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    th, ph = (torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (2 * np.pi) for _ in range(2))
    ring = 0.37 + 0.13 * ph.cos()
    return torch.stack([ring * th.cos(), ring * th.sin(), 0.13 * ph.sin()], 1), g


@pytest.mark.parametrize("n,offset,k", [(1000000, 5e3, 15), (1000000, 1e4, 10), (100000, 4e4, 15), (100000, 9e4, 16),
                                        (100000, 9e4, 1), (100000, 9e4, 32), (20000, -3e5, 8)])
def test_knn_far_from_the_origin(n, offset, k):
    # coordinates whose rounding is a cell's thousandth up to cells: cells,
    # faces and reaches have to be those of the points as they are stored.
    # Queries on the points, near them, and off the surface
    P, g = torus(n, seed=k)
    off = torch.tensor([offset, -0.7 * offset, 0.9 * offset], device="cuda", dtype=torch.float64)
    m = 6000
    sel = torch.randint(n, (3 * m,), generator=g, device="cuda")
    Q = P[sel]
    Q[m:] += torch.randn(2 * m, 3, generator=g, device="cuda", dtype=torch.float64) * 3e-3
    Q[2 * m:] *= torch.rand(m, 1, generator=g, device="cuda", dtype=torch.float64) * 1.5
    P, Q = (P + off).float().contiguous(), (Q + off).float().contiguous()
    got = turbo.KnnIndex(P).query(Q, k)
    assert torch.equal(got, brute(P, Q, k))


@pytest.mark.parametrize("n,width,k", [(300000, 2e-6, 15), (100000, 2e-6, 10), (1000000, 1e-5, 16), (100000, 1e-9, 1),
                                       (100000, 2e-6, 32), (3000, 3e-12, 15)])
def test_knn_of_tiny_clouds(n, width, k):
    # many cells an axis, each far below 1e-6: a reach has to stay a few cells
    P, g = torus(n, seed=k)
    m = 3000
    sel = torch.randint(n, (3 * m,), generator=g, device="cuda")
    Q = P[sel]
    Q[m:] += torch.randn(2 * m, 3, generator=g, device="cuda", dtype=torch.float64) * 3e-3
    Q[2 * m:] *= torch.rand(m, 1, generator=g, device="cuda", dtype=torch.float64) * 1.5
    P, Q = (P * width).float().contiguous(), (Q * width).float().contiguous()
    got = turbo.KnnIndex(P).query(Q, k)
    assert torch.equal(got, brute(P, Q, k))


@pytest.mark.parametrize("width,offset", [(4e19, 0.0), (1e21, 0.0), (1e38, 0.0), (1e38, 2.5e38), (6e37, -3e38)])
@pytest.mark.parametrize("k", [10, 15])
def test_knn_of_huge_clouds(width, offset, k):
    # squares, and sums of two coordinates, beyond the largest number: such
    # distances are all equal, and the smaller index comes first
    P, g = torus(6000, seed=k)
    Q = torch.cat([P[:500], P[500:1000] * 1.3, -P[1000:1100]])
    P, Q = (P * width + offset).float().contiguous(), (Q * width + offset).float().contiguous()
    assert torch.isfinite(P).all() and torch.isfinite(Q).all()
    Q[-20:, 1] = 3.4e38
    Q[-10:, 2] = -3.4e38
    got = turbo.KnnIndex(P).query(Q, k)
    assert torch.equal(got, brute(P, Q, k))


@pytest.mark.parametrize("n", [14, 100, 6000])
@pytest.mark.parametrize("k", [5, 14])
def test_knn_of_queries_at_infinity(n, k):
    # every distance is infinite: the smallest indices, in a grid of one cell
    # (points at one spot) as in one of many
    P = torch.full((n, 3), 0.25, device="cuda") if n < 1000 else torus(n, 1)[0].float().contiguous()
    inf = float("inf")
    Q = torch.tensor([[inf, 0, 0], [0, inf, 0], [0, 0, inf], [-inf, 0, 0], [0, -inf, 0], [0, 0, -inf],
                      [inf, -inf, inf]], device="cuda")
    got = turbo.KnnIndex(P).query(Q, k)
    assert torch.equal(got, torch.arange(k, device="cuda", dtype=torch.int32).expand(len(Q), k))


@pytest.mark.parametrize("m", [512, 513])
@pytest.mark.parametrize("k", [10, 20])
def test_knn_of_few_queries(m, k):
    # up to 512 queries are taken as they come
    P, g = torus(20000, seed=k)
    Q = P[torch.randint(20000, (m,), generator=g, device="cuda")]
    Q[::3] *= 1.7
    P, Q = P.float().contiguous(), Q.float().contiguous()
    assert torch.equal(turbo.KnnIndex(P).query(Q, k), brute(P, Q, k))
