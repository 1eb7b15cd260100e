"""The row arithmetic of the near neighbour search (k_knn_near), restated on
the CPU: how many cells a window about a query spans, and the quotient that
numbers the rows of a window."""
import numpy as np
import pytest

F = np.float32


def cells(u, inv_h, G):
    return np.clip(np.floor((u * inv_h).astype(F)), 0, G - 1).astype(np.int64)


@pytest.mark.parametrize("points", [1000, 300000, 20000000])
@pytest.mark.parametrize("width", [3e-12, 2e-6, 1.0, 1e6])
def test_windows_stay_within_the_row_numbers(points, width):
    most = min(1024, int(np.ceil(np.sqrt(points / 14.0))))
    h = max(F(width / most) * F(1.0001), F(1e-12))
    G = max(1, int(np.ceil(F(width) / h)))
    inv_h = F(1) / h
    eps = (F(1e-4) + F(G) * F(1.0 / 2097152)) * h
    rng = np.random.default_rng(points)
    u = np.concatenate([rng.uniform(-4 * h, width + 4 * h, 20000), np.arange(G + 1) * float(h)]).astype(F)
    reach = F(3.3) * h * F(1.0002) + eps  # the widest radius, its square root rounded up
    wide = cells(u + reach, inv_h, G) - cells(u - reach, inv_h, G) + 1
    assert wide.max() <= 15


def test_row_quotient_is_exact():
    # inv = trunc(65536 / ny, to 2 ulp) + 1
    for ny in range(1, 16):
        for q in (65536.0 / ny * (1 - 2.0 ** -22), 65536.0 / ny, 65536.0 / ny * (1 + 2.0 ** -22)):
            i = np.arange(min(256, 15 * ny))
            assert np.array_equal(i * (int(q) + 1) >> 16, i // ny), (ny, q)
