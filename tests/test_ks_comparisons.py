"""The KS decision as comparisons at fixed places (kernels_shp.cu:
tc_shp_ks_kernel) equals the reference's merge walk (tcoh.cl:34-54), ties, every
threshold and both choices of the centre included."""

import numpy as np
import pytest


def walk(a, b, m):
    """tcoh.cl:34-54: the centre a goes first on ties."""
    ia = ib = d = 0
    n = len(a)
    while ia < n and ib < n:
        if a[ia] <= b[ib]:
            ia += 1
        else:
            ib += 1
        d = max(d, abs(ia - ib))
    return d <= m


def comparisons(a, b, m):
    """The kernel's form: b against a shifted by m either way, NaN outside;
    the second value with b as the centre."""
    n = len(a)
    nan = np.full(n, np.nan)
    lo = np.concatenate([nan, a])[n - min(m, n):2 * n - min(m, n)]
    hi = np.concatenate([a, nan])[min(m, n):min(m, n) + n]
    with np.errstate(invalid="ignore"):
        fwd = not ((b >= hi) | (lo > b)).any()
        rev = not ((b > hi) | (lo >= b)).any()
    return fwd, rev


@pytest.mark.parametrize("n", [2, 3, 7, 10, 30, 33, 64])
def test_equals_the_merge_walk(n):
    rng = np.random.default_rng(n)
    for trial in range(150):
        levels = (2, 5, n, 10 * n)[trial % 4]  # from nearly all values tied to few
        a = np.sort(rng.integers(0, levels, n)).astype(np.float32)
        b = np.sort(rng.integers(0, levels, n) + rng.integers(0, 3)).astype(np.float32)
        for m in (0, 1, 2, n // 3, n // 2, n - 1, n, n + 3):
            assert comparisons(a, b, m) == (walk(a, b, m), walk(b, a, m)), (a, b, m)
