"""Coherences whose square is below the smallest normal float (B200 only): the
goodness of fit takes their phase all the same. Two dates whose energy lies in
different pixels of every window, 20 orders of magnitude above the rest, have
|T| of about 1e-20 while every other pair is well coherent."""

import numpy as np
import pytest

import oracle
import tcoh_b200
from conftest import TOLERANCE

pytestmark = pytest.mark.gpu

WINDOW = (9, 5)


def stack_of(n, rows, cols):
    """Dates 0 and 1 strong (1e10) in a third of the pixels each, not the same
    ones, and weak (1e-10) elsewhere; the other dates strong everywhere."""
    rng = np.random.default_rng(n)
    kind = rng.integers(0, 3, (rows, cols))
    a = np.full((n, rows, cols), 1e10)
    a[2:] *= rng.uniform(0.7, 1.3, (n - 2, rows, cols))
    a[0][kind != 0] = 1e-10
    a[1][kind != 1] = 1e-10
    ph = 0.9 * np.arange(n)[:, None, None] + rng.normal(0.0, 0.3, (n, rows, cols))
    return (a * np.exp(1j * ph)).astype(np.complex64)


def strip_of(n, rows, cols):
    stack = stack_of(n, rows, cols)
    return stack, tcoh_b200.read_strip(stack.real, stack.imag, -(WINDOW[0] // 2),
                                       rows + WINDOW[0] - 1, WINDOW[1] // 2)


@pytest.mark.parametrize("estimator", ["evd", "emi"])
@pytest.mark.parametrize("n", [2, 3, 10, 16, 17, 30, 32, 40])
def test_goodness_of_fit(n, estimator):
    """Two dates fit their one phase exactly, whatever its coherence."""
    rows, cols = 14, 11
    kw = dict(window=WINDOW, shp_test="ks", alpha=0.01, min_shp=20, estimator=estimator,
              bias=False)
    _, (slc, amp, valid) = strip_of(n, rows, cols)
    s = tcoh_b200.make_settings(n, pairs=True, pairs_all=True, **kw)
    with tcoh_b200.Backend(s, cols + WINDOW[1] - 1) as be:
        r = be.run(slc, amp, valid, rows, cols)
    o = oracle.run_oracle(slc, amp, valid, rows, cols, shp_fp32=True, npairs=s.npairs,
                          pairs_all=True, **kw)
    m = ~np.isnan(o["coh"])
    assert m.sum() > rows * cols // 3
    t01 = o["pairs"][0][m]
    assert ((t01 > 4e-23) & (t01 < 1.1e-19)).sum() > m.sum() // 2
    assert np.array_equal(r["count"], o["count"])
    assert np.isfinite(r["coh"][m]).all()
    if n == 2:
        assert np.abs(r["coh"][m] - 1.0).max() <= 1e-6
    else:
        assert np.abs(r["coh"][m] - o["coh"][m]).max() <= TOLERANCE


def test_adjoint_value():
    """The adjoint's forward part is the same stage."""
    n, rows, cols = 8, 14, 11
    kw = dict(window=WINDOW, shp_test="ks", alpha=0.01, min_shp=20, estimator="evd", bias=False)
    stack, (slc, amp, valid) = strip_of(n, rows, cols)
    ha = WINDOW[0] // 2
    re, im = (np.full((n, rows + 2 * ha, cols), np.nan, np.float32) for _ in range(2))
    re[:, ha:ha + rows], im[:, ha:ha + rows] = stack.real, stack.imag
    s = tcoh_b200.make_settings(n, **kw)
    with tcoh_b200.Backend(s, cols + WINDOW[1] - 1) as be:
        r = be.adjoint_raw(re, im, None, None, None, -ha, rows, rows, cols)
    o = oracle.run_oracle(slc, amp, valid, rows, cols, shp_fp32=True, **kw)
    m = ~np.isnan(o["coh"])
    assert m.any() and np.abs(r["coh"][m] - o["coh"][m]).max() <= TOLERANCE
