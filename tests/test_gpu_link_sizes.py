"""The link kernels at the edges of their ranges of dates (B200 only): the
half-warp kernel's padded rows and columns (up to 32 dates) and the two-warp
kernel's blocks of eight columns, its second warp's last rows and its pixels per
CTA (33 to 64 dates), the double-precision tier's rows and columns in registers,
against the double-precision oracle."""

import numpy as np
import pytest

import oracle
import tcoh_b200
import tcoh_b200.synthetic as syn
from conftest import TOLERANCE

pytestmark = pytest.mark.gpu


def compare(n, rows, cols, scale=300.0, **kw):
    """A stack with its own scale through Backend.run and the oracle: counts and
    NULL masks equal, coherence and the pair coherences of at least 0.02 (below,
    the bias correction amplifies the float sums) within the tolerance."""
    window = kw["window"]
    ha, hr = window[0] // 2, window[1] // 2
    stack = syn.generate(n, rows, cols, nregions=3, g0_max=0.95, seed=100 + n, null_frac=0.02)
    stack = (stack * np.float32(scale / 300.0)).astype(np.complex64)
    slc, amp, valid = tcoh_b200.read_strip(stack.real, stack.imag, -ha, rows + 2 * ha, hr)
    s = tcoh_b200.make_settings(n, pairs=True, pairs_all=True, **kw)
    with tcoh_b200.Backend(s, cols + 2 * hr) as be:
        r = be.run(slc, amp, valid, rows, cols, phases=True)
    o = oracle.run_oracle(slc, amp, valid, rows, cols, shp_fp32=True, npairs=s.npairs,
                          pairs_all=True, **kw)
    assert np.array_equal(r["count"], o["count"])
    assert np.array_equal(np.isnan(r["coh"]), np.isnan(o["coh"]))
    assert np.array_equal(np.isnan(r["phases"]).all(axis=2), np.isnan(o["coh"]))
    m = ~np.isnan(o["coh"])
    assert m.any()
    assert np.abs(r["coh"][m] - o["coh"][m]).max() <= TOLERANCE
    big = np.nan_to_num(o["pairs"]) >= 0.02
    assert np.abs(r["pairs"][big] - o["pairs"][big]).max() <= TOLERANCE


@pytest.mark.parametrize("estimator", ["evd", "emi"])
@pytest.mark.parametrize("n", [2, 15, 16, 17, 31, 32])
def test_half_warp_kernel(n, estimator):
    compare(n, 19, 9, window=(21, 7), shp_test="ks", alpha=0.01, min_shp=20,
            estimator=estimator, bias=n > 2 and n % 2 == 1)


@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("n", [33, 40, 41, 62, 63, 64])
def test_two_warp_kernel(n, bias):
    compare(n, 18, 7, window=(21, 7), shp_test="ks", alpha=0.01, min_shp=20, estimator="evd",
            bias=bias)


@pytest.mark.parametrize("n", [3, 5, 29, 32, 33, 34, 40, 63, 64])
def test_exact_tier_emi(n):
    """EMI in double precision: every pixel above 32 dates, below it the pixels
    that the bias correction's threshold sends there."""
    compare(n, 18, 7, window=(21, 7), shp_test="ks", alpha=0.01, min_shp=20, estimator="emi",
            bias=True)


@pytest.mark.parametrize("scale", [3.0e-12, 3.0e11])
def test_two_warp_kernel_far_scales(scale):
    """Sums beyond the branch-free quotients' range take the general form."""
    compare(35, 17, 9, scale=scale, window=(21, 7), shp_test="ks", alpha=0.01, min_shp=20,
            estimator="evd", bias=True)


def test_two_dates_with_a_binding_ks_threshold():
    """Two dates make one staged pair per candidate; alpha = 0.9 puts ks_max
    below n, so that the comparisons decide."""
    compare(2, 19, 9, window=(21, 7), shp_test="ks", alpha=0.9, min_shp=20, estimator="evd",
            bias=False)


@pytest.mark.parametrize("window", [(1, 7), (21, 1), (3, 3)])
@pytest.mark.parametrize("shp_test", ["ks", "ad", "tlog"])
def test_narrow_windows(window, shp_test):
    """Windows of one row or one column (the pair kernels divide by their
    sizes)."""
    compare(3, 23, 17, window=window, shp_test=shp_test, alpha=0.05, min_shp=3,
            estimator="evd", bias=False)
