"""The link kernels with full CTAs that take several turns (B200 only): strips
of more pixels than all SMs hold at once, so that a CTA has its most warps, its
barriers and named barriers span them, and every workspace is taken by a second
pixel; against the double-precision oracle."""

import numpy as np
import pytest

import oracle
import tcoh_b200
import tcoh_b200.synthetic as syn
from conftest import TOLERANCE

pytestmark = pytest.mark.gpu


def compare(n, window, twins=False, **kw):
    """48 x 200 pixels: 75 tiles of 128, 4,800 pixel pairs, where 148 SMs hold
    3,552 at most (48 x 80 above 32 dates: 30 tiles, 3,840 pixels, where they
    hold 888). twins: in half of the columns two dates are equal."""
    rows, cols = 48, 200 if n <= 32 else 80
    ha, hr = window[0] // 2, window[1] // 2
    stack = syn.generate(n, rows, cols, nregions=6, g0_max=0.9, seed=300 + n, null_frac=0.01)
    if twins:
        stack[1, :, cols // 2:] = stack[0, :, cols // 2:]
    slc, amp, valid = tcoh_b200.read_strip(stack.real, stack.imag, -ha, rows + 2 * ha, hr)
    s = tcoh_b200.make_settings(n, window=window, **kw)
    with tcoh_b200.Backend(s, cols + 2 * hr) as be:
        r = be.run(slc, amp, valid, rows, cols, status=True)
    o = oracle.run_oracle(slc, amp, valid, rows, cols, shp_fp32=True, window=window, **kw)
    assert np.array_equal(r["count"], o["count"])
    assert np.array_equal(np.isnan(r["coh"]), np.isnan(o["coh"]))
    m = ~np.isnan(o["coh"])
    assert m.sum() > rows * cols // 4
    assert np.abs(r["coh"][m] - o["coh"][m]).max() <= TOLERANCE
    return r, m


@pytest.mark.parametrize("n, estimator, bias", [
    (10, "evd", False), (10, "emi", True), (12, "emi", True), (16, "emi", False), (24, "evd", True),
    (24, "emi", False), (40, "evd", True), (64, "evd", False)])
def test_several_turns(n, estimator, bias):
    compare(n, (11, 7), shp_test="ks", alpha=0.05, min_shp=20, estimator=estimator, bias=bias)


@pytest.mark.parametrize("n", [16, 24])
def test_fallback_inverse_in_some_halves(n):
    """Equal dates make |T| singular: these pixels take the pseudo-inverse, the
    two halves of a warp in turn or one of them alone."""
    r, m = compare(n, (11, 7), twins=True, shp_test="ks", alpha=0.05, min_shp=20,
                   estimator="emi", bias=False)
    pinv = (r["status"] & tcoh_b200.STATUS_EMI_PINV) != 0
    assert (pinv[:, 110:] == m[:, 110:]).mean() > 0.9
    assert not pinv[:, :90].any()
