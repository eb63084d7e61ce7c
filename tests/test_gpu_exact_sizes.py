"""The exact tier at the edges of its forms (B200 only): numbers of dates around
the pivot groups and register rows of its inverse. Every window that lies in the
region holds the same samples, for which the bias correction's threshold is met
by one pair of dates to within 5e-6: all these pixels go to the tier, which the
status says (STATUS_FP64)."""

import numpy as np
import pytest

import oracle
import tcoh_b200
from conftest import TOLERANCE

pytestmark = pytest.mark.gpu

WINDOW = (15, 9)


def stack_of(n, rows, cols):
    """Unit samples, repeated with the window's period. The phase differences of
    dates 0 and 1 are +a and -a for half of the L = 135 samples each and 0 for
    one: their coherence (134 cos a + 1) / 135 has the square (1 + 5e-6) / 135."""
    rng = np.random.default_rng(200 + n)
    looks = WINDOW[0] * WINDOW[1]
    a = np.arccos((looks * np.sqrt((1 + 5e-6) / looks) - 1) / (looks - 1))
    d = np.concatenate([np.full(looks // 2, a), np.full(looks // 2, -a), [0.0]])
    rng.shuffle(d)
    # the others: coherences from 0.1 to 0.97 with one another and with dates 0, 1
    ph = rng.normal(0.0, 1.0, (n, looks)) * rng.uniform(0.2, 1.2, (n, 1))
    ph[0] = rng.normal(0.0, 0.3, looks)
    ph[1] = ph[0] + d
    ph += 0.8 * np.arange(n)[:, None]
    reps = (1, -(-rows // WINDOW[0]), -(-cols // WINDOW[1]))
    tile = np.exp(1j * ph).reshape((n,) + WINDOW)
    return np.tile(tile, reps)[:, :rows, :cols].astype(np.complex64)


def inside(rows, cols):
    ha, hr = WINDOW[0] // 2, WINDOW[1] // 2
    return np.s_[ha:rows - ha, hr:cols - hr]


@pytest.mark.parametrize("estimator", ["evd", "emi"])
@pytest.mark.parametrize("n", [2, 3, 4, 5, 6, 7, 8, 9, 15, 16, 17, 29, 30, 31, 32, 33, 34, 35, 62,
                               63, 64])
def test_every_form(n, estimator):
    rows, cols = 20, 14
    stack = stack_of(n, rows, cols)
    slc, amp, valid = tcoh_b200.read_strip(stack.real, stack.imag, -7, rows + 14, 4)
    # the same amplitudes everywhere: every pixel is an SHP
    amp[:] = (valid != 0)[..., None] * np.arange(1, n + 1, dtype=np.float32)
    kw = dict(window=WINDOW, shp_test="ks", alpha=0.01, min_shp=100, estimator=estimator,
              bias=True)
    s = tcoh_b200.make_settings(n, pairs=True, pairs_all=True, **kw)
    with tcoh_b200.Backend(s, cols + 8) as be:
        r = be.run(slc, amp, valid, rows, cols, status=True)
    o = oracle.run_oracle(slc, amp, valid, rows, cols, shp_fp32=True, npairs=s.npairs,
                          pairs_all=True, **kw)
    assert np.array_equal(r["count"], o["count"])
    assert (r["count"][inside(rows, cols)] == 135).all()
    assert np.array_equal(np.isnan(r["coh"]), np.isnan(o["coh"]))
    m = ~np.isnan(o["coh"])
    assert m[inside(rows, cols)].all()
    exact = (r["status"] & tcoh_b200.STATUS_FP64) != 0
    assert exact[inside(rows, cols)].all()
    if estimator == "emi" and n > 32:
        assert exact[m].all()
    assert np.abs(r["coh"][exact] - o["coh"][exact]).max() <= TOLERANCE
    assert np.abs(r["pairs"][:, exact] - o["pairs"][:, exact]).max() <= TOLERANCE
