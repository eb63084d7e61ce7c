"""KS selection on the GPU against the merge walk (tcoh.cl:34-54): heavily tied
amplitudes at every kind of threshold, and a strip whose window spans more than
2^31 amplitudes (B200 only)."""

import numpy as np
import pytest

import tcoh_b200

pytestmark = pytest.mark.gpu


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


def walk_counts(amp, valid, rows, cols, window, m):
    """SHP counts of the output pixels (-1 at an invalid centre)."""
    count = np.full((rows, cols), -1, np.int32)
    for y in range(rows):
        for x in range(cols):
            cy, cx = y + window[0] // 2, x + window[1] // 2
            if valid[cy, cx]:
                count[y, x] = sum(
                    walk(amp[cy, cx], amp[y + i, x + j], m)
                    for i in range(window[0]) for j in range(window[1]) if valid[y + i, x + j])
    return count


@pytest.mark.parametrize("n", [2, 3, 6, 7, 33])
@pytest.mark.parametrize("levels", [2, 5])
def test_tied_amplitudes(n, levels):
    rng = np.random.default_rng(10 * n + levels)
    rows, cols, window = 7, 6, (7, 5)
    shape = (rows + 6, cols + 4)
    # levels shifted from pixel to pixel, so that decisions of both kinds occur
    amp = rng.integers(0, levels, shape + (n,)) + rng.integers(1, 1 + levels, shape + (1,))
    amp = np.sort(amp.astype(np.float32), axis=2)
    valid = (rng.random(shape) > 0.1).astype(np.uint8)
    slc = np.zeros(shape + (n, 2), np.float32)
    slc[..., 0] = amp
    s = tcoh_b200.make_settings(n, window=window, shp_test="ks", min_shp=1)
    for m in (0, 1, n // 3, n - 1, n, n + 3):
        s.ks_max = m
        with tcoh_b200.Backend(s, cols + 4) as be:
            got = be.run(slc, amp, valid, rows, cols)["count"]
        assert np.array_equal(got, walk_counts(amp, valid, rows, cols, window, m)), m


@pytest.mark.parametrize("m", [-1, -5, -2**31, 2**31 - 1])
def test_thresholds_out_of_range(m):
    """Settings may hold any threshold: below 0 nothing passes, from n on all."""
    n, rows, cols = 6, 9, 8
    rng = np.random.default_rng(1)
    amp = np.sort(rng.uniform(1, 2, (rows, cols, n)).astype(np.float32), axis=2)
    valid = np.ones((rows, cols), np.uint8)
    slc = np.stack([amp, amp], axis=3)
    for window in ((1, 1), (5, 3)):
        s = tcoh_b200.make_settings(n, window=(5, 3), shp_test="ks", min_shp=6)
        s.win_az, s.win_rg, s.ks_max = window + (m,)
        r, c = rows - window[0] + 1, cols - window[1] + 1
        with tcoh_b200.Backend(s, cols) as be:
            got = be.run(slc, amp, valid, r, c)
        assert (got["count"] == (0 if m < 0 else window[0] * window[1])).all()
        if m < 0:
            assert np.isnan(got["coh"]).all()


def test_window_of_more_than_2_31_amplitudes():
    """1001 x 1 candidates, 33,600 columns, 64 dates: the last rows' candidates
    lie 2^31 amplitudes and more beyond the first (52 GB of device memory). With
    windows of one column, columns cut out of the strip give the same result."""
    import torch

    n, cols, window = 64, 33600, (1001, 1)
    if torch.cuda.mem_get_info()[0] < 70 << 30:
        pytest.skip("needs 70 GB of free device memory")
    assert (window[0] - 1) * cols * n > 2**31
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(1)
    amp = torch.empty((window[0], cols, n), device=dev)
    slc = torch.empty((window[0], cols, n, 2), device=dev)
    ramp = torch.linspace(1.0, 2.0, n, device=dev)
    for r in range(window[0]):
        # scales on both sides of what the KS threshold accepts
        scale = 0.6 + 0.8 * torch.rand((cols, 1), generator=g, device=dev)
        noise = 0.4 * torch.randn((cols, n), generator=g, device=dev)
        amp[r] = scale * ramp
        ph = 0.7 * torch.arange(n, device=dev) + noise
        slc[r, ..., 0] = amp[r] * torch.cos(ph)
        slc[r, ..., 1] = amp[r] * torch.sin(ph)
    valid = torch.ones((window[0], cols), dtype=torch.uint8, device=dev)
    s = tcoh_b200.make_settings(n, window=window, shp_test="ks", alpha=0.05, min_shp=64)

    def run(*strip):
        w = strip[0].shape[1]
        coh = torch.empty((1, w), device=dev)
        count = torch.empty((1, w), dtype=torch.int32, device=dev)
        with tcoh_b200.Backend(s, w) as be:
            be.run_device(*strip, 1, w, coh, count)
            torch.cuda.synchronize()
        return coh.cpu().numpy(), count.cpu().numpy()

    coh, count = run(slc, amp, valid)
    some = [0, 1, 16799, 33598, 33599]
    cut = [t[:, some].contiguous() for t in (slc, amp, valid)]
    del slc, amp, valid
    torch.cuda.empty_cache()
    c_coh, c_count = run(*cut)
    assert np.array_equal(count[:, some], c_count)
    assert np.array_equal(coh[:, some], c_coh, equal_nan=True)
    small = cut[1].cpu().numpy()
    ones = np.ones(small.shape[:2], np.uint8)
    want = walk_counts(small, ones, 1, len(some), window, s.ks_max)
    assert (want > 64).all() and (want < 1001).all()
    assert np.array_equal(c_count, want)
