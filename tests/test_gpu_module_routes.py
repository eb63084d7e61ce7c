"""temporal_coherence on strips prepared on the device against strips prepared
on the host (B200 only): every output, selection test and estimator, over several
strips, and every form of stack it takes. The regions are large enough for the
device route (tests/test_strip_routes.py)."""

import numpy as np
import pytest

import tcoh_b200
import tcoh_b200.synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.fixture
def raw_strips(monkeypatch):
    """Rows of the strips that went the device route."""
    rows, run_raw = [], tcoh_b200.Backend.run_raw

    def recorded(self, re, im, elevation, row0, region_rows, nrows, cols, **kw):
        rows.append(nrows)
        return run_raw(self, re, im, elevation, row0, region_rows, nrows, cols, **kw)

    monkeypatch.setattr(tcoh_b200.Backend, "run_raw", recorded)
    return rows


def equal(got, want, names):
    for name in names:
        assert np.array_equal(got[name], want[name], equal_nan=name in ("coh", "pairs", "phases"))


def both_routes(raw_strips, stack, **kw):
    """A phase of zero is removed on the host and changes no sample, so giving
    one takes the host route, over the same strips."""
    got = tcoh_b200.temporal_coherence(stack, **kw)
    assert len(raw_strips) > 1 and sum(raw_strips) == stack.shape[1]
    want = tcoh_b200.temporal_coherence(stack, phase=np.zeros(stack.shape), **kw)
    assert sum(raw_strips) == stack.shape[1] and got.keys() == want.keys()
    assert got["strip_rows"] == want["strip_rows"]
    equal(got, want, set(want) - {"strip_rows"})


@pytest.mark.parametrize("estimator, bias", [("evd", False), ("emi", True)])
@pytest.mark.parametrize("shp_test", ["ks", "ad", "tlog"])
def test_every_output(raw_strips, shp_test, estimator, bias):
    stack = syn.generate(14, 180, 150, nregions=3, seed=8, null_frac=0.02)
    both_routes(raw_strips, stack, window=(7, 5), shp_test=shp_test, min_shp=14,
                estimator=estimator, bias_correction=bias, pairs=True, with_phases=True,
                with_status=True, memory=3)


@pytest.mark.parametrize("estimator", ["evd", "emi"])
def test_long_stacks(raw_strips, estimator):
    stack = syn.generate(35, 130, 100, nregions=3, seed=9, null_frac=0.02)
    both_routes(raw_strips, stack, window=(7, 7), min_shp=20, estimator=estimator, pairs=True,
                pairs_mode="all", with_phases=True, with_status=True, memory=25)


def forms():
    base = syn.generate(9, 130, 110, nregions=2, seed=5, null_frac=0.03)
    odd = base.copy()
    odd[2, 5, 7] = np.inf
    odd[3, 9, 9] = 1e25  # its square overflows
    yield "complex128", base.astype(np.complex128) * (1 + 1e-9)
    yield "strided", np.asfortranarray(base)
    yield "reversed", base[:, ::-1, ::-1]
    yield "real", np.nan_to_num(base.real).astype(np.float64)
    yield "integer", np.nan_to_num(base.real).astype(np.int16)
    yield "infinite", odd


@pytest.mark.parametrize("elevation", [False, True])
@pytest.mark.parametrize("name", [name for name, _ in forms()])
def test_every_form_of_stack(raw_strips, name, elevation):
    stack = dict(forms())[name]
    n, rows, cols = stack.shape
    elev = None
    if elevation:
        elev = np.zeros((rows, cols), np.float32)
        elev[4:9, 3:6] = np.nan
        elev[20, 30] = np.inf
    kw = dict(window=(7, 5), shp_test="ad", min_shp=10)
    got = tcoh_b200.temporal_coherence(stack, elevation=elev, **kw)
    assert raw_strips == [rows]
    slc, amp, valid = tcoh_b200.read_strip(stack.real, stack.imag, -3, rows + 6, 2, elevation=elev)
    with tcoh_b200.Backend(tcoh_b200.make_settings(n, **kw), cols + 4) as be:
        want = be.run(slc, amp, valid, rows, cols)
    equal(got, want, ["coh", "count"])
