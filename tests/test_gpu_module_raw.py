"""temporal_coherence prepares its strips on the device where it can: the result
equals that of strips prepared on the host, for every form of stack it takes
(B200 only)."""

import numpy as np
import pytest

import tcoh_b200
import tcoh_b200.synthetic as syn

pytestmark = pytest.mark.gpu


def by_host_strips(stack, window, elevation=None, **kw):
    """The region as one strip through read_strip and Backend.run."""
    n, rows, cols = stack.shape
    ha, hr = window[0] // 2, window[1] // 2
    slc, amp, valid = tcoh_b200.read_strip(stack.real, stack.imag, -ha, rows + 2 * ha, hr,
                                           elevation=elevation)
    s = tcoh_b200.make_settings(n, window=window, **kw)
    with tcoh_b200.Backend(s, cols + 2 * hr) as be:
        return be.run(slc, amp, valid, rows, cols)


def stacks():
    base = syn.generate(9, 37, 21, nregions=2, seed=5, null_frac=0.03)
    odd = base.copy()
    odd[2, 5, 7] = np.inf
    odd[3, 9, 9] = 1e25  # its square overflows
    yield "complex64", base
    yield "complex128", base.astype(np.complex128) * (1 + 1e-9)
    yield "strided", np.asfortranarray(base)
    yield "reversed", base[:, ::-1, ::-1]
    yield "real", np.nan_to_num(base.real).astype(np.float64)
    yield "infinite", odd


@pytest.mark.parametrize("memory", [300, 1])
@pytest.mark.parametrize("name", ["complex64", "complex128", "strided", "reversed", "real",
                                  "infinite"])
def test_equals_host_strips(name, memory):
    stack = dict(stacks())[name]
    window, kw = (7, 5), dict(shp_test="ad", min_shp=10)
    want = by_host_strips(stack, window, **kw)
    got = tcoh_b200.temporal_coherence(stack, window=window, memory=memory, **kw)
    assert np.array_equal(got["count"], want["count"])
    assert np.array_equal(got["coh"], want["coh"], equal_nan=True)


def test_elevation_nulls_and_a_callers_geometry():
    stack = dict(stacks())["complex64"]
    elev = np.zeros(stack.shape[1:])
    elev[4:9, 3:6] = np.nan
    window = (7, 5)
    want = by_host_strips(stack, window, elevation=elev, min_shp=10)
    got = tcoh_b200.temporal_coherence(stack, window=window, elevation=elev, min_shp=10)
    assert np.array_equal(got["count"], want["count"])
    assert np.array_equal(got["coh"], want["coh"], equal_nan=True)
    # a context with a geometry attached keeps out of the device preparation
    import tcoh_b200.scene as scene

    geo, orbits = scene.acquisition(9, *stack.shape[1:], seed=3)
    g = tcoh_b200.make_geometry(h0=0.0, **geo)
    s = tcoh_b200.make_settings(9, window=window, min_shp=10)
    with tcoh_b200.Backend(s, stack.shape[2] + 4) as be:
        be.set_geometry(g, tcoh_b200.geometry_grid(g, orbits))
        got = tcoh_b200.temporal_coherence(stack, window=window, elevation=elev, min_shp=10,
                                           backend=be)
    assert np.array_equal(got["coh"], want["coh"], equal_nan=True)
