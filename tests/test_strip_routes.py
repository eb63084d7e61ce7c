"""Where temporal_coherence prepares its strips: on the device from the raw rows,
except small strips, a host phase, rows that would take too much of the device's
memory and a context with a geometry of its own (a recording stand-in for the
context; no GPU)."""

import numpy as np
import pytest

import tcoh_b200


class Context:
    def __init__(self, max_alloc=60 << 30, grid=None):
        self.max_alloc = max_alloc
        self.routes = []
        if grid is not None:
            self._grid = grid

    def _outputs(self, rows, cols):
        return {"coh": np.zeros((rows, cols), np.float32),
                "count": np.zeros((rows, cols), np.int32)}

    def run(self, slc, amp, valid, rows, cols, phases, status):
        self.routes.append("host")
        return self._outputs(rows, cols)

    def run_raw(self, re, im, elevation, row0, region_rows, rows, cols, phases, status):
        self.routes.append("device")
        return self._outputs(rows, cols)


def routes(n, rows, cols, backend=None, **kw):
    be = backend or Context()
    stack = np.ones((n, rows, cols), np.complex64)
    tcoh_b200.temporal_coherence(stack, window=(11, 7), min_shp=10, backend=be, **kw)
    return set(be.routes)


@pytest.mark.parametrize("n, rows, cols, route", [
    (2, 20, 20, "host"), (2, 114, 100, "host"), (2, 115, 100, "device"), (10, 80, 80, "host"),
    (10, 120, 120, "device"), (20, 59, 100, "host"), (20, 60, 100, "device"),
    (60, 54, 100, "host"), (60, 55, 100, "device"), (60, 40, 40, "host"),
    (30, 200, 300, "device")])
def test_by_size(n, rows, cols, route):
    assert routes(n, rows, cols) == {route}


def test_by_what_the_call_asks_for():
    assert routes(10, 120, 120, phase=np.zeros((10, 120, 120))) == {"host"}
    assert routes(10, 120, 120, Context(grid=np.zeros(1))) == {"host"}
    assert routes(10, 120, 120, Context(max_alloc=8 * 8 * 10 * 130 * 120 - 8)) == {"host"}
    assert routes(10, 120, 120, Context(max_alloc=8 * 8 * 10 * 130 * 120)) == {"device"}
    assert routes(10, 120, 120, elevation=np.zeros((120, 120))) == {"device"}
