"""Two contexts on two host threads (B200 only): calls of any size and settings
run side by side, as the library's calls release the interpreter's lock."""

import threading

import numpy as np
import pytest

import tcoh_b200
import tcoh_b200.synthetic as syn

pytestmark = pytest.mark.gpu


class Job:
    """A context and a strip, with the outputs of a call made alone."""

    def __init__(self, n, rows, cols, estimator, shp_test="ks"):
        window = (11, 7)
        stack = syn.generate(n, rows, cols, seed=n, nregions=3)
        self.strip = tcoh_b200.read_strip(stack.real, stack.imag, -5, rows + 10, 3)
        self.size = rows, cols
        s = tcoh_b200.make_settings(n, window=window, shp_test=shp_test, min_shp=20,
                                    estimator=estimator)
        self.backend = tcoh_b200.Backend(s, cols + 6, chunk_pixels=2048)
        self.alone = self.call()

    def call(self):
        return self.backend.run(*self.strip, *self.size)


def side_by_side(large, small, calls=150):
    """`calls` calls of the large job on one thread while another repeats the
    small one; every output equals that of the call made alone."""
    errors, done = [], threading.Event()

    def work(job, go_on):
        k = 0
        try:
            while go_on(k):
                r = job.call()
                assert np.array_equal(r["coh"], job.alone["coh"], equal_nan=True)
                assert np.array_equal(r["count"], job.alone["count"])
                k += 1
        except Exception as e:
            errors.append(e)
        finally:
            if job is large:
                done.set()

    threads = [threading.Thread(target=work, args=(large, lambda k: k < calls and not errors)),
               threading.Thread(target=work, args=(small, lambda k: not done.is_set()))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    large.backend.close()
    small.backend.close()
    assert not errors, errors[0]


@pytest.mark.parametrize("n, estimator", [(10, "evd"), (20, "evd"), (20, "emi"), (40, "evd")])
def test_same_settings_different_sizes(n, estimator):
    side_by_side(Job(n, 256, 128, estimator), Job(n, 9, 7, estimator))


@pytest.mark.parametrize("n, other", [(20, 31), (34, 64)])
def test_different_settings(n, other):
    side_by_side(Job(n, 128, 128, "emi" if n > 32 else "evd", "ad"),
                 Job(other, 9, 7, "emi" if n > 32 else "evd", "ad"), calls=100)
