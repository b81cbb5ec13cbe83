"""GPU: host calls from many threads that end one after another, and from some
at a time: each call's result and status are its own."""
import threading

import numpy as np
import pytest

from tests._helpers import rel_l2, tol

pytestmark = pytest.mark.gpu


def test_threads_that_come_and_go():
    import jtransforms_gb300 as J
    errors = []

    def work(seed):
        try:
            x = np.random.default_rng(seed).standard_normal(2 * 512)
            a = x.copy()
            J.DoubleFFT_1D(512).complexForward(a)
            if rel_l2(a.view(np.complex128), np.fft.fft(x.view(np.complex128))) > tol(512, np.float64):
                errors.append(seed)
        except Exception as e:  # reported below
            errors.append(repr(e))

    for seed in range(0, 60, 3):
        th = [threading.Thread(target=work, args=(seed + i,)) for i in range(3)]
        for t in th:
            t.start()
        for t in th:
            t.join()
    assert not errors, errors
