"""A model's parameters read by several threads while another sets them: a read is one of the sets
that were written, whole, and what a set wrote is what the model then holds."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from protlocus_b200 import prefilter as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("readers", [1, 4])
def test_params_from_threads(readers):
    m = P.PrefilterModel(seed=3)
    rng = np.random.default_rng(readers)
    sets = [rng.standard_normal(m.size()).astype(np.float32) for _ in range(3)]
    m.set_params(sets[0])
    stop, bad = threading.Event(), []

    def reader():
        while not stop.is_set():
            p = m.params()
            if not any(np.array_equal(p, s) for s in sets):
                bad.append(p)

    threads = [threading.Thread(target=reader) for _ in range(readers)]
    for t in threads:
        t.start()
    try:
        for k in range(60):
            m.set_params(sets[k % 3])
            assert np.array_equal(m.params(), sets[k % 3])
    finally:
        stop.set()
        for t in threads:
            t.join()
    assert not bad
