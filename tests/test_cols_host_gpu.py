"""Host column calls: one plan shared by several threads."""
import threading

import numpy as np
import pytest

from conftest import crandn
from openvsip_b200 import Fftm, col

pytestmark = pytest.mark.gpu


def test_threads_share_a_column_plan():
    # calls of different widths, so that the plan's device block also grows while others wait
    rows, widths, turns = 756, (40, 300, 900, 64), 12
    rng = np.random.default_rng(1)
    xs = [crandn(rng, (rows, w)) for w in widths]
    want = [Fftm(rows, w, axis=col)(x) for w, x in zip(widths, xs)]
    f = Fftm(rows, max(widths), axis=col)
    wrong, start = [], threading.Barrier(len(xs))

    def run(i):
        start.wait()
        for _ in range(turns):
            if not np.array_equal(f(xs[i]), want[i]):
                wrong.append(i)

    ts = [threading.Thread(target=run, args=(i,)) for i in range(len(xs))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not wrong
