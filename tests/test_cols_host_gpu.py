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


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("n,cols", [(2, 1), (16, 5), (1960, 20), (2000, 3), (2000, 4), (2000, 32), (2000, 33), (2048, 1), (14336, 9),
                                    (756, 2774), (756, 2775), (756, 9000), (14000, 400)])
def test_blocks_and_strides_equal_the_device(n, cols, pinned):
    # one block, several (16 MB each) and their edges; packed, strided and in place
    import torch

    def host(width):
        t = torch.zeros(n, width, 2)
        return torch.view_as_complex(t.pin_memory() if pinned else t).numpy()

    rng = np.random.default_rng(n + cols)
    x = crandn(rng, (n, cols))
    f = Fftm(n, cols, axis=col)
    want = f(torch.from_numpy(x).cuda()).cpu().numpy()
    for wi, wo in ((cols, cols), (cols + 3, cols), (cols, cols + 2)):
        a, b = host(wi), host(wo)
        a[:, :cols] = x
        f(a[:, :cols], b[:, :cols])
        assert np.array_equal(b[:, :cols], want) and not b[:, cols:].any()
        assert np.array_equal(a[:, :cols], x) and not a[:, cols:].any()
    a = host(cols + 1)
    a[:, 1:] = x
    f.in_place(a[:, 1:])
    assert np.array_equal(a[:, 1:], want) and not a[:, 0].any()
    if cols > 2:
        few = f(x[:, :cols - 2])  # fewer columns than planned
        assert np.array_equal(few, want[:, :cols - 2])


@pytest.mark.parametrize("n,cols", [(2048, 20), (14000, 20)])
def test_narrow_host_columns_cost_no_more_than_transposing(n, cols):
    import time
    x = crandn(np.random.default_rng(2), (n, cols))
    y = np.empty_like(x)
    f, rows = Fftm(n, cols, axis=col), Fftm(cols, n)

    def transposing():
        y[...] = rows(np.ascontiguousarray(x.T)).T

    def median(call):
        times = []
        for _ in range(25):
            t = time.perf_counter()
            call()
            times.append(time.perf_counter() - t)
        return sorted(times)[12]

    direct, ref = median(lambda: f(x, y)), median(transposing)
    assert direct <= 1.2 * ref, (direct, ref)
