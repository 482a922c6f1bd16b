"""Few long rows of lengths whose last mixed-radix stage has bank conflicts (multiples of 256,
28000): plans for up to 33 rows, and for more, on both sides of the change of algorithm."""
import numpy as np
import pytest

from conftest import crandn
from openvsip_b200 import Fftm, FftmReal, col, fft_fwd, fft_inv

pytestmark = pytest.mark.gpu
RTOL = 2e-6


@pytest.mark.parametrize("n", [24576, 25088, 28000, 28672])
@pytest.mark.parametrize("rows", [1, 33, 34])
def test_vs_fp64(oracle, n, rows):
    x = crandn(np.random.default_rng(n + rows), (rows, n))
    want = np.fft.fft(x.astype(np.complex128))
    assert oracle.rel_l2(Fftm(rows, n)(x), want) <= RTOL
    assert oracle.rel_l2(Fftm(rows, n, fft_inv, 1.0 / n)(want.astype(np.complex64)), x) <= RTOL
    assert oracle.rel_l2(Fftm(n, rows, axis=col)(np.ascontiguousarray(x.T)), want.T) <= RTOL
    r = np.ascontiguousarray(x.view(np.float32))  # rows of 2n real samples
    half = np.fft.rfft(r.astype(np.float64))
    assert oracle.rel_l2(FftmReal(rows, 2 * n, fft_fwd)(r), half) <= RTOL
    assert oracle.rel_l2(FftmReal(rows, 2 * n, fft_inv, 0.5 / n)(half.astype(np.complex64)), r) <= RTOL


@pytest.mark.parametrize("n", [26880, 28000, 28672])
def test_few_planned_rows_are_spread_over_the_gpu(n):
    import torch
    x = torch.ones(8, n, dtype=torch.complex64, device="cuda")
    y = torch.empty_like(x)

    def us(plan):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        best = float("inf")
        for _ in range(7):
            e[0].record()
            for _ in range(30):
                plan(x, y)
            e[1].record()
            e[1].synchronize()
            best = min(best, e[0].elapsed_time(e[1]) * 1e3 / 30)
        return best

    few, many = us(Fftm(8, n)), us(Fftm(64, n))
    assert few <= 0.85 * many, (few, many)
