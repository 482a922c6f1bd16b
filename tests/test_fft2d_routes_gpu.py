"""2-D transforms by each of their routes against FP64: tall matrices of few columns
(rows and transposes, or the column kernel), the two transposing passes, columns that
have no kernel of their own."""
import numpy as np
import pytest

from conftest import crandn
from openvsip_b200 import Fft2d, Fftm, fft_fwd, fft_inv

pytestmark = pytest.mark.gpu
RTOL = 2e-6


def _check(rows, cols):
    """Forward and inverse, strided and in place, on the device and on the host."""
    import torch
    rng = np.random.default_rng(rows + 3 * cols)
    x = crandn(rng, (rows, cols))
    dx = torch.from_numpy(x).cuda()
    f, g = Fft2d(rows, cols, fft_fwd, 0.5), Fft2d(rows, cols, fft_inv, 2.0 / (rows * cols))
    want = 0.5 * torch.fft.fft2(dx.to(torch.complex128))
    out = torch.zeros(rows, cols + 3, dtype=torch.complex64, device="cuda")
    got = f(dx, out[:, 1:cols + 1])
    assert ((got - want).norm() / want.norm()).item() <= RTOL
    assert not out[:, 0].any() and not out[:, cols + 1:].any()
    back = g(got)  # strided in
    assert ((back - dx).norm() / dx.norm()).item() <= RTOL
    y = dx.clone()
    f(y, y)
    assert torch.equal(y, got)
    if rows * cols <= 1 << 22:
        assert np.array_equal(f(x), y.cpu().numpy())


@pytest.mark.parametrize("rows,cols", [(8192, 1), (8192, 7), (8192, 8), (8192, 16), (8192, 32), (8192, 100), (8192, 128),
                                       (8192, 129), (4096, 32), (4096, 1), (2048, 16), (16384, 32)])
def test_tall_matrices(rows, cols):
    _check(rows, cols)


# two transposing passes: rows of 16384 (one a CTA), columns whose rest is too long for the
# column kernel, and the sizes below those of the row pass that takes the columns along
@pytest.mark.parametrize("rows,cols", [(128, 16384), (4096, 16384), (16384, 8192), (2048, 256), (2048, 64)])
def test_transposing_passes(rows, cols):
    _check(rows, cols)


# columns of a length with a large prime factor, or too long: a row pass, a transpose,
# a row pass and a transpose back; their transposed sizes take the column kernel
@pytest.mark.parametrize("rows,cols", [(67, 100), (100, 67), (1007, 64), (1, 777), (16384, 100), (100, 16384), (17, 17)])
def test_columns_without_a_kernel(rows, cols):
    _check(rows, cols)


def test_few_tall_columns_cost_no_more_than_rows_and_transposes():
    import torch
    rows, cols = 8192, 32
    x = torch.ones(rows, cols, dtype=torch.complex64, device="cuda")
    y, z = torch.empty_like(x), torch.empty(cols, rows, dtype=torch.complex64, device="cuda")
    f, a, b = Fft2d(rows, cols), Fftm(rows, cols), Fftm(cols, rows)

    def by_hand():
        a(x, y)
        z.copy_(y.t())
        b(z, z)
        y.copy_(z.t())

    def us(call):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        best = float("inf")
        for _ in range(7):
            e[0].record()
            for _ in range(30):
                call()
            e[1].record()
            e[1].synchronize()
            best = min(best, e[0].elapsed_time(e[1]) * 1e3 / 30)
        return best

    one, hand = us(lambda: f(x, y)), us(by_hand)
    assert one <= 1.15 * hand, (one, hand)  # 33.8 against 26.8 us by the column kernel
