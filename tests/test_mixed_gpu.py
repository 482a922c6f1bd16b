"""GPU parity of the mixed-radix kernel (lengths whose prime factors are at
most 13, up to 28672 samples) against the FP64 oracle: relative L2 <= 2e-6, the
bar of the other row kernels.  The sizes are where its plan changes: one to six
stages, every radix, several rows per CTA with a partial last one, the longest
rows (512-thread CTAs)."""
import numpy as np
import pytest

from conftest import crandn
from openvsip_b200 import Fastconv, Fftm, fft_fwd, fft_inv

pytestmark = pytest.mark.gpu
RTOL = 2e-6

#        one stage      two               every prime, three and more          six stages  largest
SHAPES = [(7, 3), (33, 15), (5, 26), (65, 143), (9, 1001), (3, 1144), (147, 756), (2, 9216), (2, 15625), (3, 28672)]


@pytest.mark.parametrize("rows,n", SHAPES)
@pytest.mark.parametrize("direction", [fft_fwd, fft_inv])
def test_rows_strided_and_in_place(oracle, rows, n, direction):
    import torch
    rng = np.random.default_rng(n)
    exponent, scale = (-1, 0.5) if direction == fft_fwd else (+1, 1.0 / n)
    x = crandn(rng, (rows, n + 3))[:, :n]
    want = oracle.fft_rows(np.ascontiguousarray(x), exponent, scale)
    f = Fftm(rows, n, direction, scale)
    buf = torch.zeros(rows, n + 5, dtype=torch.complex64, device="cuda")  # guard columns
    src = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    f(src, buf[:, 2:n + 2])
    assert oracle.rel_l2(buf[:, 2:n + 2].cpu().numpy(), want) <= RTOL
    assert not buf[:, :2].any() and not buf[:, n + 2:].any()
    out = buf[:, 2:n + 2].clone()
    f.in_place(src)
    assert torch.equal(src, out)
    if rows > 2:  # fewer rows than planned: another split over CTAs, the same numbers
        src = torch.from_numpy(np.ascontiguousarray(x[:2])).cuda()
        assert torch.equal(f(src), out[:2])


@pytest.mark.parametrize("rows,n", SHAPES)
def test_fastconv_vector_and_matrix(oracle, rows, n):
    import torch
    rng = np.random.default_rng(1000 + n)
    x = crandn(rng, (rows, n))
    for w in (crandn(rng, (n,)), crandn(rng, (rows, n))):
        y = Fastconv(w, rows)(torch.from_numpy(x).cuda())
        assert oracle.rel_l2(y.cpu().numpy(), oracle.fastconv(x, w)) <= RTOL
