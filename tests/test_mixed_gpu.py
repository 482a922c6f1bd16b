"""GPU parity of the mixed-radix kernel (lengths whose prime factors are at
most 13, up to 28672 samples) against the FP64 oracle: relative L2 <= 2e-6, the
bar of the other row kernels.  The sizes are where its plan changes: one to six
stages, every radix, several rows per CTA with a partial last one, the longest
rows (512-thread CTAs); columns likewise, and the forms of a matrix that go
through rows instead."""
import numpy as np
import pytest

from conftest import crandn
from openvsip_b200 import FcbError, Fastconv, Fftm, col, fft_fwd, fft_inv

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


#       one column, one stage, partial last CTA, ragged, two columns per CTA, the longest, longer: through rows
COLUMNS = [(13, 1), (2, 70), (756, 45), (1000, 67), (4096, 9), (4096, 130), (8192, 5), (14336, 3), (16384, 3), (67, 5)]


@pytest.mark.parametrize("n,m", COLUMNS)
@pytest.mark.parametrize("direction", [fft_fwd, fft_inv])
def test_columns_host_device_views_and_in_place(n, m, direction):
    import torch
    rng = np.random.default_rng(n + m)
    big = crandn(rng, (n, m + 6))
    x = big[:, 1:m + 1]
    scale = 0.25 if direction == fft_fwd else 1.0 / n
    x64 = x.astype(np.complex128)
    want = scale * (np.fft.fft(x64, axis=0) if direction == fft_fwd else n * np.fft.ifft(x64, axis=0))
    rel = lambda y: np.linalg.norm(y - want) / np.linalg.norm(want)  # noqa: E731
    f = Fftm(n, m, direction, scale, axis=col)
    host = f(x)
    assert rel(host) <= RTOL
    dbig = torch.from_numpy(big.copy()).cuda()
    dx = dbig[:, 1:m + 1]
    out = torch.zeros(n, m + 4, dtype=torch.complex64, device="cuda")
    f(dx, out[:, 3:m + 3])
    assert np.array_equal(out[:, 3:m + 3].cpu().numpy(), host)
    assert not out[:, :3].any() and not out[:, m + 3:].any()
    # inputs that no column kernel takes as they are: a lazy conjugate, a transposed
    # view, an output that overlaps the input
    assert rel(f(torch.from_numpy(np.ascontiguousarray(x).conj()).cuda().conj()).cpu().numpy()) <= RTOL
    assert rel(f(torch.from_numpy(np.ascontiguousarray(x.T)).cuda().t()).cpu().numpy()) <= RTOL
    over = dbig.clone()
    assert rel(f(over[:, 1:m + 1], over[:, 2:m + 2]).cpu().numpy()) <= RTOL
    h = np.ascontiguousarray(x)
    assert np.array_equal(f.in_place(h), host)
    f.in_place(dx)
    assert np.array_equal(dx.cpu().numpy(), host)
    assert torch.equal(dbig[:, m + 1:].cpu(), torch.from_numpy(big[:, m + 1:].copy()))  # neighbours untouched
    if m > 2:  # fewer columns than planned
        assert np.array_equal(f(np.ascontiguousarray(x[:, :2])), host[:, :2])
    with pytest.raises(FcbError):
        f(crandn(rng, (n, m + 1)))
