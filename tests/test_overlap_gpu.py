"""Back-to-back calls, whose launches overlap, see each other's results: chains
of in-place calls without a wait between them equal the same chains with one,
bit for bit, on data small enough to stay in the SMs' caches."""
import numpy as np
import pytest

from conftest import crandn
from openvsip_b200 import Fastconv, Fft2d, Fftm, FftmReal, col, fft_fwd, fft_inv, vmmul

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,n", [(148, 64), (592, 512), (148, 2048), (37, 8192), (20, 32768), (148, 480), (600, 1144)])
def test_chains_of_in_place_calls(rows, n):
    import torch
    rng = np.random.default_rng(n)
    rep = crandn(rng, (n,))
    rep /= np.abs(rep)
    f, b = Fftm(rows, n, fft_fwd, 1.0 / np.sqrt(n)), Fftm(rows, n, fft_inv, 1.0 / np.sqrt(n))
    c, m = Fastconv(rep, rows), Fftm(rows, n, fft_fwd, 1.0 / np.sqrt(rows), axis=col)
    s = Fft2d(rows, n, fft_fwd, 1.0 / np.sqrt(rows * n))
    r, q = FftmReal(rows, n, fft_fwd, 1.0 / np.sqrt(n)), FftmReal(rows, n, fft_inv, 1.0 / np.sqrt(n))
    v = torch.from_numpy(rep).cuda()
    x0 = torch.from_numpy(crandn(rng, (rows, n))).cuda()
    real0 = torch.randn(rows, n, device="cuda")
    half = torch.empty(rows, n // 2 + 1, dtype=torch.complex64, device="cuda")

    def chain(wait):
        x, real = x0.clone(), real0.clone()
        for _ in range(12):
            for step in (lambda: f.in_place(x), lambda: vmmul(v, x, x), lambda: b.in_place(x), lambda: c.in_place(x),
                         lambda: m.in_place(x), lambda: s(x, x), lambda: r(real, half), lambda: q(half, real)):
                step()
                if wait:
                    torch.cuda.synchronize()
        torch.cuda.synchronize()
        return x, real

    want = chain(True)
    for _ in range(5):
        got = chain(False)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert torch.isfinite(torch.view_as_real(want[0])).all()
