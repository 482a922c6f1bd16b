"""Calls of few rows run kernels of their own (more registers, wider clusters);
their rows come out exactly as in a call that fills the GPU, at the row counts
around the change from one to the other."""
import numpy as np
import pytest

from conftest import crandn
from openvsip_b200 import Fastconv, Fftm, FftmReal, fft_fwd, fft_inv

pytestmark = pytest.mark.gpu
RTOL = 2e-6
# a length of every CTA shape, one of Bluestein (n = 67 * 16: work rows of 4096)
LENGTHS = [32, 128, 512, 2048, 4096, 8192, 16384, 32768, 65536, 1072]


@pytest.mark.parametrize("n", LENGTHS)
def test_rows_do_not_depend_on_their_number(oracle, n):
    import torch
    many = min(4096, max(600, (1 << 21) // n))
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.view_as_complex(torch.randn(many, n, 2, generator=g, device="cuda"))
    rep = crandn(np.random.default_rng(n), (n,))
    plans = [Fastconv(rep, many), Fftm(many, n, fft_fwd), Fftm(many, n, fft_inv, 1.0 / n)]
    refs = [lambda v: oracle.fastconv(v, rep), lambda v: oracle.fft_rows(v, -1),
            lambda v: oracle.fft_rows(v, +1, 1.0 / n)]
    for p, ref in zip(plans, refs):
        full = p(x)
        for rows in (1, 2, 3, 15, 16, 17, 18, 19, 36, 37, 74, 75, 148, 149, 296, 297, 592):
            if rows <= many:
                assert torch.equal(p(x[:rows]), full[:rows]), (n, rows)
        assert oracle.rel_l2(full[:2].cpu().numpy(), ref(x[:2].cpu().numpy())) <= RTOL
    if n <= 32768 and n % 2 == 0:
        real = torch.view_as_real(x).reshape(many, 2 * n)
        f, b = FftmReal(many, 2 * n, fft_fwd), FftmReal(many, 2 * n, fft_inv, 1.0 / n)
        spec = f(real)
        back = b(spec)
        for rows in (1, 18, 37, 75, 149, 297):
            assert torch.equal(f(real[:rows], torch.empty_like(spec[:rows])), spec[:rows]), (n, rows)
            assert torch.equal(b(spec[:rows], torch.empty_like(back[:rows])), back[:rows]), (n, rows)


@pytest.mark.parametrize("n,many", [(512, 5000), (4096, 1300), (16384, 400), (32768, 80)])
def test_matrix_of_coefficients_equals_its_rows(n, many):
    # more rows than are resident at once take the kernel that fetches replica rows ahead
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    x, w = (torch.view_as_complex(torch.randn(many, n, 2, generator=g, device="cuda")) for _ in range(2))
    full = Fastconv(w, many)(x)
    for lo, hi in ((0, 3), (many // 2, many // 2 + 100), (many - 2, many)):
        hi = min(hi, many)
        part = Fastconv(w[lo:hi], hi - lo)(x[lo:hi])
        assert torch.equal(part, full[lo:hi])
    assert torch.equal(Fastconv(w[5], 2)(x[5:7])[:1], full[5:6])
