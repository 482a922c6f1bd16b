"""Real rows of power-of-two length on device data, where the split and the
merge of the half spectrum are part of the row kernel: every alignment of the
output rows (its 16-byte stores start at bin 0 or at bin 1), unaligned real
rows, a padded in-place forward transform, infinities in bins that do not count.
Against FP64 numpy, relative L2 <= 2e-6 as for the other real transforms."""
import numpy as np
import pytest

from openvsip_b200 import FftmReal, fft_fwd, fft_inv

pytestmark = pytest.mark.gpu
RTOL = 2e-6
# one-stage rows, several rows per CTA, every CTA size, the wide variant (32768), clusters
LENGTHS = [2, 4, 32, 64, 512, 4096, 16384, 32768, 65536, 131072]


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("pad,shift", [(0, 0), (1, 0), (1, 1), (4, 3)])
def test_forward_output_alignments(n, pad, shift):
    import torch
    rows, bins = 5, n // 2 + 1
    x = np.random.default_rng(n).standard_normal((rows, n)).astype(np.float32)
    want = 0.5 * np.fft.rfft(x.astype(np.float64), axis=1)
    out = torch.zeros(rows, bins + pad + 4, dtype=torch.complex64, device="cuda")
    view = out[:, shift:shift + bins]
    f = FftmReal(rows, n, fft_fwd, 0.5)
    f(torch.from_numpy(x).cuda(), view)
    got = view.cpu().numpy()
    assert _rel(got, want) <= RTOL
    assert not got[:, 0].imag.any() and not got[:, -1].imag.any()
    assert not out[:, :shift].any() and not out[:, shift + bins:].any()
    # real rows that start on odd floats go through a copy
    big = torch.zeros(rows, n + 3, device="cuda")
    big[:, 1:n + 1] = torch.from_numpy(x).cuda()
    assert np.array_equal(f(big[:, 1:n + 1]).cpu().numpy(), got)
    # in place: rows of bins complex values, the real rows at their start
    work = torch.zeros(rows, bins, 2, device="cuda")
    real = work.reshape(rows, 2 * bins)[:, :n]
    real.copy_(torch.from_numpy(x))
    f(real, torch.view_as_complex(work))
    assert np.array_equal(torch.view_as_complex(work).cpu().numpy(), got)


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("pad,shift", [(0, 0), (3, 1)])
def test_inverse_output_alignments(n, pad, shift):
    import torch
    rows, bins = 5, n // 2 + 1
    rng = np.random.default_rng(n)
    h = (rng.standard_normal((rows, bins)) + 1j * rng.standard_normal((rows, bins))).astype(np.complex64)
    ref = h.astype(np.complex128)
    ref[:, 0] = ref[:, 0].real
    ref[:, -1] = ref[:, -1].real
    want = np.fft.irfft(ref, n, axis=1)
    h[:, 0].imag = np.inf  # ignored, as FFTW's c2r does
    h[:, -1].imag = -np.inf
    out = torch.zeros(rows, n + pad + 2, device="cuda")
    view = out[:, shift:shift + n]
    FftmReal(rows, n, fft_inv, 1.0 / n)(torch.from_numpy(h).cuda(), view)
    assert _rel(view.cpu().numpy(), want) <= RTOL
    assert not out[:, :shift].any() and not out[:, shift + n:].any()
