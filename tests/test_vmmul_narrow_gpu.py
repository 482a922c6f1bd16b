"""vmmul on narrow matrices and on widths around its CTA's 256 threads: results, and
that narrow ones keep the GPU as busy as wide ones.  Bound: three roundings of products
and a sum, 4 * 2^-24 of |v| |m|."""
import numpy as np
import pytest

from conftest import crandn
from openvsip_b200 import vmmul

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(1, 2), (255, 1), (256, 1), (4099, 1), (127, 2), (129, 2), (300000, 2), (86, 3), (700, 16),
                                       (9, 170), (2, 255), (2, 256), (5, 257), (3, 511), (3, 512), (6, 514), (1200, 66)])
@pytest.mark.parametrize("pad,shift", [(0, 0), (2, 0), (1, 1)])
def test_narrow_and_ragged_widths(rows, cols, pad, shift):
    import torch
    rng = np.random.default_rng(rows + cols)
    m, v = crandn(rng, (rows, cols + pad)), crandn(rng, (cols,))
    x = torch.from_numpy(m).cuda()[:, shift:shift + cols]
    mx = m[:, shift:shift + cols].astype(np.complex128)
    out = torch.zeros(rows + 1, cols + pad + 2, dtype=torch.complex64, device="cuda")
    vmmul(torch.from_numpy(v).cuda(), x, out[:rows, shift:shift + cols])
    got = out[:rows, shift:shift + cols].cpu().numpy()
    assert (np.abs(got - v.astype(np.complex128) * mx) <= 4 * 2.0 ** -24 * np.abs(v) * np.abs(mx)).all()
    assert not out[:, :shift].any() and not out[:, shift + cols:].any() and not out[rows:].any()


def _us(fn, n=50):
    import torch
    e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    best = float("inf")
    for _ in range(5):
        e[0].record()
        for _ in range(n):
            fn()
        e[1].record()
        e[1].synchronize()
        best = min(best, e[0].elapsed_time(e[1]) * 1e3 / n)
    return best


def test_narrow_matrices_take_no_longer_than_twice_a_wide_one():
    import torch

    def time(cols):
        m = torch.ones((1 << 22) // cols, cols, dtype=torch.complex64, device="cuda")
        v, out = torch.ones(cols, dtype=torch.complex64, device="cuda"), torch.empty_like(m)
        vmmul(v, m, out)
        return _us(lambda: vmmul(v, m, out))

    wide = time(256)
    slow = {c: t for c in (1, 2, 3, 4, 8, 16, 64) if (t := time(c)) > 2 * wide}
    assert not slow, (wide, slow)
