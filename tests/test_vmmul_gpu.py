"""vmmul on the GPU where its kernel changes: odd and even widths, rows that do
and do not start 16-byte aligned, row counts around the four a thread holds, in
place.  Bound: three roundings of products and a sum, 4 * 2^-24 of |v| |m|."""
import numpy as np
import pytest

from conftest import crandn
from openvsip_b200 import vmmul

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 7), (5, 8), (1, 1000), (4, 514), (70000, 6), (1200, 1025), (33, 4096)])
@pytest.mark.parametrize("pad,shift", [(0, 0), (2, 0), (3, 1), (2, 1)])
def test_vmmul_shapes_and_alignments(rows, cols, pad, shift):
    import torch
    rng = np.random.default_rng(rows + cols)
    m, v = crandn(rng, (rows, cols + pad)), crandn(rng, (cols,))
    dm, dv = torch.from_numpy(m).cuda(), torch.from_numpy(v).cuda()
    x = dm[:, shift:shift + cols]
    mx = m[:, shift:shift + cols].astype(np.complex128)
    want = v.astype(np.complex128) * mx
    out = torch.zeros(rows, cols + pad + 2, dtype=torch.complex64, device="cuda")
    vmmul(dv, x, out[:, shift:shift + cols])
    got = out[:, shift:shift + cols].cpu().numpy()
    assert (np.abs(got - want) <= 4 * 2.0 ** -24 * np.abs(v) * np.abs(mx)).all()
    assert not out[:, :shift].any() and not out[:, shift + cols:].any()
    vmmul(dv, x, x)  # in place
    assert np.array_equal(x.cpu().numpy(), got)
    assert torch.equal(dm[:, :shift].cpu(), torch.from_numpy(m[:, :shift].copy()))
    assert torch.equal(dm[:, shift + cols:].cpu(), torch.from_numpy(m[:, shift + cols:].copy()))
