"""The native call path for CUDA tensors (csrc/fcb_torch.cpp): it takes plain
matrices only, and what it takes comes out as through the ctypes path."""
import numpy as np
import pytest

from openvsip_b200 import FcbError, Fftm, FftmReal, col, fft_inv, vsip

torch = pytest.importorskip("torch")


def _module():
    from openvsip_b200 import build
    build.build_torch()
    from openvsip_b200 import _fcb_torch
    return _fcb_torch


def test_leaves_everything_but_plain_cuda_matrices_to_the_general_path():
    m = _module()
    x = torch.zeros(2, 4, dtype=torch.complex64)
    for kind in range(4):
        assert m.exec(kind, 1, x, x, 4, 4) is None  # host tensors
        assert m.exec(kind, 1, np.zeros((2, 4)), [0], 4, 4) is None
    assert m.exec(7, 1, x, x, 4, 4) is None
    with pytest.raises(TypeError):
        m.exec(0, 1, x)
    with pytest.raises(TypeError):
        m.exec(0, 1, x, x, "4", 4)


def _forms(n):
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.view_as_complex(torch.randn(6, n + 4, 2, generator=g, device="cuda"))
    yield x[:, :n].contiguous()
    yield x[:, 1:n + 1]                       # odd start, wider rows
    yield x[::2, 2:n + 2]                     # every other row
    yield x[:1, 3:n + 3]                      # one row
    yield x[2, :n]                            # a vector
    yield torch.nn.Parameter(x[:, :n].contiguous())
    yield x.t().contiguous().t()[:, :n]       # columns apart: refused
    yield x[:, :n - 1]                        # wrong length: refused
    yield x[:, :n].real                       # wrong type: refused
    yield x[:1, :n].expand(4, n)              # rows on top of each other: refused


@pytest.mark.gpu
@pytest.mark.parametrize("n", [16, 100])
def test_same_results_and_refusals_as_the_ctypes_path(n, monkeypatch):
    _module()
    f, c = Fftm(6, n), Fftm(n, 6, fft_inv, axis=col)
    r = FftmReal(6, 2 * n)

    def outcome(call, x):
        try:
            with torch.no_grad():
                return call(x).detach().cpu()
        except (TypeError, ValueError, FcbError) as e:
            return type(e)

    calls = [(lambda x: f(x), lambda x: x), (lambda x: f.in_place(x.clone()), lambda x: x),
             (lambda x: c(x.t().contiguous() if x.dim() == 2 else x), lambda x: x),
             (lambda x: r(x), lambda x: torch.view_as_real(x).reshape(*x.shape[:-1], -1) if x.is_complex() else x)]
    for call, form in calls:
        for x in _forms(n):
            fast = outcome(call, form(x.detach()))
            with monkeypatch.context() as m:
                m.setattr(vsip, "_native", vsip._no_native)
                slow = outcome(call, form(x.detach()))
            assert torch.equal(fast, slow) if isinstance(slow, torch.Tensor) else fast is slow, (x.shape, fast, slow)
    p = torch.nn.Parameter(torch.ones(6, n, dtype=torch.complex64, device="cuda"))
    assert torch.equal(f(p).detach(), f(p.detach().clone()))
