"""Calls that the native path takes (plain matrices, vectors, an output that requires
grad), and that they come out as through the ctypes path.  What it leaves to that path
pays for a second library call there."""
import pytest

from openvsip_b200 import Fastconv, Fft2d, Fftm, FftmReal, build, col, fft_inv, vmmul, vsip

pytestmark = pytest.mark.gpu
R, N = 6, 80


def _x(*shape, seed=0):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.view_as_complex(torch.randn(*shape, 2, generator=g, device="cuda"))


def _calls():
    """(name, call) of every kind and form; a call returns its output."""
    import torch
    w = _x(N, seed=1)
    torch.cuda.synchronize()
    f, fc, f2 = Fftm(R, N), Fastconv(w, R), Fft2d(R, N)
    c, r, b = Fftm(N, R, axis=col), FftmReal(R, N), FftmReal(R, N, fft_inv)
    x, xv, real, half = _x(R, N), _x(N), torch.randn(R, N, device="cuda"), _x(R, N // 2 + 1)

    def grad(t):
        return torch.zeros_like(t).requires_grad_()

    yield "rows", lambda: f(x, torch.empty_like(x))
    yield "in place", lambda: f.in_place(x.clone())
    yield "submit", lambda: f.submit(x, torch.empty_like(x))
    yield "vector", lambda: f(xv, torch.empty_like(xv))
    yield "requires grad", lambda: f(x, grad(x)).detach()
    yield "fastconv", lambda: fc(x)
    yield "2-D", lambda: f2(x)
    yield "columns", lambda: c(x.t().contiguous())
    yield "r2c", lambda: r(real)
    yield "r2c vector", lambda: r(real[0], torch.empty_like(half[0]))
    yield "c2r", lambda: b(half)
    yield "vmmul", lambda: vmmul(w, x)
    yield "vmmul in place", lambda: (lambda y: vmmul(w, y, y))(x.clone())
    yield "vmmul vector", lambda: vmmul(w, xv)
    yield "vmmul strided", lambda: vmmul(w, _x(R, N + 3)[:, 3:])


def test_taken_and_the_same(monkeypatch):
    import torch
    build.build_torch()
    monkeypatch.setattr(vsip, "_native", vsip._load_native)
    monkeypatch.setattr(vsip, "_native_vmmul", vsip._load_vmmul)
    assert vsip._load()
    taken = []

    def spy(fn):
        def call(*args):
            taken.append(fn(*args))
            return taken[-1]
        return call

    monkeypatch.setattr(vsip, "_native", spy(vsip._native))
    monkeypatch.setattr(vsip, "_native_vmmul", spy(vsip._native_vmmul))
    for name, call in _calls():
        taken.clear()
        fast = call()
        assert taken == [0], name
        with monkeypatch.context() as m:
            m.setattr(vsip, "_native", vsip._no_native)
            m.setattr(vsip, "_native_vmmul", vsip._no_native)
            assert torch.equal(fast, call()), name


@pytest.mark.parametrize("v,m,o", [((N,), (R, N + 1), (R, N + 1)), ((N,), (R, N), (R + 1, N)), ((N,), (R, N), (R, N - 1)),
                                   ((N - 1,), (R, N), (R, N))])
def test_vmmul_refuses_other_shapes(v, m, o):
    with pytest.raises(ValueError):
        vmmul(_x(*v), _x(*m), _x(*o))
