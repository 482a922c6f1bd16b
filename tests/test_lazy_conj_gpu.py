"""Tensors that torch conjugates or negates lazily (their memory holds other
values), as inputs, weights and outputs of every entry point, against FP64."""
import numpy as np
import pytest

from conftest import crandn
from openvsip_b200 import Fastconv, Fft2d, Fftm, FftmReal, col, fft_fwd, fft_inv, replica_spectrum, vmmul
from openvsip_b200.batch import Batch
from openvsip_b200.serve import Server

pytestmark = pytest.mark.gpu
RTOL = 2e-6  # the suite's bound for single-precision transforms
ROWS, N = 6, 96


def _forms():
    """(name, tensor from its values, its values from it) of lazy tensors."""
    import torch
    return [("conj", lambda v: v.conj().resolve_conj().conj()),
            ("neg", lambda v: torch._neg_view(-v)),
            ("both", lambda v: torch._neg_view(-v.conj().resolve_conj()).conj()),
            ("padded", lambda v: torch.nn.functional.pad(v.conj().resolve_conj(), (1, 2)).conj()[..., 1:-2])]


def _cuda(x):
    import torch
    return torch.from_numpy(x).cuda()


def _data(seed, shape):
    return crandn(np.random.default_rng(seed), shape)


def _plans():
    rep = _data(3, (N,))
    r = rep.astype(np.complex128)
    c = np.complex128
    yield Fftm(ROWS, N, fft_fwd), lambda x: np.fft.fft(x.astype(c))
    yield Fftm(ROWS, N, fft_inv, axis=col), lambda x: np.fft.ifft(x.astype(c), axis=0) * ROWS
    yield Fft2d(ROWS, N, fft_fwd), lambda x: np.fft.fft2(x.astype(c))
    yield Fastconv(rep, ROWS), lambda x: np.fft.ifft(np.fft.fft(x.astype(c)) * r)


@pytest.mark.parametrize("form", range(4))
def test_lazy_inputs_and_outputs(oracle, form):
    import torch
    name, make = _forms()[form]
    x = _data(1, (ROWS, N))
    for plan, ref in _plans():
        lazy = make(_cuda(x))
        assert (lazy.is_conj() or lazy.is_neg()) and np.array_equal(lazy.cpu().resolve_conj().resolve_neg().numpy(), x)
        assert oracle.rel_l2(plan(lazy).cpu().numpy(), ref(x)) <= RTOL, (name, plan)
        for inp in (_cuda(x), lazy):
            out = make(torch.zeros(ROWS, N, dtype=torch.complex64, device="cuda"))
            assert plan(inp, out) is out
            assert oracle.rel_l2(out.resolve_conj().resolve_neg().cpu().numpy(), ref(x)) <= RTOL, (name, plan)
        if not isinstance(plan, Fft2d):
            plan.in_place(lazy)
            assert oracle.rel_l2(lazy.resolve_conj().resolve_neg().cpu().numpy(), ref(x)) <= RTOL, (name, plan)


@pytest.mark.parametrize("form", range(4))
def test_lazy_weights_and_operands(oracle, form):
    import torch
    _, make = _forms()[form]
    x, w, wm = _data(1, (ROWS, N)), _data(2, (N,)), _data(4, (ROWS, N))
    d = lambda a: a.astype(np.complex128)  # noqa: E731
    spec = np.fft.fft(d(x))
    for weights in (w, wm):
        y = Fastconv(make(_cuda(weights)), ROWS)(_cuda(x))
        assert oracle.rel_l2(y.cpu().numpy(), np.fft.ifft(spec * d(weights))) <= RTOL
    for v, m in ((make(_cuda(w)), _cuda(x)), (_cuda(w), make(_cuda(x)))):
        assert oracle.rel_l2(vmmul(v, m).resolve_conj().resolve_neg().cpu().numpy(), d(w) * d(x)) <= RTOL
        out = make(torch.zeros(ROWS, N, dtype=torch.complex64, device="cuda"))
        assert vmmul(v, m, out) is out
        assert oracle.rel_l2(out.resolve_conj().resolve_neg().cpu().numpy(), d(w) * d(x)) <= RTOL
    got = replica_spectrum(make(_cuda(w)), matched=False)
    assert oracle.rel_l2(got.cpu().numpy(), np.fft.fft(d(w))) <= RTOL


def test_lazy_half_spectra_and_real_rows(oracle):
    import torch
    x = np.random.default_rng(5).standard_normal((ROWS, N)).astype(np.float32)
    f, b = FftmReal(ROWS, N, fft_fwd), FftmReal(ROWS, N, fft_inv, 1.0 / N)
    want = np.fft.rfft(x.astype(np.float64))
    assert oracle.rel_l2(f(torch._neg_view(-_cuda(x))).cpu().numpy(), want) <= RTOL
    out = torch.zeros(ROWS, N // 2 + 1, dtype=torch.complex64, device="cuda").conj()
    f(_cuda(x), out)
    assert oracle.rel_l2(out.resolve_conj().cpu().numpy(), want) <= RTOL
    back = torch._neg_view(torch.zeros(ROWS, N, device="cuda"))
    b(_cuda(want.conj().astype(np.complex64)).conj(), back)
    assert oracle.rel_l2(back.resolve_neg().cpu().numpy(), x) <= RTOL


def test_lazy_tensors_in_batches_and_served(oracle):
    n = 512
    x, r = _data(6, (4, n)), _data(7, (n,))
    want = np.fft.ifft(np.fft.fft(x.astype(np.complex128)) * r.astype(np.complex128))
    lazy = _cuda(x.conj()).conj()
    b = Batch()
    rid = b.add_replica(_cuda(r.conj()).conj(), kind="spectrum")
    out = _cuda(np.zeros_like(x))
    for jobs in ([(lazy, out, rid)], [(_cuda(x), out.conj(), rid)]):
        with pytest.raises(TypeError):
            b.set_jobs(jobs)  # the table would hold the other values
    xd = _cuda(x)
    b.set_jobs([(xd, out, rid)])
    import torch
    torch.cuda.synchronize()
    b.run()
    b.sync()
    assert oracle.rel_l2(out.cpu().numpy(), want) <= RTOL
    with Server([r], kind="spectrum", reserve_bytes=0) as s:
        assert oracle.rel_l2(s.submit(lazy, 0).wait(30).cpu().numpy(), want) <= RTOL
