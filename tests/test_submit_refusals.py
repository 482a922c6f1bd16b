"""submit() on plans that cannot queue calls refuses with the library's error."""
import numpy as np
import pytest

from openvsip_b200 import FcbError, FftmReal, _lib, vsip


class _Library:
    """Plans succeed; a real plan answers fcb_exec as the library does."""

    def fcb_plan_fftm_real(self, *args):
        return 0

    def fcb_exec_async(self, *args):
        return 1  # FCB_ERR_INVALID

    def fcb_last_error(self):
        return b"real-FFT plans run through fcb_exec_r2c / fcb_exec_c2r"

    def fcb_destroy(self, h):
        return 0


def test_real_plans_refuse_submit(monkeypatch):
    fake = _Library()
    monkeypatch.setattr(vsip, "lib", lambda: fake)
    monkeypatch.setattr(_lib, "lib", lambda: fake)
    p = FftmReal(2, 8)
    x = np.zeros((2, 8), dtype=np.complex64)
    with pytest.raises(FcbError):
        p.submit(x, x)
    with pytest.raises(TypeError):
        p.submit(x.real.copy(), x)
    with pytest.raises(ValueError):
        p.submit(x[:, :5], x[:, :5])
