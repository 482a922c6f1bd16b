"""The native call path is built again, and not used, when it was made for another
torch or Python (it relies on the layout of their objects)."""
import os
import subprocess
import sys
import types

import pytest

pytest.importorskip("torch")

from openvsip_b200 import _lib, build, vsip  # noqa: E402


class _Compiled(Exception):
    pass


def test_rebuilt_for_another_torch(monkeypatch):
    out = build.build_torch()
    assert os.path.exists(out)

    def run(cmd, **kw):
        assert any("another torch" in c for c in cmd)
        raise _Compiled

    monkeypatch.setattr(subprocess, "run", run)
    assert build.build_torch() == out  # up to date: not compiled
    monkeypatch.setattr(_lib, "torch_tag", lambda: "another torch")
    with pytest.raises(_Compiled):
        build.build_torch()


@pytest.mark.parametrize("built_for", [None, "another torch"])
def test_not_used_for_another_torch(monkeypatch, built_for):
    def never(*args):
        raise AssertionError("the module was used")

    stale = types.ModuleType("openvsip_b200._fcb_torch")
    stale.bind = stale.exec = never
    if built_for:
        stale.built_for = built_for
    import openvsip_b200
    monkeypatch.setitem(sys.modules, "openvsip_b200._fcb_torch", stale)
    monkeypatch.setattr(openvsip_b200, "_fcb_torch", stale, raising=False)
    monkeypatch.setattr(vsip, "_native", vsip._load_native)
    assert vsip._load_native(0, 1, None, None, 1, 1) is None
    assert vsip._native is vsip._no_native
