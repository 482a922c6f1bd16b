"""Host parts of the library in small C++ programs that answer some of its calls
themselves (of the CUDA runtime, of the allocator).  No GPU is used."""
import os
import shutil
import subprocess

import pytest

from openvsip_b200 import build as b

HERE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native")


def _run(tmp_path, program, source):
    """Builds tests/native/<program>.cpp with one of the library's .cu files and runs it."""
    if not (shutil.which("nvcc") or os.path.exists("/usr/local/cuda/bin/nvcc")) or not shutil.which("g++"):
        pytest.skip("needs nvcc and g++")
    obj, exe = str(tmp_path / "part.o"), str(tmp_path / program)
    include = [f"-I{b.CSRC}", f"-I{os.path.join(b.ROOT, 'include')}"]
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(b.nvcc())))
    subprocess.run([b.nvcc(), *b.ARCH, "-std=c++17", *include, "-c", os.path.join(b.CSRC, source), "-o", obj], check=True)
    subprocess.run(["g++", "-std=c++17", "-O1", *include, f"-I{cuda}/include", os.path.join(HERE, program + ".cpp"), obj, "-o", exe,
                    "-Wl,--unresolved-symbols=ignore-all", f"-L{cuda}/lib64", f"-Wl,-rpath,{cuda}/lib64", "-lcudart", "-lpthread"], check=True)
    return subprocess.run([exe], capture_output=True, text=True, timeout=60)


def test_bound_of_few_rows_is_stored_once_final(tmp_path):
    r = _run(tmp_path, "resident_bound", "fcb200.cu")
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)


def test_mixed_plans_report_failed_allocations(tmp_path):
    r = _run(tmp_path, "mixed_alloc", "fcb_mixed.cu")
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
