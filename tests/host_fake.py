"""Child processes whose CUDA runtime is tests/fake_cudart.c: the library's host
code runs as on a B200, no kernel does."""
import os
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
LIB = os.path.join(ROOT, "newton-stein-variational-particle-filter_b200", "libsvpf_b200.so")

PRELUDE = r"""
import ctypes as C, os, sys
sys.path.insert(0, %r)
import numpy as np
import __graft_entry__ as ge
pkg = ge.load_package()
fake = C.CDLL(os.environ["LD_PRELOAD"])
fake.fake_launch.restype = C.c_char_p
fake.fake_set_memory.argtypes = [C.c_size_t]
fake.fake_memory_used.restype = C.c_size_t

def launches():
    # (kernel's mangled name, grid, block, dynamic shared memory) since the last call
    out = []
    for i in range(fake.fake_launches()):
        g, b, m = C.c_int(), C.c_int(), C.c_size_t()
        name = fake.fake_launch(i, C.byref(g), C.byref(b), C.byref(m)).decode()
        out.append((name, g.value, b.value, m.value))
    fake.fake_clear_launches()
    return out

def created(make):
    try:
        return make()
    except RuntimeError:
        return None
""" % ROOT


@pytest.fixture(scope="session")
def on_fake(tmp_path_factory):
    """Runs Python code after PRELUDE in a child on the fake runtime; its output."""
    cc = shutil.which("gcc") or shutil.which("cc")
    inc = "/usr/local/cuda/include"
    if cc is None or not os.path.exists(os.path.join(inc, "cuda_runtime_api.h")) or not os.path.exists(LIB):
        pytest.skip("no host compiler, CUDA headers or built library")
    so = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.run([cc, "-shared", "-fPIC", "-O1", "-I" + inc, os.path.join(HERE, "fake_cudart.c"), "-o", so], check=True)

    def run(code):
        r = subprocess.run([sys.executable, "-c", PRELUDE + code], env=dict(os.environ, LD_PRELOAD=so),
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
        return r.stdout

    return run
