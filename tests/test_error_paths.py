"""Calls that spread their work over streams of the context, when a CUDA call inside
them fails: the library's objects linked against a fake runtime (fake_cudart.cpp)
that runs no kernels and fails its n-th call.  Wherever the call stops it leaves no
work that nobody has waited for, the next call succeeds, and the context's streams
and events are made once and destroyed with it."""
import os
import subprocess
import sys

import pytest

from fem25_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))

RUN = r"""
import ctypes as C, sys
import numpy as np
from fem25_b200 import Context, synth
L = sys.modules["fem25_b200.lib"]
L.LIB_PATH = sys.argv[1]
fake = C.CDLL(sys.argv[1])
fake.fake_fail_at.argtypes = [C.c_longlong]
mesh, pairs, _ = synth.make_config(0, nx=30, nz=15)
ctx = Context(mesh)
if sys.argv[2] == "driver":
    out = np.empty(ctx.nzero, np.complex64)
    call = lambda: L.lib().fem25_asmble_driver(ctx.h, ctx.nzero, b"B", 0.5, 1e-4, out.ctypes.data)
else:
    a = np.zeros(ctx.nzero, np.complex128)
    call = lambda: L.lib().fem25_sparse_factor_dev(ctx.h, a.ctypes.data, None)
failed, n, live = 0, 0, None
while True:  # the first failures come in a context that has made nothing yet
    n += 1 if n < 400 else 7
    fake.fake_fail_at(n)
    r = call()
    assert fake.fake_pending() == 0, f"work left running: failure {n}, status {r}"
    if r == 0:
        break
    failed += 1
fake.fake_fail_at(0)
assert failed > 20, failed
assert call() == 0 and fake.fake_pending() == 0
made = [fake.fake_live(k) for k in (0, 1)]
ctx.close()
assert [fake.fake_live(k) for k in (0, 1)] == [0, 0], (made, [fake.fake_live(k) for k in (0, 1)])
"""


@pytest.fixture(scope="module")
def fake_library(tmp_path_factory):
    build.build()
    tmp = tmp_path_factory.mktemp("fake")
    obj, so = str(tmp / "fake_cudart.o"), str(tmp / "libfem25gpu_fake.so")
    cuda = os.path.dirname(os.path.dirname(build.NVCC))
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-I", os.path.join(cuda, "include"), "-c", "-o",
                    obj, os.path.join(HERE, "fake_cudart.cpp")], check=True)
    names = [u[2] if len(u) > 2 else u[0] + ".o" for u in build.UNITS] + [h[0] + ".o" for h in build.HOST]
    subprocess.run(["g++", "-shared", "-o", so, obj] + [os.path.join(build.OBJ, f) for f in names]
                   + ["-lgomp", "-Wl,-Bsymbolic"], check=True)
    return so


@pytest.mark.parametrize("what", ["driver", "factor"])
def test_failures_leave_nothing_behind(fake_library, what):
    r = subprocess.run([sys.executable, "-c", RUN, fake_library, what], capture_output=True, text=True,
                       cwd=os.path.dirname(HERE))
    assert r.returncode == 0, r.stderr[-2000:]
