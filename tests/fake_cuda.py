"""The native library on a recorded stand-in for the CUDA runtime (fake_cudart.cpp).

``run(script)`` compiles the stand-in once, preloads it in a child process and
runs ``script`` there after a prelude that loads the library and gives

- ``nat``, ``lib``: the ctypes binding and the library (no torch in this process);
- ``plan(n, torus, separable, mixed, flags, reach)``: a plan of one full-torus system with
  taps up to ``reach``, not yet solved;
- ``side``: a caller's stream handle; ``buf(plan)``: a device vector of the plan;
- ``report(prefix)``: the recorded names that follow ``prefix`` ("unordered", "launch").
"""

from __future__ import annotations

import atexit
import functools
import os
import pathlib
import shutil
import subprocess
import sys
import tempfile

from multiscat_b200 import build

HERE = pathlib.Path(__file__).resolve().parent
PRELUDE = '''
import ctypes, importlib.util, sys
import numpy as np
spec = importlib.util.spec_from_file_location("native", sys.argv[1])
nat = importlib.util.module_from_spec(spec)
sys.modules["native"] = nat
spec.loader.exec_module(nat)
lib = nat.load()
fake = ctypes.CDLL(None)
fake.fake_report.restype = ctypes.c_char_p
side = ctypes.c_void_p(0x7770)
D = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
I = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_int32))
keep = []

def report(prefix):
    lines = fake.fake_report().decode().splitlines()
    return [x.split(" ", 1)[1] for x in lines if x.startswith(prefix + " ")]

def plan(n, torus, separable, mixed=False, flags=0, reach=1):
    rng = np.random.default_rng(n)
    d = nat.PlanDesc()
    d.n_z, d.nkx, d.nky, d.n_systems = n, torus, torus, 1
    d.restart, d.max_iterations, d.rtol, d.precision, d.flags = 30, 100, 1e-10, int(mixed), flags
    v = np.zeros((torus, torus, n), complex)
    k = np.arange(-reach, reach + 1)
    f = rng.uniform(0.5, 1.0, (k.size, k.size))
    if separable:
        f = np.outer(f[0], f[1])
    v[np.ix_(k % torus, k % torus)] = f[:, :, None] * rng.uniform(0.5, 1.0, n)
    v[0, 0] = 1.0
    t = np.eye(n)
    c = torus * torus
    ix, iy = (x.astype(np.int32) for x in np.divmod(np.arange(c), torus))
    w = np.ones(2 * c)
    h = ctypes.c_void_p()
    for st in (lib.msc_plan_create(ctypes.byref(h), ctypes.byref(d)),
               lib.msc_plan_set_potential(h, D(v.view(float)), D(t)),
               lib.msc_plan_set_system(h, 0, c, I(ix), I(iy), D(np.ones(c)), D(w), D(-w), 0, D(np.zeros(2)))):
        assert st == 0, nat.last_error()
    h.cells = c * n
    return h

def buf(h):
    keep.append(np.zeros(2 * h.cells))
    return ctypes.c_void_p(keep[-1].ctypes.data)
'''


@functools.cache
def stand_in() -> str:
    folder = tempfile.mkdtemp(prefix="fake_cudart_")
    atexit.register(shutil.rmtree, folder, ignore_errors=True)
    so = pathlib.Path(folder) / "libfake_cudart.so"
    include = pathlib.Path(build.nvcc_path()).resolve().parent.parent / "include"
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", f"-I{include}", str(HERE / "fake_cudart.cpp"),
                    "-o", str(so)], check=True)
    return str(so)


def run(script: str, **env) -> str:
    full = {k: v for k, v in os.environ.items() if k != "MSC_TUNE"}
    full.update(env, LD_PRELOAD=stand_in())
    p = subprocess.run([sys.executable, "-c", PRELUDE + script, str(HERE.parent / "multiscat_b200" / "_native.py")],
                       env=full, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout + p.stderr
    return p.stdout
