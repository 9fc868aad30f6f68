"""Runs a script against the library's host code with tests/cpp/fake_cudart.cpp
in place of the CUDA runtime, in a process of its own, on the CPU.

The script sees `lib` (the library), `N` (its ctypes binding), `fake` (the
stand-in's switches), `C` (ctypes) and the helpers below; what it leaves in
`result` comes back."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PRELUDE = r"""
import ctypes as C, json, os, sys, types
root = %(root)r
pkg = types.ModuleType("panopaea_gb300")  # the binding alone: no torch, which has a CUDA runtime of its own
pkg.__path__ = [os.path.join(root, "panopaea_gb300")]
sys.modules["panopaea_gb300"] = pkg
from panopaea_gb300 import _native as N
lib = N.load(build_if_missing=False)
fake = C.CDLL(%(fake)r)
for f in ("fake_fail_allocation", "fake_fail_attribute", "fake_fail_launch"):
    getattr(fake, f).argtypes = [C.c_long]
for f in ("fake_allocations", "fake_live", "fake_live_bytes", "fake_captures"):
    getattr(fake, f).restype = C.c_long
fake.fake_log_name.restype = C.c_char_p

def log():
    out = [(fake.fake_log_name(i).decode(), fake.fake_log_grid(i), fake.fake_log_block(i)) for i in range(fake.fake_log_size())]
    fake.fake_log_clear()
    return out

def kernels(of=None):
    return [n for n, _, _ in (log() if of is None else of)]

def grid(dims):
    g = C.c_void_p()
    make = lib.pg_grid_create_2d if len(dims) == 2 else lib.pg_grid_create_3d
    assert make(*dims, C.byref(g)) == 0, lib.pg_last_error()
    return g

def cells(dims, bytes_each=4):
    n = bytes_each
    for d in dims:
        n *= d
    # (16-byte aligned, as device memory is)
    buf = C.create_string_buffer(n + 256)
    keep.append(buf)
    return C.c_void_p((C.addressof(buf) + 255) // 256 * 256)

def solver(**kw):
    p = N.SolverParams()
    p.max_iter, p.rel_stop, p.rel_tol, p.mg_smooth = 100, 1, 1e-6, 2
    for k, v in kw.items():
        setattr(p, k, v)
    return p

keep, result = [], None
"""


@pytest.fixture(scope="session")
def host_cuda(tmp_path_factory):
    from panopaea_gb300 import build as B

    B.build()
    fake = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(B.nvcc()))), "include")
    cmd = [os.environ.get("CXX") or "g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-I" + include,
           os.path.join(ROOT, "tests", "cpp", "fake_cudart.cpp"), "-o", fake]
    p = subprocess.run(cmd, capture_output=True, text=True)
    assert p.returncode == 0, p.stderr

    def run(script, **env):
        code = PRELUDE % dict(root=ROOT, fake=fake) + script + "\nprint('RESULT ' + json.dumps(result))\n"
        e = {k: v for k, v in os.environ.items() if not k.startswith("PG_")}
        e.update(env, LD_PRELOAD=fake, CUDA_VISIBLE_DEVICES="")
        p = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, env=e, timeout=300)
        assert p.returncode == 0, (p.returncode, p.stdout[-2000:], p.stderr[-4000:])
        return json.loads(p.stdout.split("RESULT ", 1)[1])

    return run
