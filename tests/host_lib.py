"""The library's own objects linked against the runtime of host_cudart.cpp, for
tests of its host code on a machine without a GPU.  Kernels are recorded, not
run; each script runs in a process of its own."""
import glob
import json
import os
import shutil
import subprocess
import sys
import tempfile

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "hos-nwt_gb300")
INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

PRELUDE = r"""
import ctypes, json, sys
sys.path[:0] = [ROOT, ROOT + "/hos-nwt_gb300", ROOT + "/tests"]
import numpy as np
import hosnwt, workloads
lib = hosnwt.load_library(LIB)
for f in ("host_cudart_bytes", "host_cudart_peak"):
    getattr(lib, f).restype = ctypes.c_longlong
lib.host_cudart_pinned.restype = ctypes.c_void_p
lib.host_cudart_pinned.argtypes = [ctypes.c_longlong]
lib.host_cudart_blocks.argtypes = [ctypes.c_longlong, ctypes.POINTER(ctypes.c_void_p), ctypes.c_int]

def tank(n1, n2, n3, M, p1, p2=1, wmk=1, icase=2, **kw):
    if icase == 1:
        inp = workloads.base_input(icase=1, islosh=3, aslosh=0.02, T_stop=5.0, toler=1e-7, **kw)
    else:
        inp = workloads.base_input(icase=2, amp_mono=0.02, nu_mono=0.7, i_wmk=wmk, T_stop=5.0, toler=1e-7, **kw)
    return hosnwt.Tank(inp, n1, n2, n3, M, p1, p2)

def launches(part):
    most = ctypes.c_longlong()
    return lib.host_cudart_launches(part.encode(), ctypes.byref(most)), most.value
"""


def link():
    """Build the library, link its objects once per session; path of the result."""
    if shutil.which("g++") is None or not os.path.isdir(INC):
        pytest.skip("needs g++ and the CUDA headers")
    import build
    build.build()
    objs = sorted(glob.glob(os.path.join(PKG, "_build", "*.o")))
    out = os.path.join(tempfile.mkdtemp(prefix="hosnwt_host_"), "libhosnwt_host.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-I", INC, os.path.join(ROOT, "tests", "host_cudart.cpp")]
                   + objs + ["-Wl,-z,defs", "-Wl,-Bsymbolic", "-o", out], check=True)
    return out


def run(lib_path, script, env=None):
    """Run `script` after the prelude; its last line of output is JSON."""
    e = {k: v for k, v in os.environ.items() if not k.startswith("HOSNWT_FFT")}
    e.update(env or {})
    r = subprocess.run([sys.executable, "-c", f"ROOT = {ROOT!r}\nLIB = {lib_path!r}\n" + PRELUDE + script], cwd=ROOT, env=e,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, (r.returncode, r.stdout[-2000:], r.stderr[-3000:])
    return json.loads(r.stdout.strip().splitlines()[-1])
