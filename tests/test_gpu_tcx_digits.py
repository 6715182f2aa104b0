"""All the digit products of the tensor-core passes (tcx.cu), forced on with
HOSNWT_FFT = 2, on the kinds that have a matrix along both axes: F2S in cosines
and sines, S2F in cosines.

Tolerance: per pass the products left out are below 6 2^-54 of the largest input per
term, K terms of either parity, on outputs of about sqrt(2 K) inputs: 2.4e-16
sqrt(K), and the fixed-point sums are rounded to 2^-50 of the largest (9e-16 over
sqrt(2 K), less than 2e-16 from K = 17 on).  Two passes, and 5e-16 for the oracle's own
FFT: 4.8e-16 sqrt(K) + 9e-16, 4e-15 at the smallest length.  A product of level 5
that is missing costs up to 2^-45 = 2.8e-14 of the largest per term.
"""
import json
import os
import subprocess
import sys

import pytest

from test_gpu_fft import ROOT

pytestmark = pytest.mark.gpu

SIZES = [(65, 33, 3, 3), (129, 97, 2, 2), (194, 128, 1, 1), (66, 130, 3, 3)]

SCRIPT = r"""
import json, sys
import numpy as np
sys.path[:0] = [ROOT, ROOT + "/hos-nwt_gb300"]
import hosnwt
from oracle.hos_oracle import Fourier, default_input
rng = np.random.default_rng(17)
out = []
for n1, n2, p1, p2 in SIZES:
    inp = default_input(T_stop=5.0, amp_mono=0.02, nu_mono=0.7, theta_mono=10.0, ylen=20.0, toler=1e-7)
    g = hosnwt.Tank(inp, n1, n2, 9, 3, p1, p2)
    nd1, nd2 = ((p1 + 1) * n1) // 2, ((p2 + 1) * n2) // 2
    F = Fourier(n1, n2, nd1, nd2, 16)
    for grid, shp in (("n", (n1, n2)), ("big", (nd1, nd2))):
        for csx, csy, d in (("cos", "cos", 1), ("cos", "cos", -1), ("sin", "cos", -1), ("cos", "sin", -1), ("sin", "sin", -1)):
            a = rng.standard_normal(shp)
            f = {("n", 1): F.S2F, ("n", -1): F.F2S, ("big", 1): F.S2F_big, ("big", -1): F.F2S_big}[grid, d]
            ref = f(a, csx, csy)
            rel = float(np.max(np.abs(g.transform(grid, d, csx, csy, a) - ref)) / np.max(np.abs(ref)))
            out.append([f"{shp[0]}x{shp[1]} {csx} {csy} {d}", rel, 4.8e-16 * np.sqrt((max(shp) + 1) // 2) + 9e-16])
    g.close()
print(json.dumps(out))
"""


def test_digit_products(lib):
    env = dict(os.environ, HOSNWT_FFT="2")
    env.pop("HOSNWT_FFT_DF", None)
    r = subprocess.run([sys.executable, "-c", f"ROOT = {ROOT!r}\nSIZES = {SIZES!r}\n" + SCRIPT], cwd=ROOT, env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, (r.stdout[-2000:], r.stderr[-3000:])
    out = json.loads(r.stdout.strip().splitlines()[-1])
    print(out)
    assert [o for o in out if not o[1] < o[2]] == []
