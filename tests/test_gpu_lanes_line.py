"""Direct sums along y (axis_pass_lanes_line) with eight, four and two outputs per
thread, against the oracle.

HOSNWT_FFT = 0 and lengths D = N - 1 that are prime send every y pass there.  The
sizes sit on the edges of its split: 64 lines per CTA, an odd number of lane
outputs (D / 2 + 1), and enough lines for eight outputs per thread.

Tolerance: a sum of K products of the inputs and rounded cosines is off by at
most (K + 2) 2^-53 of the sum of their sizes, about sqrt(K) of an output; two
passes of at most K = N terms give 2.3e-16 K^(1/2) K, below 1e-13 sqrt(N) for
N <= 430 along y (the x passes are shorter sums in two levels).
"""
import json
import os
import subprocess
import sys

import pytest

from test_gpu_fft import ROOT, SCRIPT

pytestmark = pytest.mark.gpu

SIZES = [
    (65, 36, 3, 3),     # D 71: one line more than a CTA; 36 lane outputs
    (64, 38, 1, 1),     # D 37: 19 lane outputs, one CTA of lines
    (257, 54, 3, 3),    # D 53, 107: truncated outputs too
    (9700, 228, 1, 1),  # D 227: eight outputs per thread
]


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
def test_passes_match_oracle(lib, size):
    script = f"ROOT = {ROOT!r}\nSIZES = [{size!r}]\n" + SCRIPT
    env = dict(os.environ, HOSNWT_FFT="0")
    env.pop("HOSNWT_FFT_DF", None)
    r = subprocess.run([sys.executable, "-c", script], cwd=ROOT, env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, (r.stdout[-2000:], r.stderr[-3000:])
    out = json.loads(r.stdout.strip().splitlines()[-1])
    print(size, out)
    assert out["worst_fraction_of_tol"] < 1.0
