"""The tensor-core transform passes (tcx.cu) against the oracle, forced on
with HOSNWT_FFT = 2 wherever the tank has a matrix.

The sizes sit on the edges of the passes' tiles: 128 lines and 96 outputs per
parity (97 = D / 2 + 1 for D = 193, 192), 32 terms per stage, 64 terms per
digit block; even and odd D, lines one more than a tile, tiles split over
segments and (with the eight fields of test_many_fields) whole tiles.

Tolerance: a pass leaves out products below 2^-54 of the largest per term
(level 6 of the digits and the remainders, six of them), so an output is off
by at most 6 * 2^-54 * K of the largest input for K terms, and its size is
about sqrt(K) of it: 3.3e-16 * sqrt(K) per pass.  1e-14 * sqrt(N) for two
passes leaves room for the passes that keep the FFT (S2F in sin) and for the
rounding of the fixed-point sums (2^-50).
"""
import json
import os
import subprocess
import sys

import pytest

from test_gpu_fft import NAN_SCRIPT, ROOT, SCRIPT

pytestmark = pytest.mark.gpu

SIZES = [
    (65, 33, 3, 3),    # D 64, 32 | 129, 65: fewer lines than a tile
    (129, 97, 2, 2),   # D 128, 96 | 192, 144: one line more than a tile, 97 outputs per parity
    (194, 128, 1, 1),  # D 193 (97 outputs per parity), 127; no dealiased grid of its own
    (257, 130, 3, 3),  # D 256, 129 | 513, 259: two tiles and one line
    (514, 33, 3, 3),   # D 513 | 1027: the sums drained several times
]


def _run(script, env_more):
    env = dict(os.environ, HOSNWT_FFT="2")
    env.pop("HOSNWT_FFT_DF", None)
    env.update(env_more)
    r = subprocess.run([sys.executable, "-c", script], cwd=ROOT, env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, (r.stdout[-2000:], r.stderr[-3000:])
    return json.loads(r.stdout.strip().splitlines()[-1])


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
def test_passes_match_oracle(lib, size):
    script = f"ROOT = {ROOT!r}\nSIZES = [{size!r}]\n" + SCRIPT.replace("1e-13 * np.sqrt", "1e-14 * np.sqrt")
    out = _run(script, {})
    print(size, out)
    assert out["worst_fraction_of_tol"] < 1.0


def test_nan_and_inf_reach_the_outputs(lib):
    out = _run(f"ROOT = {ROOT!r}\n" + NAN_SCRIPT, {})
    for bad in ("nan", "inf"):
        assert out[bad], (bad, out)
        assert out[bad + "_after"] < 1e-13 * 23, (bad, out)


STEP_SCRIPT = r"""
import json, sys, tempfile
import numpy as np
sys.path[:0] = [ROOT, ROOT + "/hos-nwt_gb300", ROOT + "/tests"]
import hosnwt
from oracle.hos_oracle import Tank as OTank, default_input
inp = default_input(T_stop=5.0, amp_mono=0.02, nu_mono=0.7, theta_mono=10.0, ylen=20.0, toler=1e-7)
args = dict(n1=129, n2=65, n3=9, mHOS=4, p1=3, p2=3)
g, o = hosnwt.Tank(inp, **args), OTank(inp, **args)
rng = np.random.default_rng(7)
decay = np.exp(-0.2 * (np.arange(129)[:, None] + np.arange(65)[None, :]))
st = [a.copy() for a in o.state_tuple()]
st[0] = o.fourier.F2S(1e-3 * decay * rng.standard_normal((129, 65)))
st[1] = o.fourier.F2S(1e-3 * decay * rng.standard_normal((129, 65)))
res, err, _, _ = o.runge4_adapt2(0.0, *st, o.delt)
got, gerr = g.runge4_adapt2(0.0, *st, o.delt)
keys = ("eta", "phis", "a_add_1", "a_add_2", "a_add_ramp", "a_add_3", "eta1st", "eta2nd", "a1st", "a2nd")
worst = max(float(np.max(np.abs(a - res[k]))) / max(float(np.max(np.abs(res[k]))), 1e-300) for k, a in zip(keys, got))
print(json.dumps({"worst": worst, "err": abs(gerr - err) / err}))
"""


def test_many_fields(lib):
    """One RK4(5) step with every pass forced on: batches of many fields, the
    accumulation epilogue, truncated dealiasing, the three streams."""
    out = _run(f"ROOT = {ROOT!r}\n" + STEP_SCRIPT, {})
    assert out["worst"] <= 1e-10 and out["err"] <= 1e-6, out
