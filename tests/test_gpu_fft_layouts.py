"""Every layout that the FFT layout tuner may pick (threads per CTA, sequences
per CTA) gives the bits of the default one: the lines' arithmetic does not
depend on it.  Held with HOSNWT_FFT_LAYOUT, on lengths of each plan (powers of
two, generic radices, Rader with up to 16 lines per CTA, Bluestein)."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# n1, n2, M, p1, p2; Rader: D = 37, 193, 131, 257; Bluestein: 1407, 2 x 41; radices 13, 27, 64, 65
SIZES = [(194, 38, 1, 1, 1), (352, 33, 7, 7, 7), (129, 65, 3, 3, 3), (84, 66, 3, 3, 1)]

SCRIPT = r"""
import hashlib, json, sys
import numpy as np
sys.path[:0] = [ROOT, ROOT + "/hos-nwt_gb300", ROOT + "/tests"]
import hosnwt
from oracle.hos_oracle import default_input
out = []
for n1, n2, M, p1, p2 in SIZES:
    t = hosnwt.Tank(default_input(T_stop=5.0, toler=1e-7, f_out=10.0), n1, n2, 9, M, p1, p2)
    i = t.info()
    rng = np.random.default_rng(11)
    for grid, shape in (("n", (n1, n2)), ("big", (i["nd1"], i["nd2"]))):
        x = rng.standard_normal(shape)
        for d in (1, -1):
            for cx in ("cos", "sin"):
                for cy in ("cos", "sin"):
                    h = hashlib.sha256(np.ascontiguousarray(t.transform(grid, d, cx, cy, x)).tobytes()).hexdigest()
                    out.append([f"{n1}x{n2} {grid} {d} {cx} {cy}", h])
    t.close()
print(json.dumps(out))
"""


def _run(layout):
    env = {k: v for k, v in os.environ.items() if not k.startswith("HOSNWT_FFT")}
    env.update({"HOSNWT_FFT": "1", "HOSNWT_FFT_TUNE": "0"})
    if layout:
        env["HOSNWT_FFT_LAYOUT"] = layout
    r = subprocess.run([sys.executable, "-c", f"ROOT = {ROOT!r}\nSIZES = {SIZES!r}\n" + SCRIPT], cwd=ROOT, env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, (r.stdout[-2000:], r.stderr[-3000:])
    return json.loads(r.stdout.strip().splitlines()[-1])


@pytest.fixture(scope="module")
def default(lib):
    return _run(None)


@pytest.mark.parametrize("nt", [256, 512])
@pytest.mark.parametrize("shift", [-2, -1, 0, 1])
def test_layout_gives_the_same_bits(default, nt, shift):
    got = _run(f"{nt},{shift}")
    wrong = [a[0] for a, b in zip(got, default) if a != b]
    assert len(got) == len(default) and wrong == []
