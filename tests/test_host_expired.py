"""A wait of a tensor-core pass that ran out: the kernel leaves a mark in page-locked
host memory (and one in device memory for the kernel that finishes split tiles).
Every call that runs passes reports it once it has synchronised, and clears both, so
that the tank can go on.  The marks are set here as the kernel would."""
import pytest

from host_lib import link, run


@pytest.fixture(scope="module")
def host_lib():
    return link()


SCRIPT = r"""
t = tank(65, 33, 9, 3, 3, 3)
host = ctypes.cast(lib.host_cudart_pinned(4), ctypes.POINTER(ctypes.c_uint))
found = (ctypes.c_void_p * 8)()
n = lib.host_cudart_blocks(4, found, 8)
words = [ctypes.cast(found[i], ctypes.POINTER(ctypes.c_uint)) for i in range(n)]
i = t.info()
x = np.zeros((65, 33))
arrs = t.get_rk_state()
calls = {
    "transform": lambda: t.transform("n", 1, "cos", "cos", x),
    "runge4_adapt2": lambda: t.runge4_adapt2(0.0, *arrs, i["delt"]),
    "step": lambda: t.step(i["delt"]),
    "advance": lambda: t.advance(t.info()["time_cur"] + 0.5 * i["delt"], 0.5 * i["delt"]),
    "advance_many": lambda: hosnwt.advance_many([t], [t.info()["time_cur"] + 0.5 * i["delt"]], [0.5 * i["delt"]]),
    "solveHOS2": lambda: t.solveHOS2(arrs, 0.0, 0.0, 0.0, 0.0),
}
out = {"words": n}
for name, call in calls.items():
    call()  # runs
    host[0] = 1
    for w in words:
        w[0] = 1
    try:
        call()
        out[name] = "no error"
    except hosnwt.HosError as e:
        out[name] = str(e)
    out[name + " left"] = int(host[0]) + sum(int(w[0]) for w in words)
    call()  # and runs again
host[0] = 2
try:
    calls["transform"]()
except hosnwt.HosError as e:
    out["lost"] = str(e)
print(json.dumps(out))
"""


def test_expired_wait_is_reported_once(host_lib):
    out = run(host_lib, SCRIPT)
    assert out["words"] == 1
    for name in ("transform", "runge4_adapt2", "step", "advance", "advance_many", "solveHOS2"):
        assert "(CUDA)" in out[name] and ("ran out" in out[name] or name == "advance_many") and out[name + " left"] == 0, (name, out)
    assert "must not be used further" in out["lost"]
