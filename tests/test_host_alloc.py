"""A device allocation that is refused while a tank is created, each one in
turn: hosnwt_create reports it and launches nothing afterwards.  What a tank can
do without (the matrices of the tensor-core passes, the layout tuner's scratch
outputs) may be refused and the tank still comes up, on the other passes."""
import pytest

from host_lib import link, run


@pytest.fixture(scope="module")
def host_lib():
    return link()


SCRIPT = r"""
size = SIZE
lib.host_cudart_reset()
t = tank(*size)
n = lib.host_cudart_mallocs()
t.close()
base = lib.host_cudart_bytes()
came_up, launched, leaked = [], [], []
for k in range(1, n + 1):
    lib.host_cudart_reset()
    lib.host_cudart_refuse(k)
    try:
        t = tank(*size)
        came_up.append(k)
        t.close()
    except hosnwt.HosError as e:
        if lib.host_cudart_launches_after_refusal():
            launched.append(k)
    if lib.host_cudart_bytes() != base:
        leaked.append(k)
print(json.dumps({"n": n, "came_up": came_up, "launched": launched, "leaked": leaked}))
"""


@pytest.mark.parametrize("size,optional", [((65, 33, 9, 3, 3, 3), 15), ((129, 65, 9, 4, 3, 3, 2), 15), ((65, 1, 9, 3, 3, 1, 2), 0)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else None)
def test_refused_allocation(host_lib, size, optional):
    out = run(host_lib, SCRIPT.replace("SIZE", repr(size)), {"HOSNWT_FFT": "2"})
    print(out)
    assert out["launched"] == [] and out["leaked"] == []
    # the optional allocations are the last ones of the creation
    assert len(out["came_up"]) <= optional and all(k > out["n"] - optional for k in out["came_up"]), out


LAUNCH_SCRIPT = r"""
out = []
for kern in KERNELS:
    lib.host_cudart_reset()
    lib.host_cudart_fail_launch(kern.encode())
    try:
        t = tank(*SIZE, icase=1)
        out.append([kern, "came up"])
        t.close()
    except hosnwt.HosError as e:
        out.append([kern, str(e)])
print(json.dumps(out))
"""


@pytest.mark.parametrize("size", [(65, 1, 9, 3, 3, 1), (65, 33, 9, 3, 3, 3)], ids=lambda v: "x".join(map(str, v)))
def test_refused_launch(host_lib, size):
    """A kernel of the step that cannot be launched while the step is captured:
    hosnwt_create says so (icase 1 launches none of them before)."""
    kernels = ["k_rk_err", "k_assemble", "k_rk_out"] + (["two_level"] if size[1] == 1 else ["k_fft_pass"])
    out = run(host_lib, LAUNCH_SCRIPT.replace("SIZE", repr(size)).replace("KERNELS", repr(kernels)))
    for kern, msg in out:
        assert "step capture" in msg, (kern, msg)
