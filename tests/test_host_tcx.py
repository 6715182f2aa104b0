"""Which transforms go to the tensor cores when they are forced there (HOSNWT_FFT =
2): every kind with a matrix takes one pass per axis, no FFT and no sums."""
import pytest

from host_lib import link, run


@pytest.fixture(scope="module")
def host_lib():
    return link()


SCRIPT = r"""
out = []
for n1, n2, p1, p2 in SIZES:
    t = tank(n1, n2, 9, 3, p1, p2)
    i = t.info()
    for grid, shape in (("n", (n1, n2)), ("big", (i["nd1"], i["nd2"]))):
        for cx, cy, d in (("cos", "cos", 1), ("cos", "cos", -1), ("sin", "cos", -1), ("cos", "sin", -1), ("sin", "sin", -1)):
            lib.host_cudart_reset()
            t.transform(grid, d, cx, cy, np.zeros(shape))
            out.append([f"{shape} {cx} {cy} {d}", launches("k_tc_pass")[0], launches("k_tc_digits")[0],
                        sum(launches(k)[0] for k in ("k_fft_pass", "two_level", "ytl_", "axis_pass", "direct_pass"))])
    t.close()
print(json.dumps(out))
"""


def test_forced_transforms_take_the_tensor_cores(host_lib):
    sizes = [(65, 33, 3, 3), (129, 97, 2, 2), (194, 128, 1, 1), (66, 130, 3, 3), (257, 130, 3, 3), (514, 33, 3, 3)]
    for r in run(host_lib, SCRIPT.replace("SIZES", repr(sizes)), {"HOSNWT_FFT": "2"}):
        assert r[1:] == [2, 2, 0], r
