"""Device memory of small 3-D tanks: those whose passes never go to the tensor
cores hold no matrices and no scratch for them (six tiles of sums per SM are 90 MB
for each of the three branches), and those that are sent there have both."""
import pytest

from host_lib import link, run


@pytest.fixture(scope="module")
def host_lib():
    return link()


SCRIPT = r"""
out = []
for size in SIZES:
    base = lib.host_cudart_bytes()
    lib.host_cudart_reset()
    t = tank(*size)
    out.append({"size": size, "MB": (lib.host_cudart_bytes() - base) / 1e6, "passes": launches("k_tc_pass")[0],
                "matrices": launches("k_tc_matrix")[0], "pending": lib.host_cudart_pending()})
    t.close()
print(json.dumps(out))
"""

# n1, n2, n3, M, p1, p2 and the MB of its fields and transform scratch, with a
# quarter to spare (29, 26 and 117 MB; 298, 295 and 362 with the sums)
SMALL = [((65, 17, 9, 3, 3, 3), 36), ((65, 33, 9, 2, 1, 1), 33), ((256, 32, 9, 3, 3, 3), 146)]


def test_small_tanks_hold_no_tensor_core_scratch(host_lib):
    for r, (size, mb) in zip(run(host_lib, SCRIPT.replace("SIZES", repr([s for s, _ in SMALL]))), SMALL):
        assert r["passes"] == 0 and r["matrices"] == 0 and r["MB"] < mb and r["pending"] == 0, r


def test_large_and_forced_tanks_have_them(host_lib):
    for r in run(host_lib, SCRIPT.replace("SIZES", "[(257, 129, 9, 5, 4, 4), (129, 129, 9, 7, 5, 5)]")):
        assert r["passes"] > 0 and r["matrices"] > 0, r
    for r in run(host_lib, SCRIPT.replace("SIZES", repr([s for s, _ in SMALL])), {"HOSNWT_FFT": "2"}):
        assert r["passes"] > 0 and r["matrices"] > 0 and r["pending"] == 0, r
    for r in run(host_lib, SCRIPT.replace("SIZES", repr([s for s, _ in SMALL])), {"HOSNWT_FFT": "1"}):
        assert r["passes"] == 0 and r["matrices"] == 0, r
