"""Long axes: every pass of a tank is launched within the shared memory of its
kernel, for lengths on both sides of what the staged tables of the two-level
passes can hold (D = 25599 points a table)."""
import pytest

from host_lib import link, run


@pytest.fixture(scope="module")
def host_lib():
    return link()


SCRIPT = r"""
out = []
for n1, p in SIZES:
    lib.host_cudart_reset()
    t = tank(n1, 1, 5, 3, p, icase=1)
    one, two = launches("two_level_pass1"), launches("two_level_pass2")
    out.append({"n1": n1, "pending": lib.host_cudart_pending(), "one": one[0], "two": two[0], "smem": max(one[1], two[1])})
    t.close()
print(json.dumps(out))
"""

# n1, p
SIZES = [(12800, 3),   # D = 25599 on the dealiased grid: the last whose table fits
         (16385, 3),   # D = 16384 | 32769 = 331 x 99
         (25600, 1), (25601, 1), (25606, 1), (32769, 1)]
# D = 4 x 3847, 4 x 4999, 4 x 5147 and 4 x 6553: the first level's table of 2 A
# pairs with A on both sides of 5119
WIDE = [(15389, 1), (19997, 1), (20589, 1), (26213, 1)]


@pytest.mark.parametrize("sizes", [SIZES, WIDE], ids=["long", "wide"])
def test_long_axes(host_lib, sizes):
    for r in run(host_lib, SCRIPT.replace("SIZES", repr(sizes))):
        assert r["one"] > 0, r
        assert r["pending"] == 0 and r["one"] == r["two"] and r["smem"] <= 200 * 1024, r
