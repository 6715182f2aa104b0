"""Which kernels the context-free transform launches, by length and lines, on
both sides of its rules."""
import pytest

from host_lib import link, run


@pytest.fixture(scope="module")
def host_lib():
    return link()


SCRIPT = r"""
out = []
for n, lines in CALLS:
    lib.host_cudart_reset()
    hosnwt.transform_noalloc(1, "cos", n, lines, 1 << 30, 1 << 31, 0)
    out.append({"n": n, "lines": lines, "pending": lib.host_cudart_pending(),
                **{k: launches(k)[0] for k in ("two_level_pass1", "two_level_pass2_lines", "two_level_pass2", "direct_pass",
                                               "axis_pass_lanes_k")}})
print(json.dumps(out))
"""


def _run(host_lib, calls):
    return run(host_lib, SCRIPT.replace("CALLS", repr(calls)))


def test_many_lines_gather_their_twiddles(host_lib):
    """16 lines and more of a length that factors: the pass that shares a staged
    tile of twiddles took five times as long (1024 points, 16 lines)."""
    for r in _run(host_lib, [(1024, 15), (1024, 16), (723, 32), (1026, 24), (513, 100), (2052, 16)]):
        assert r["pending"] == 0 and r["two_level_pass1"] == r["two_level_pass2"] > 0, r
        assert r["two_level_pass2_lines"] == 0, r


def test_long_lines_go_in_chunks(host_lib):
    """16 lines and more of 7900 points and up, of which fewer than 16 fit the fixed
    scratch at a time: two levels in chunks, not direct sums over every pair."""
    for r, want in zip(_run(host_lib, [(8193, 15), (8193, 16), (8193, 46), (16385, 4), (16385, 8), (8161, 33)]), (1, 2, 4, 1, 2, 3)):
        assert r["pending"] == 0 and r["axis_pass_lanes_k"] == 0 and r["two_level_pass1"] == want, r


def test_direct_sums_of_a_wave_and_a_rest(host_lib):
    """A few lines over 16 of a length that does not factor: a launch of 16 and one
    of the rest, not a last wave that is nearly empty; whole waves in one launch."""
    for r, want in zip(_run(host_lib, [(3000, 17), (3000, 20), (4202, 17), (3000, 16), (3000, 32), (1300, 40), (600, 300)]),
                       (2, 2, 2, 1, 1, 1, 1)):
        assert r["pending"] == 0 and r["axis_pass_lanes_k"] + r["direct_pass"] == want, r
