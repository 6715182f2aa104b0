"""Transforms of long axes against numpy's FFT of the extended line: 32770 points
(D = 331 x 99), past what one staged twiddle table holds; 15389 (4 x 3847) and
20589 (4 x 5147) points, on both sides of what the table of the first level holds.

Tolerance: two sums of at most 5148 and 99 terms, each off by (K + 2) 2^-53 of
the sum of its terms' sizes, about sqrt(K) of an output: 1e-13 sqrt(N) as for
the other lengths is far above it and below any wrong term (1 / sqrt(N))."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu



def _ref(x, direction, cs):
    n, D = len(x), len(x) - 1
    if cs == "cos":
        f = np.fft.rfft(np.concatenate([x, x[D - 1:0:-1]])).real
        if direction > 0:
            f = f / D
            f[[0, D]] *= 0.5
            return f
        return 0.5 * (f + x[0] + x[D] * (1.0 - 2.0 * (np.arange(n) % 2)))
    x = x.copy()
    x[[0, D]] = 0.0
    f = -0.5 * np.fft.rfft(np.concatenate([x, -x[D - 1:0:-1]])).imag
    f[[0, D]] = 0.0
    return f * (2.0 / D) if direction > 0 else f


@pytest.mark.parametrize("n1,p,grid", [(16385, 3, "big"), (15389, 1, "n"), (20589, 1, "n")])
def test_long_axis_matches_fft(lib, n1, p, grid):
    import hosnwt
    from oracle.hos_oracle import default_input
    tank = hosnwt.Tank(default_input(icase=1, T_stop=5.0, toler=1e-7, f_out=10.0), n1, 1, 5, p, p, 1)
    n = tank.info()["nd1" if grid == "big" else "n1"]
    x = np.random.default_rng(3).standard_normal(n)
    for direction in (1, -1):
        for cs in ("cos", "sin"):
            got = tank.transform(grid, direction, cs, "cos", x[:, None])[:, 0]
            ref = _ref(x, direction, cs)
            err = np.max(np.abs(got - ref)) / np.max(np.abs(ref))
            print(direction, cs, err)
            assert err < 1e-13 * np.sqrt(n), (direction, cs, err)
    tank.close()
