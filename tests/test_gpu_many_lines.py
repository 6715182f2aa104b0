"""hosnwt_transform_noalloc over many lines against numpy's FFT of the extended
lines: chunks of the fixed scratch used again between launches (2052 points: 63
lines a chunk, so 64, 72 and 130 lines end in chunks of one, nine and four; 8193
points: 15 a chunk), lengths that do not factor with split sums and their counters
(1300, 3000, 4202 points; D = 1299 = 3 x 433, 2999 and 4201 prime), few lines of
them (direct sums), both sides of 16 lines.  Each call runs twice, so that the second
meets the counters and partial sums of the first.

Tolerance: sums of K products of the inputs and rounded cosines, off by at most
(K + 2) 2^-53 of the sum of their sizes, about sqrt(K) of an output: 1.2e-16 K^(3/2)
/ sqrt(K) stays below 1e-13 sqrt(N) for every N here."""
import numpy as np
import pytest

from test_gpu_long_axis import _ref

pytestmark = pytest.mark.gpu

CALLS = [(2052, 64), (2052, 72), (2052, 130), (1024, 15), (1024, 16), (1024, 17), (723, 48), (66, 513),
         (1300, 9), (1300, 40), (3000, 17), (3000, 24), (4202, 9), (4202, 17), (5000, 20), (600, 9), (515, 20),
         (8193, 15), (8193, 16), (8193, 33), (4097, 3), (2048, 2), (1024, 1), (3000, 20)]


@pytest.mark.parametrize("direction,cs", [(1, "cos"), (-1, "cos"), (1, "sin"), (-1, "sin")])
@pytest.mark.parametrize("n,lines", CALLS, ids=lambda v: str(v))
def test_many_lines(lib, n, lines, direction, cs):
    torch = pytest.importorskip("torch")
    import hosnwt
    x = np.random.default_rng(n + lines).standard_normal((lines, n))
    d_in = torch.from_numpy(x).cuda()
    d_out = torch.full_like(d_in, float("nan"))
    stream = torch.cuda.current_stream().cuda_stream
    ref = np.stack([_ref(r, direction, cs) for r in x])
    for rep in range(2):
        d_out.fill_(float("nan"))
        hosnwt.transform_noalloc(direction, cs, n, lines, d_in.data_ptr(), d_out.data_ptr(), stream)
        err = np.max(np.abs(d_out.cpu().numpy() - ref)) / np.max(np.abs(ref))
        assert err < 1e-13 * np.sqrt(n), (rep, err)
