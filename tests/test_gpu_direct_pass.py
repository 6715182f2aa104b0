"""The direct sums of few lines (direct_pass) on the truncated transforms of 2-D
tanks, which pair their inputs, and the full ones, which pair their outputs: one
RK4(5) step against the oracle where the dealiased length does not factor (D =
127, 509, 1019 and 2053 are prime).  The batches of a step, one to nine fields, take four
to 32 outputs per CTA."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1", [64, 255, 510, 1027])
def test_step_matches_oracle(lib, n1):
    import hosnwt
    from oracle.hos_oracle import Tank as OTank, default_input
    inp = default_input(T_stop=5.0, amp_mono=0.02, nu_mono=0.7, toler=1e-7)
    args = dict(n1=n1, n2=1, n3=9, mHOS=4, p1=3, p2=1)
    g, o = hosnwt.Tank(inp, **args), OTank(inp, **args)
    assert g.info()["nd1"] == 2 * n1
    rng = np.random.default_rng(n1)
    decay = np.exp(-20.0 * np.arange(n1) / n1)[:, None]
    st = [a.copy() for a in o.state_tuple()]
    st[0] = o.fourier.F2S(1e-3 * decay * rng.standard_normal((n1, 1)))
    st[1] = o.fourier.F2S(1e-3 * decay * rng.standard_normal((n1, 1)))
    res, err, _, _ = o.runge4_adapt2(0.0, *st, o.delt)
    got, gerr = g.runge4_adapt2(0.0, *st, o.delt)
    keys = ("eta", "phis", "a_add_1", "a_add_2", "a_add_ramp", "a_add_3", "eta1st", "eta2nd", "a1st", "a2nd")
    for k, a in zip(keys, got):
        assert np.max(np.abs(a - res[k])) <= 1e-10 * max(np.max(np.abs(res[k])), 1e-300), k
    assert abs(gerr - err) <= 1e-6 * err
    g.close()
