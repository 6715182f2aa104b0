"""Operands of different numbers of terms are refused before anything is read: a
transposed view is handed to the kernel as the matrix under it, whose rows the
other operand counts."""
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("ka,kb", [(64, 56), (56, 64), (64, 0)])
@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
def test_terms_must_agree(monkeypatch, ka, kb, ta, tb):
    import hosnwt
    import surrogate

    def launched(*a, **k):
        raise AssertionError("launched")

    monkeypatch.setattr(hosnwt, "tc_gemm_views", launched)
    A = torch.zeros(ka, 32).t() if ta else torch.zeros(32, ka)
    B = torch.zeros(kb, 40).t() if tb else torch.zeros(40, kb)
    with pytest.raises(hosnwt.HosError, match="terms"):
        surrogate.gemm_bf16(A, B)
