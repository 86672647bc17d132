"""Rounding of the window-row tensor-core leaf (boxes of 4 points, and wherever the shared-operand form does not
apply) against the FP64 transform: its operator has no zero columns between expansion and samples, which
would move the samples to other MMA steps.  The limits are the errors without them on the same inputs
(rel-L2 2.54e-7, 2.33e-7, 2.56e-7) and 2%; with them 2.67e-7, 2.42e-7, 2.71e-7."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,P,T,b,limit", [(1 << 17, 32, 12, 4, 2.54e-7), (1 << 15, 2, 20, 4, 2.33e-7),
                                           (1 << 19, 256, 36, 4, 2.56e-7)])
def test_window_rows_keep_their_k_order(monkeypatch, N, P, T, b, limit):
    import torch
    import fmmfft
    monkeypatch.setenv("FMMFFT_AUTOTUNE", "0")  # the default routing
    gen = torch.Generator(device="cuda").manual_seed(1)
    x = torch.view_as_complex(torch.randn(N, 2, generator=gen, device="cuda"))
    plan = fmmfft.Plan(N, P, T, b, "f32_tc")
    assert "leaf_form=window_rows" in plan.describe(), plan.describe()
    y = plan(x).to(torch.complex128)
    plan.close()
    want = torch.fft.fft(x.to(torch.complex128))
    assert float((y - want).norm() / want.norm()) <= 1.02 * limit
