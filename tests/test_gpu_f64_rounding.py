"""Rounding of FP64 plans against the exact transform, near the format's resolution.

The leaf adds the box's own samples, whose weights reach P / pi, after everything else: added earlier, every
later product is rounded at their size.  The limit is the error of the direct leaf kernel, whose place the row
contractions take, on the same inputs (rel-L2 7.78e-16, 7.43e-16, 7.86e-16, 8.42e-16 against an FFT in 80
bits) and 2%.  With the box's own samples before the last neighbour's it is 4 to 11% higher."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,P,T,b,limit", [(1 << 16, 32, 16, 64, 7.78e-16), (1 << 15, 16, 24, 64, 7.43e-16),
                                           (1 << 21, 64, 24, 64, 7.86e-16), (1 << 16, 16, 16, 32, 8.42e-16)])
def test_leaf_order_keeps_the_rounding(N, P, T, b, limit):
    import torch
    import fmmfft
    gen = torch.Generator(device="cuda").manual_seed(1)
    x = torch.view_as_complex(torch.randn(N, 2, generator=gen, device="cuda", dtype=torch.float64))
    plan = fmmfft.Plan(N, P, T, b, "f64")
    y = plan(x).cpu().numpy()
    plan.close()
    want = np.fft.fft(x.cpu().numpy().astype(np.clongdouble))
    assert want.dtype == np.clongdouble
    assert np.linalg.norm((y - want).astype(np.complex128)) <= 1.02 * limit * np.linalg.norm(want.astype(np.complex128))
