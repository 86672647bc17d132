"""FP32 FFT passes with two sequences a thread (k_fft_pair): their 16-byte accesses to the user's arrays need
an address of 16 bytes, complex64 pointers need only 8.  The same transform from and to arrays one
element off must give the same bits (the same sums, other accesses), for passes in both orders and every
kind of first stage, the plain FFT and the FMM-FFT; against the FP64 FFT <= 1e-6, the FP32 tolerance."""
import numpy as np
import pytest

import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fm():
    import fmmfft
    fmmfft.load()
    return fmmfft


def _both(run, x, torch):
    s = torch.cuda.current_stream().cuda_stream
    n = x.numel()
    y, far = torch.empty_like(x), torch.zeros(n + 1, dtype=x.dtype, device="cuda")
    run(x.data_ptr(), y.data_ptr(), s)
    src = torch.cat([x[:1], x])
    assert src[1:].data_ptr() % 16 == 8
    run(src[1:].data_ptr(), far[1:].data_ptr(), s)
    torch.cuda.synchronize()
    assert torch.equal(y, far[1:]) and far[0] == 0
    return y.cpu().numpy().astype(np.complex128)


@pytest.mark.parametrize("lg", [13, 14, 16, 17, 19, 20, 22, 23])
def test_plain_fft_one_element_off(fm, lg):
    import torch
    x = ol.seeded_input(1 << lg, lg)
    f = fm.PlainFFT(1 << lg, "f32")
    y = _both(f.execute_ptr, torch.from_numpy(x).to(torch.complex64).cuda(), torch)
    f.close()
    assert ol.rel_l2(y, np.fft.fft(x)) < 1e-6


@pytest.mark.parametrize("N,P,T,b", [(1 << 14, 16, 16, 16), (1 << 18, 32, 20, 32), (1 << 19, 64, 20, 32), (1 << 20, 512, 16, 16)])
def test_transform_one_element_off(fm, N, P, T, b):
    import torch
    x = ol.seeded_input(N, 7)
    plan = fm.Plan(N, P, T, b, "f32")
    y = _both(plan.execute_ptr, torch.from_numpy(x).to(torch.complex64).cuda(), torch)
    plan.check()
    plan.close()
    assert ol.rel_l2(y, ol.forward(x, P, T, b)) < 1e-6
