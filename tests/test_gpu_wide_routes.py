"""Which kernel makes the leaf multipoles of wide boxes (b >= 128), and its results.

The wide kernel (a block a row) is for few rows: its time grows with rows times b while the row contraction's
is constant until its blocks fill the device, so plans change over at 24 b rows, and tensor-core plans from
4096 rows keep the tensor cores.  Each shape lies near a limit: rows 4032 against 3072 (b = 128), 1984
against 3072 and 6144, 8064 on the tensor cores.  Against the FP64 oracle of the same terms: rel-L2 <= 1e-12
(FP64) and 1e-6 (FP32), the tolerances of the plans' other tests; a batch of two has the bits of each alone.
P = 2 and b = 1024: the operator fits beside the sections tile up to 20 terms (FP64; FP32 48), not above."""
import numpy as np
import pytest

import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fm():
    import fmmfft
    fmmfft.load()
    return fmmfft


@pytest.mark.parametrize("N,P,T,b,prec,route", [
    (1 << 19, 64, 16, 128, "f32_tc", "tensor_cores"), (1 << 18, 64, 8, 128, "f32", "general"),
    (1 << 18, 64, 20, 128, "f64", "general"), (1 << 17, 32, 24, 128, "f32", "wide"),
    (1 << 18, 32, 7, 256, "f64", "wide"), (1 << 18, 32, 12, 256, "f32_tc", "wide"),
    (1 << 14, 2, 24, 1024, "f64", "wide"), (1 << 14, 2, 56, 1024, "f32", "wide"), (1 << 13, 2, 20, 1024, "f64", "fused")])
def test_wide_box_multipoles(fm, monkeypatch, N, P, T, b, prec, route):
    import torch
    monkeypatch.setenv("FMMFFT_AUTOTUNE", "0")  # the default routing
    ct = np.complex128 if prec == "f64" else np.complex64
    xs = [ol.seeded_input(N, 90 + i).astype(ct) for i in range(2)]
    plan = fm.Plan(N, P, T, b, prec, max_transforms=2)
    assert "s2m=" + route + " " in plan.describe(), plan.describe()
    x = torch.from_numpy(np.concatenate(xs)).cuda()
    y, z = torch.empty_like(x), torch.empty_like(x)
    st = torch.cuda.current_stream().cuda_stream
    plan.execute_many_ptr(2, x.data_ptr(), y.data_ptr(), st)
    for i in range(2):
        plan.execute_ptr(x[i * N:].data_ptr(), z[i * N:].data_ptr(), st)
    torch.cuda.synchronize()
    plan.check()
    plan.close()
    assert torch.equal(y, z)
    want = ol.forward(xs[0].astype(np.complex128), P, T, b)
    assert ol.rel_l2(y[:N].cpu().numpy(), want) <= (1e-12 if prec == "f64" else 1e-6)
