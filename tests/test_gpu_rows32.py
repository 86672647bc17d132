"""FP32 row contractions of the tree and leaf (k_rows_f32): tiles of 2, 4 or 8 rows a thread inside one
plane and over several whole planes (few boxes a plane, many sections), the last tile short, terms that
are no multiple of 4 (padded columns, unaligned rows, unpaired stores), every box width, P = 2 (the
section sc = P/2: the mean of two first points), S2M of its own where it is not fused.  A batch must have
the bits of its transforms alone.  The transform and u against the FP64 oracle: <= 1e-6, the FP32 plans'
tolerance, and <= 1e-5 (sums of at most 3b + T products, each rounded to 2^-24 of O(P / pi) weights).
The expansions against the general stage kernels (which FMMFFT_FUSE_S2M keeps) <= 1e-5: both sum the same
FP32 operators' products in another order; the operators' own rounding, common to both, grows with the
number of levels and shows against the oracle."""
import numpy as np
import pytest

import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fm():
    import fmmfft
    fmmfft.load()
    return fmmfft


# (N, P, T, b), sections too large for one block
CASES = [(1 << 17, 2, 5, 16), (1 << 18, 4, 3, 8), (1 << 18, 2, 24, 32), (1 << 18, 8, 13, 16), (1 << 19, 4, 30, 8),
         (1 << 19, 16, 17, 64), (1 << 20, 32, 20, 32), (1 << 20, 32, 32, 64), (1 << 20, 64, 8, 32)]


@pytest.mark.parametrize("N,P,T,b", CASES)
def test_rows_match_oracle_alone_and_in_a_batch(fm, monkeypatch, N, P, T, b):
    import torch
    monkeypatch.setenv("FMMFFT_AUTOTUNE", "0")  # the default routing
    xs = [ol.seeded_input(N, 50 + i) for i in range(3)]
    plan = fm.Plan(N, P, T, b, "f32", max_transforms=3)
    assert "sections=one_block" not in plan.describe(), plan.describe()
    x = torch.from_numpy(np.concatenate(xs)).to(torch.complex64).cuda()
    y, alone = torch.empty_like(x), torch.empty_like(x)
    s = torch.cuda.current_stream().cuda_stream
    plan.execute_many_ptr(3, x.data_ptr(), y.data_ptr(), s)
    for i in (2, 1, 0):
        plan.execute_ptr(x[i * N:].data_ptr(), alone[i * N:].data_ptr(), s)
    torch.cuda.synchronize()
    plan.check()
    d = plan.debug_fetch()  # of the last execute: transform 0
    plan.close()
    assert torch.equal(y, alone)
    monkeypatch.setenv("FMMFFT_FUSE_S2M", "1")
    general = fm.Plan(N, P, T, b, "f32")
    general.execute_ptr(x.data_ptr(), alone.data_ptr(), s)
    torch.cuda.synchronize()
    g = general.debug_fetch()
    general.close()
    for name in ("phi", "psi"):
        assert ol.rel_l2(d[name], g[name]) < 1e-5, name
    o = ol.forward_ex(xs[0], P, T, b)
    assert ol.rel_l2(d["u"], o["u"]) < 1e-5
    got = y.cpu().numpy().astype(np.complex128).reshape(3, N)
    assert ol.rel_l2(got[0], o["y"]) < 1e-6
    assert ol.rel_l2(got[2], ol.forward(xs[2], P, T, b)) < 1e-6


@pytest.mark.parametrize("prec,T,tol", [("f32_tc", 8, 1e-6), ("f32_tc", 16, 1e-6), ("f32_tc", 20, 1e-6), ("f32_tc", 24, 1e-6),
                                        ("bf16x3", 12, 1e-4), ("bf16x3", 24, 1e-4)])
def test_rows_beside_tensor_core_stages(fm, monkeypatch, prec, T, tol):
    """Tensor-core plans on both sides of the terms where S2M, M2M and M2L change units, their small levels
    as row contractions below the tensor cores' and above the coarse tree; the plans' accuracy classes."""
    import torch
    monkeypatch.setenv("FMMFFT_AUTOTUNE", "0")
    N, P, b = 1 << 20, 32, 32
    xs = [ol.seeded_input(N, 60 + i) for i in range(2)]
    plan = fm.Plan(N, P, T, b, prec, max_transforms=2)
    assert "leaf_form=shared_operands" in plan.describe(), plan.describe()
    x = torch.from_numpy(np.concatenate(xs)).to(torch.complex64).cuda()
    y, alone = torch.empty_like(x), torch.empty_like(x)
    s = torch.cuda.current_stream().cuda_stream
    plan.execute_many_ptr(2, x.data_ptr(), y.data_ptr(), s)
    for i in (1, 0):
        plan.execute_ptr(x[i * N:].data_ptr(), alone[i * N:].data_ptr(), s)
    torch.cuda.synchronize()
    plan.check()
    plan.close()
    assert torch.equal(y, alone)
    got = y.cpu().numpy().astype(np.complex128).reshape(2, N)
    for i in range(2):
        assert ol.rel_l2(got[i], ol.forward(xs[i], P, T, b)) < tol
