"""Small sections run whole in one block (k_tree): sections of 4 boxes up to the most that shared memory
holds, terms that are no multiple of the tiles (padded rows and columns, unpaired stores, one column
group), P = 2 and the section sc = P/2 (the mean of two first points), more sections than the device
has block slots.  Two forms of the kernel: a few blocks with every operator in shared memory and small
tiles, or blocks that fill the device with larger tiles and one operator at a time; their bits must
agree, so each transform of a batch large enough for the second is compared with its own execute.
Against the FP64 oracle: rel-L2 <= 1e-12 (FP64) and <= 1e-6 (FP32), the plans' tolerances; the FP32
stages <= 1e-5 (sums of at most 3b + T products, each rounded to 2^-24 of O(P / pi) weights)."""
import numpy as np
import pytest

import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fm():
    import fmmfft
    fmmfft.load()
    return fmmfft


# (N, P, T, b); n = 2 .. 7
CASES = [(64, 2, 3, 8), (512, 4, 9, 16), (512, 2, 16, 64), (2048, 8, 10, 16), (2048, 2, 17, 32), (1 << 14, 16, 20, 32),
         (1 << 15, 8, 24, 64), (1 << 15, 1024, 12, 8), (1 << 17, 128, 13, 8), (1 << 18, 64, 20, 32)]


@pytest.mark.parametrize("prec", ["f64", "f32", "f32_tc"])
@pytest.mark.parametrize("N,P,T,b", CASES)
def test_whole_sections_match_oracle_alone_and_in_batches(fm, N, P, T, b, prec):
    import torch
    dt = torch.complex128 if prec == "f64" else torch.complex64
    nbt = max(2, min(64, 320 // P + 1))  # P nbt > 2 x 148 blocks where 64 transforms allow
    xs = [ol.seeded_input(N, 90 + i) for i in range(nbt)]
    plan = fm.Plan(N, P, T, b, prec, max_transforms=nbt)
    if prec != "f64":
        assert "sections=one_block" in plan.describe(), plan.describe()
    x = torch.from_numpy(np.concatenate(xs)).to(dt).cuda()
    y, alone, inv = torch.empty_like(x), torch.empty_like(x), torch.empty_like(x[:N])
    s = torch.cuda.current_stream().cuda_stream
    plan.execute_many_ptr(nbt, x.data_ptr(), y.data_ptr(), s)
    for i in range(nbt):
        plan.execute_ptr(x[i * N:].data_ptr(), alone[i * N:].data_ptr(), s)
    plan.execute_ptr(x.data_ptr(), inv.data_ptr(), s, inverse=True)
    plan.execute_ptr(x.data_ptr(), alone.data_ptr(), s)
    torch.cuda.synchronize()
    plan.check()
    d = plan.debug_fetch()
    plan.close()
    assert torch.equal(y, alone)
    tol, tol_stage = (1e-12, 1e-12) if prec == "f64" else (1e-6, 1e-5)
    got = y.cpu().numpy().astype(np.complex128).reshape(nbt, N)
    for i in (0, nbt - 1):
        assert ol.rel_l2(got[i], ol.forward(xs[i], P, T, b)) < tol, i
    o = ol.forward_ex(xs[0], P, T, b)
    n = (N // P // b).bit_length() - 1
    for lev in range(2, n + 1):
        for name in ("phi", "psi"):
            g = fm.level_planar(d[name], P, T, n, lev)
            g = (g[:, 0] + 1j * g[:, 1]).transpose(1, 0, 2)
            assert ol.rel_l2(g, o[name][ol.level_slice(lev)]) < tol_stage, (name, lev)
    assert ol.rel_l2(d["u"], o["u"]) < tol_stage
    conj = np.conj(ol.forward(np.conj(xs[0]), P, T, b))  # the inverse: conj F conj
    assert ol.rel_l2(inv.cpu().numpy().astype(np.complex128), conj) < tol
