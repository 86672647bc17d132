"""When a plan runs its sections whole in one block (k_tree) and when in stages, and one block with more than
32 terms.

FP32 plans take one block where the P sections of one transform are on the 148 SMs at once, by the shared
memory of a block, above 512 sections only up to 32 points each; twice as many sections of any number with
33 to 44 terms; FP64 plans up to 1024 points a section.  The shapes lie on both sides of each limit.  A BF16x3 plan
whose sections would fit a block computes in FP32 in either form: in stages with the bits of an FP32 plan.  Results: terms 33 to 64 (padded and whole rows), one block an
SM (512 threads however many sections run) and several, a batch of more blocks than the device holds
against each transform alone (same bits), the transform against the FP64 oracle <= 1e-6, the stages <=
1e-5, as for fewer terms."""
import numpy as np
import pytest

import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fm():
    import fmmfft
    fmmfft.load()
    return fmmfft


@pytest.mark.parametrize("M,P,T,b,prec,one_block", [
    (4096, 512, 24, 32, "f32_tc", False), (2048, 512, 24, 16, "f32", False), (1024, 512, 16, 32, "f32_tc", True),
    (4096, 256, 24, 32, "f32_tc", False), (4096, 256, 16, 16, "bf16x3", False), (2048, 256, 16, 32, "f32", True),
    (256, 1024, 33, 32, "f32_tc", True), (256, 1024, 40, 64, "f32", False), (128, 256, 64, 16, "f32", False), (128, 128, 64, 16, "f32_tc", True), (64, 256, 64, 16, "f32", True),
    (4096, 128, 24, 32, "f32_tc", True), (8192, 64, 16, 64, "f32", True), (2048, 256, 33, 32, "f32_tc", True),
    (64, 1024, 8, 8, "f32_tc", False), (256, 1024, 24, 32, "f32_tc", False), (32, 1024, 12, 8, "f32", True),
    (1024, 1024, 8, 32, "f64", True), (2048, 64, 8, 32, "f64", False)])
def test_route(fm, M, P, T, b, prec, one_block):
    plan = fm.Plan(M * P, P, T, b, prec)
    text = plan.describe()
    plan.close()
    assert ("sections=one_block" in text) == one_block, text


@pytest.mark.parametrize("M,P,T,b", [(64, 1024, 12, 8), (256, 1024, 8, 32), (2048, 512, 16, 16)])
def test_bf16x3_stages_of_small_sections_in_fp32(fm, monkeypatch, M, P, T, b):
    import torch
    monkeypatch.setenv("FMMFFT_AUTOTUNE", "0")  # the default routing of both plans
    x = torch.from_numpy(ol.seeded_input(M * P, 7)).to(torch.complex64).cuda()
    out = []
    for prec in ("bf16x3", "f32"):
        plan = fm.Plan(M * P, P, T, b, prec)
        assert "sections=one_block" not in plan.describe(), plan.describe()
        out.append(plan(x))
        plan.check()
        plan.close()
    assert torch.equal(*out)


# (N, P, T, b, transforms)
@pytest.mark.parametrize("N,P,T,b,nbt", [(1 << 12, 8, 64, 32, 41), (1 << 12, 4, 33, 32, 3), (1 << 13, 8, 40, 16, 41),
                                         (1 << 15, 32, 47, 64, 11), (1 << 9, 2, 50, 8, 3), (1 << 18, 128, 33, 32, 3)])
@pytest.mark.parametrize("prec", ["f32", "f32_tc"])
def test_many_terms_in_one_block(fm, N, P, T, b, nbt, prec):
    import torch
    xs = [ol.seeded_input(N, 40 + i) for i in range(nbt)]
    plan = fm.Plan(N, P, T, b, prec, max_transforms=nbt)
    assert "sections=one_block" in plan.describe(), plan.describe()
    x = torch.from_numpy(np.concatenate(xs)).to(torch.complex64).cuda()
    y, alone = torch.empty_like(x), torch.empty_like(x)
    s = torch.cuda.current_stream().cuda_stream
    plan.execute_many_ptr(nbt, x.data_ptr(), y.data_ptr(), s)
    for i in reversed(range(nbt)):
        plan.execute_ptr(x[i * N:].data_ptr(), alone[i * N:].data_ptr(), s)
    torch.cuda.synchronize()
    plan.check()
    d = plan.debug_fetch()
    plan.close()
    assert torch.equal(y, alone)
    o = ol.forward_ex(xs[0], P, T, b)
    assert ol.rel_l2(y[:N].cpu().numpy(), o["y"]) < 1e-6
    n = (N // P // b).bit_length() - 1
    for lev in range(2, n + 1):
        for name in ("phi", "psi"):
            g = fm.level_planar(d[name], P, T, n, lev)
            g = (g[:, 0] + 1j * g[:, 1]).transpose(1, 0, 2)
            assert ol.rel_l2(g, o[name][ol.level_slice(lev)]) < 1e-5, (name, lev)
    assert ol.rel_l2(d["u"], o["u"]) < 1e-5
