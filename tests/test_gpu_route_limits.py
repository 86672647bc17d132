"""Kernels at ends of their range that the default shapes do not reach, each with its route asserted.

The shared-operand leaf with one stage of shared memory (36 to 48 terms at b = 32; up to 32 terms two fit):
one tile and several a block, one and several strips, a batch.  FP64 row contractions for sections above 1024
points (smaller ones run whole in one block): terms that are no multiple of 4 or 8, one to four column tiles,
P = 2 with fewer rows than a warp's tiles.  The coarse levels in one launch with 32 to 52 terms, FP32 and
FP64.  Against the FP64 oracle of the same terms: FP64 <= 1e-12 at every stage; FP32 <= 1e-6, expansions and
field <= 1e-5, as at fewer terms; transforms of a batch have the bits of each alone."""
import numpy as np
import pytest

import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fm():
    import fmmfft
    fmmfft.load()
    return fmmfft


def check(fm, plan, nbt):
    """All transforms of a batch and each alone; the expansions and field of the first."""
    import torch
    N, P, T, b, prec = plan.N, plan.P, plan.terms, plan.b, plan.precision
    xs = [ol.seeded_input(N, 20 + i) for i in range(nbt)]
    x = torch.from_numpy(np.concatenate(xs)).to(torch.complex128 if prec == "f64" else torch.complex64).cuda()
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
    tol, tol_stage = (1e-12, 1e-12) if prec == "f64" else (1e-6, 1e-5)
    o = ol.forward_ex(xs[0], P, T, b)
    assert ol.rel_l2(y[:N].cpu().numpy(), o["y"]) < tol
    n = (N // P // b).bit_length() - 1
    for lev in range(2, n + 1):
        for name in ("phi", "psi"):
            g = fm.level_planar(d[name], P, T, n, lev)
            g = (g[:, 0] + 1j * g[:, 1]).transpose(1, 0, 2)
            assert ol.rel_l2(g, o[name][ol.level_slice(lev)]) < tol_stage, (name, lev)
    assert ol.rel_l2(d["u"], o["u"]) < tol_stage


@pytest.mark.parametrize("N,P,T,b,stages", [(1 << 13, 2, 36, 32, 1), (1 << 17, 8, 48, 32, 1), (1 << 20, 64, 40, 32, 1),
                                            (1 << 18, 16, 44, 32, 1), (1 << 17, 8, 32, 32, 2)])
def test_leaf_stages(fm, monkeypatch, N, P, T, b, stages):
    monkeypatch.setenv("FMMFFT_AUTOTUNE", "0")  # the default routing
    plan = fm.Plan(N, P, T, b, "f32_tc", max_transforms=2)
    assert f"leaf_form=shared_operands leaf_stages={stages} " in plan.describe(), plan.describe()
    check(fm, plan, 2)


@pytest.mark.parametrize("N,P,T,b", [(1 << 16, 8, 15, 16), (1 << 15, 8, 9, 8), (1 << 17, 8, 31, 16), (1 << 12, 2, 15, 32),
                                     (1 << 12, 2, 4, 64), (1 << 16, 16, 23, 64)])
def test_f64_rows(fm, N, P, T, b):
    plan = fm.Plan(N, P, T, b, "f64", max_transforms=3)
    assert "s2m=rows" in plan.describe(), plan.describe()
    check(fm, plan, 3)


@pytest.mark.parametrize("N,P,T,b,prec", [(1 << 17, 8, 40, 32, "f32"), (1 << 17, 4, 46, 16, "f32"), (1 << 18, 8, 52, 32, "f32_tc"),
                                          (1 << 17, 8, 33, 64, "f32"), (1 << 16, 8, 32, 32, "f64")])
def test_coarse_levels_of_many_terms(fm, monkeypatch, N, P, T, b, prec):
    monkeypatch.setenv("FMMFFT_AUTOTUNE", "0")
    plan = fm.Plan(N, P, T, b, prec, max_transforms=2)
    levels = (N // P // b).bit_length() - 1
    x = np.zeros(N, plan.complex_dtype)
    plan.profile_start(1)
    plan.execute_host(x)
    _, stages = plan.profile_stop()
    assert stages["coarse_tree"][1] == 1 and stages["m2l_l2l"][1] < levels - 2, stages  # some levels in its launch
    check(fm, plan, 2)
