"""The split-TF32 leaf with both operands in shared memory (k_tc_ss): tiles of 128 boxes with a halo box on
either side.  Sections of one tile (both halo boxes wrap) and of several, terms that are no multiple of
the K step (zero columns between expansion and samples), one and several producer warps a chunk quad, one
stage of shared memory instead of two, P = 2 (its only section is sc = P/2: the mean of two first
points), sections below and above P/2, and a batch.  u against the FP64 oracle <= 1e-5 and the transform
<= 1e-6, the split-TF32 tolerances of the other leaf forms; a batch has the bits of its transforms alone."""
import numpy as np
import pytest

import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fm():
    import fmmfft
    fmmfft.load()
    return fmmfft


# (N, P, T, b): boxes a section N / P / b
CASES = [(1 << 11, 2, 8, 8), (1 << 13, 2, 12, 32), (1 << 14, 4, 4, 16), (1 << 15, 8, 20, 8), (1 << 17, 32, 28, 32),
         (1 << 18, 64, 32, 32), (1 << 20, 256, 24, 32), (1 << 20, 8, 20, 32)]


@pytest.mark.parametrize("N,P,T,b", CASES)
def test_leaf_matches_oracle_alone_and_in_a_batch(fm, monkeypatch, N, P, T, b):
    import torch
    monkeypatch.setenv("FMMFFT_FUSE_S2M", "0")  # small sections too take the stage kernels
    xs = [ol.seeded_input(N, 70 + i) for i in range(3)]
    plan = fm.Plan(N, P, T, b, "f32_tc", max_transforms=3)
    assert "leaf_form=shared_operands" in plan.describe(), plan.describe()
    x = torch.from_numpy(np.concatenate(xs)).to(torch.complex64).cuda()
    y, alone = torch.empty_like(x), torch.empty_like(x)
    s = torch.cuda.current_stream().cuda_stream
    plan.execute_many_ptr(3, x.data_ptr(), y.data_ptr(), s)
    for i in (2, 1, 0):
        plan.execute_ptr(x[i * N:].data_ptr(), alone[i * N:].data_ptr(), s)
    torch.cuda.synchronize()
    plan.check()
    u = plan.debug_fetch()["u"]  # of the last execute: transform 0
    plan.close()
    assert torch.equal(y, alone)
    o = ol.forward_ex(xs[0], P, T, b)
    assert ol.rel_l2(u, o["u"]) < 1e-5
    got = y.cpu().numpy().astype(np.complex128).reshape(3, N)
    assert ol.rel_l2(got[0], o["y"]) < 1e-6
    assert ol.rel_l2(got[2], ol.forward(xs[2], P, T, b)) < 1e-6
