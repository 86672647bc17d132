"""FP64 plans' row contractions on the matrix instructions, and the wide-box S2M and leaf.

The row kernels (S2M, M2M, M2L + L2L, leaf for b 8 to 64 and at most 32 terms) work on tiles of 8 rows
and 8 columns with K in steps of 4: terms that are no multiple of 4 or 8 (padded K, padded columns,
unpaired stores), one to four column tiles and the two column groups of b = 64, fewer rows than a
warp's tiles, the half-shifted first points (sc > P/2, = P/2, P = 2), batches.  The wide kernels take
b >= 128 where few blocks would run: the smallest width, a window of several shared tiles, terms
above and below the shares' rounding.  Against the FP64 oracle at every stage: rel-L2 <= 1e-12, the
FP64 plans' tolerance (sums of at most 3b + T terms in FP64, errors ~1e-15)."""
import numpy as np
import pytest

import oracle_lib as ol

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.fixture(scope="module")
def fm():
    import fmmfft
    fmmfft.load()
    return fmmfft


CASES = [(64, 2, 4, 8), (256, 4, 9, 16), (2048, 8, 15, 8), (8192, 2, 17, 32), (8192, 16, 31, 16), (16384, 8, 32, 64),
         (32768, 32, 24, 8), (65536, 4, 5, 64), (1 << 17, 64, 20, 32),
         (2048, 4, 7, 128), (16384, 2, 33, 512), (65536, 4, 16, 2048)]


@pytest.mark.parametrize("N,P,T,b", CASES)
def test_f64_rows_and_wide_boxes_match_oracle(fm, N, P, T, b):
    import torch
    xs = [ol.seeded_input(N, 60 + i) for i in range(3)]
    plan = fm.Plan(N, P, T, b, "f64", max_transforms=3)
    x = torch.from_numpy(np.concatenate(xs)).cuda()
    y = torch.empty_like(x)
    plan.execute_many_ptr(3, x.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    plan.check()
    d = plan.debug_fetch()
    plan.close()
    got = y.cpu().numpy().reshape(3, N)
    for i in range(3):
        assert ol.rel_l2(got[i], ol.forward(xs[i], P, T, b)) < TOL, i
    o = ol.forward_ex(xs[0], P, T, b)
    n = (N // P // b).bit_length() - 1
    for lev in range(2, n + 1):
        for name in ("phi", "psi"):
            g = fm.level_planar(d[name], P, T, n, lev)
            g = (g[:, 0] + 1j * g[:, 1]).transpose(1, 0, 2)
            assert ol.rel_l2(g, o[name][ol.level_slice(lev)]) < TOL, (name, lev)
    assert ol.rel_l2(d["u"], o["u"]) < TOL
