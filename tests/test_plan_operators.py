"""Device bytes of a plan's operators on the host (no GPU): fmmfft_plan_bytes of one transform less what each
further transform adds.  A form of an operator that no kernel of the plan reads takes no room."""
import os

import pytest

import oracle_lib as ol  # noqa: F401  (puts the package on sys.path)


@pytest.fixture(scope="module")
def fm():
    import fmmfft
    if not os.path.exists(fmmfft.LIB_PATH):
        import build_lib  # fmm-fft_b200/build_lib.py
        build_lib.build()
    fmmfft.load()
    return fmmfft


def operators(fm, N, P, T, b, prec):
    one, two = fm.plan_bytes(N, P, T, b, prec), fm.plan_bytes(N, P, T, b, prec, 2)
    return 2 * one - two


@pytest.mark.parametrize("N,P,T,b", [(1 << 24, 256, 24, 32), (1 << 22, 64, 20, 32), (1 << 24, 256, 16, 16)])
@pytest.mark.parametrize("prec", ["f32_tc", "bf16x3"])
def test_shared_operand_leaf_has_one_image(fm, N, P, T, b, prec):
    """Per section: the leaf's image (hi and lo of (T + 3 b) x (b + 1), padded to 8 and 16), the tables it is
    made from (T b, 4 b) and the first points' (T).  The rest: the size-M twiddles, and per level a tree
    operator of 10 T^2 in the forms of both kinds of kernel, below 40 values each."""
    S1, M, T8, b16 = P - 1, N // P, (T + 7) // 8 * 8, (b + 16) // 16 * 16
    section = 4 * (2 * (T8 + 3 * b) * b16 + T * b + 4 * b + T)
    levels = (M // b).bit_length()
    rest = 8 * M + 4 * 40 * 10 * T * T * levels + (64 << 10)
    assert operators(fm, N, P, T, b, prec) <= S1 * section + rest
