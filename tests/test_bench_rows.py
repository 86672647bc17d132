"""The levels that bench.py's roofline counts to the coarse-tree launch follow the plan's own threshold."""
import sys

import pytest

import oracle_lib as ol

sys.path.insert(0, ol.REPO)


@pytest.fixture(scope="module")
def bench():
    argv = sys.argv
    sys.argv = ["bench.py"]
    try:
        import bench as b
    finally:
        sys.argv = argv
    return b


@pytest.mark.parametrize("text,rows", [
    ("fft_threads=512 coarse_rows=1024 fuse_s2m=1 s2m=rows tuned=0", 1024),
    ("fft_threads=512 coarse_rows=2048 tc_min_rows=4096 fuse_s2m=1 tensor_cores=none tuned=0", 2048),
    ("fft_threads=512 coarse_rows=8192 tc_min_rows=1024 fuse_s2m=1 tensor_cores=none tuned=1", 8192),
    ("fft_threads=512 coarse_rows=8192 tc_min_rows=1024 fuse_s2m=1 tensor_cores=tf32x3 tuned=1", 1024)])
def test_coarse_rows_of_a_description(bench, text, rows):
    assert bench.coarse_rows(text) == rows


def test_levels_move_between_launches(bench):
    N, P, T, b = 1 << 24, 64, 24, 32
    lv = lambda l: 2 * (P - 1) * T * (1 << l) * 4
    old, new = bench.stage_bytes(N, P, T, b, 8, 4096), bench.stage_bytes(N, P, T, b, 8, 2048)
    # 126 planes: M2M parents of level 4 (2016 rows) stay, of level 5 (4032 rows) leave the coarse launch
    assert new["m2m"] - old["m2m"] == lv(6) + lv(5)
    assert new["m2l_l2l"] - old["m2l_l2l"] == lv(5) + 2 * lv(6)  # its child level 6
    tree = ("m2m", "coarse_tree", "m2l_l2l")
    assert sum(new[k] for k in tree) == sum(old[k] for k in tree)
    assert all(new[k] == old[k] for k in new if k not in tree)
