"""The launch-shape rules of csrc/nk_launch_rules.h, compiled for the host (no GPU needed)."""
import ctypes as C
import os
import subprocess

import pytest

HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "neureka_b200", "csrc", "nk_launch_rules.h")
SOURCE = """
#include "%s"
extern "C" void dgemm_parts(int64_t tiles, int64_t k_panels, int64_t sms, int64_t* out) {
    const NkDgemmParts p = nk_dgemm_parts(tiles, k_panels, sms);
    out[0] = p.splits;
    out[1] = p.kb_per;
}
extern "C" int sum_by_groups(int64_t tiles, int merged_dims, int64_t sms) { return nk_sum_by_groups(tiles, merged_dims, sms); }
extern "C" int64_t sum_last() { return NK_SUM_LAST; }
extern "C" int grad_form(int64_t vectors, int64_t positions, int64_t sms) { return nk_fused_grad_form(vectors, positions, sms); }
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    src, lib = d / "rules.cpp", d / "librules.so"
    src.write_text(SOURCE % HEADER)
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-fPIC", "-shared", "-o", str(lib), str(src)], check=True)
    return C.CDLL(str(lib))


def dgemm_parts(rules, m, k, n, sms=148):
    out = (C.c_int64 * 2)()
    tiles = -(-m // 64) * -(-n // 64)
    rules.dgemm_parts(C.c_int64(tiles), C.c_int64(-(-k // 16)), C.c_int64(sms), out)
    return tiles, int(out[0]), int(out[1])


@pytest.mark.parametrize("mkn", [(4096, 4096, 4096), (6000, 6000, 6000), (8192, 8192, 8192), (16384, 16384, 16384), (16384, 4096, 16384),
                                 (40000, 2048, 40000), (49152, 2048, 49152), (3000, 100000, 3000)])
def test_large_f64_products_need_no_scratch_for_parts(rules, mkn):
    """Products with many tiles fill the chip by themselves: splitting k would write and read back 64 KB per part."""
    tiles, splits, kb_per = dgemm_parts(rules, *mkn)
    assert splits == 1 and kb_per * 16 >= mkn[1]


def test_parts_of_f64_products_are_bounded_and_cover_k(rules):
    for m in (64, 200, 777, 1536, 2048, 3000, 10000, 50000):
        for n in (64, 515, 1280, 2048, 9000):
            for k in (16, 100, 1023, 4096, 20000, 1 << 20, (1 << 33) + 5):
                for sms in (1, 132, 148):
                    tiles, splits, kb_per = dgemm_parts(rules, m, k, n, sms)
                    panels = -(-k // 16)
                    assert 1 <= splits <= 16 and (splits - 1) * kb_per < panels <= splits * kb_per    # every part has work
                    assert splits == 1 or tiles * splits * 32768 <= 64 << 20


def test_few_tiles_and_a_long_sum_are_split(rules):
    assert dgemm_parts(rules, 64, 20000, 64)[1] == 16
    assert dgemm_parts(rules, 777, 1023, 515)[1] > 1


def test_form_of_a_fused_gradient(rules):
    """Nothing or little summed: no form that evaluates positions it does not add; many vectors: vectors at any depth."""
    ONE, VEC, STEPS = 0, 1, 2

    def form(vectors, positions):
        return rules.grad_form(C.c_int64(vectors), C.c_int64(positions), C.c_int64(148))
    for positions in (1, 2, 3, 4):
        assert form(0, positions) == ONE and form(1000, positions) == ONE and form(100_000, positions) == VEC
    for positions in (5, 7, 8, 9, 1000):
        assert form(0, positions) == STEPS and form(100_000, positions) == (STEPS if positions >= 8 else VEC)
    assert all(form(1 << 20, positions) == VEC for positions in (1, 4, 5, 9, 1000))


def test_sums_of_views_go_by_groups_only_where_groups_fill_the_chip(rules):
    rules.sum_last.restype = C.c_int64
    assert rules.sum_last() == 32 * 128                  # a tile per warp of one CTA
    for dims in range(0, 9):
        for n in (8192, 16385, 300_000, 1_000_000, 1 << 21, 8_000_000):
            assert not rules.sum_by_groups(C.c_int64(-(-n // 128)), C.c_int(dims), C.c_int64(148)), (n, dims)
        assert rules.sum_by_groups(C.c_int64((1 << 25) // 128), C.c_int(dims), C.c_int64(148))
