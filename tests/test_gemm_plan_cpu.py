"""The estimates by which a GEMM goes to a tile width or to a weight-streaming kernel (csrc/rules.h), compiled for the host and
checked against times measured on a B200 (us, fp16, one launch behind the other). 148 SMs."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_WRAPPERS = """
#include "rules.h"
using namespace b200ait;
extern "C" double tile_us(long long m, long long n, long long k, int e, int width) {
  return gemm_tile_us(GemmProblem{1, m, n, k, e, e, k, false}, width, 148);
}
extern "C" double swap_us(long long m, long long n, long long k, int e, int mx, int r) {
  return gemm_swap_us(GemmProblem{1, m, n, k, e, e, k, false}, mx, r, r == 2 ? 74 : r == 4 ? 33 : 15);
}
extern "C" int batched_width(long long b, long long m, long long n, long long k, int row_major, int pairs) {
  return gemm_best_width(GemmProblem{b, m, n, k, 0, 0, row_major ? 64 : k, row_major != 0, pairs != 0}, 148);
}
extern "C" int width_of(long long m, long long n, long long k, int e, int pairs) {
  return gemm_best_width(GemmProblem{1, m, n, k, e, e, k, false, pairs != 0}, 148);
}
extern "C" double batched_us(long long b, long long m, long long n, long long k, int row_major, int width) {
  return gemm_tile_us(GemmProblem{b, m, n, k, 0, 0, row_major ? 64 : k, row_major != 0}, width, 148);
}
extern "C" bool swap_in_range(long long m, long long units, int resident) { return gemm_swap_in_range(m, units, resident); }
extern "C" bool may_split(long long m, long long n, long long k) { return gemm_may_split(m, n, k); }
extern "C" int best_width(long long b, long long m, long long n, long long k, int e) {
  return gemm_best_width(GemmProblem{b, m, n, k, e, e, k, false}, 148);
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    work = tmp_path_factory.mktemp("plan")
    src, lib = work / "plan.cpp", work / "plan.so"
    src.write_text(_WRAPPERS)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-Wall", "-Werror", "-I",
                    os.path.join(ROOT, "aitemplate_b200", "csrc"), str(src), "-o", str(lib)], check=True)
    lib = ctypes.CDLL(str(lib))
    lib.tile_us.restype = lib.swap_us.restype = lib.batched_us.restype = ctypes.c_double
    lib.swap_in_range.restype = lib.may_split.restype = ctypes.c_bool
    return lib


def _ll(*v):
    return [ctypes.c_longlong(x) for x in v]


# times of the sweep that the estimates were fitted to, which they match to 5 % (root mean square); one problem may lie a few
# times that off
@pytest.mark.parametrize(
    "m,n,k,e,width,us",
    [
        (256, 2304, 768, 0, 128, 5.97), (1055, 768, 3072, 0, 64, 11.3), (2048, 1024, 4096, 0, 128, 17.1),
        (1055, 4096, 4096, 0, 256, 29.2), (1055, 4096, 4096, 0, 512, 43.9),
        (384, 2305, 768, 0, 64, 10.0), (1055, 2305, 768, 1, 128, 21.5), (384, 3000, 640, 0, 128, 5.75),
        (2048, 2048, 2040, 0, 512, 19.2), (2048, 2048, 2040, 0, 64, 43.6),
    ])
def test_tile_estimates(plan, m, n, k, e, width, us):
    got = plan.tile_us(*_ll(m, n, k), e, width)
    assert abs(got / us - 1) < 0.16, got


@pytest.mark.parametrize("m,n,k,e,mx,r,us", [(1055, 256, 2048, 0, 32, 2, 7.1), (1055, 512, 8192, 0, 64, 2, 14.95),
                                            (130, 769, 768, 0, 16, 2, 6.97), (384, 2305, 768, 0, 32, 2, 22.5)])
def test_weight_streaming_estimates(plan, m, n, k, e, mx, r, us):
    got = plan.swap_us(*_ll(m, n, k), e, mx, r)
    assert abs(got / us - 1) < 0.2, got


@pytest.mark.parametrize(
    "batch,m,n,k,e,width",
    [
        (1, 24576, 3072, 768, 2, 512), (1, 8192, 8192, 8192, 0, 512),  # many tiles, deep K: pairs
        (1, 1055, 4096, 4096, 0, 256),                                # one wave of single tiles, two of pairs
        (1, 512, 3072, 768, 2, 128), (1, 1055, 768, 3072, 0, 64),      # few tiles
        (1, 384, 3000, 640, 0, 128),                                  # rows that are not whole sectors
        (1, 300, 200, 512, 0, 128),                                   # (no pair tile is wider than the result)
        (1, 2048, 2048, 2040, 0, 512),                                # rows off every 32-byte boundary: as few copies as can be
        (1, 625, 368, 320, 0, 128), (1, 458, 368, 384, 2, 128),       # a chunk of 32 columns that the edge cuts
    ])
def test_widths(plan, batch, m, n, k, e, width):
    assert plan.best_width(*_ll(batch, m, n, k), e) == width


@pytest.mark.parametrize("m,n,taken", [(2048, 8192, True), (2049, 128, True), (4096, 128, True), (4800, 128, False), (8192, 640, False)])
def test_weight_streaming_of_many_rows_is_one_wave(plan, m, n, taken):
    """No K in parts from 128 columns on, so whatever splitting was for has to be in reach of the kernel that takes its place."""
    assert not plan.may_split(*_ll(m, n, 8192))
    units = -(-m // 64) * -(-n // 128)
    assert plan.swap_in_range(*_ll(m, units), 74) == taken
    if taken and m > 2048:
        assert plan.swap_us(*_ll(m, n, 8192), 0, 64, 2) < 0.97 * min(plan.tile_us(*_ll(m, n, 8192), 0, w) for w in (64, 128, 256, 512))


@pytest.mark.parametrize("m,n,k,split", [(4, 8192, 8192, False), (4, 8192, 20488, True), (2, 64, 40960, False), (2, 64, 40968, True),
                                          (1, 63, 4096, True), (5, 127, 4096, True), (5, 128, 4096, False), (3, 64, 1016, True)])
def test_where_k_may_be_split(plan, m, n, k, split):
    assert plan.may_split(*_ll(m, n, k)) == split


# times of products with every width forced (us: 64, 128, 256, 512), at which the estimate of single products chose the slowest but one
@pytest.mark.parametrize(
    "b,m,n,k,row_major,us",
    [
        (78, 160, 80, 72, 1, (11.9, 5.6, 8.2, 8.1)), (159, 131, 176, 40, 1, (17.4, 11.2, 12.0, 11.1)),
        (285, 374, 136, 88, 0, (34.5, 22.4, 17.9, 19.8)), (445, 295, 392, 40, 0, (89.8, 50.9, 39.8, 49.8)),
        (101, 202, 144, 328, 0, (17.4, 12.2, 9.7, 8.9)), (183, 69, 112, 352, 1, (14.3, 7.3, 10.3, 12.4)),
        (892, 48, 216, 88, 0, (70.7, 19.6, 16.6, 22.4)), (19, 151, 624, 816, 1, (15.4, 11.6, 11.2, 10.5)),
        (706, 133, 64, 40, 1, (13.3, 17.8, 26.1, 24.8)), (80, 1006, 632, 648, 0, (188.5, 111.7, 97.0, 81.6)),
    ])
def test_batched_widths(plan, b, m, n, k, row_major, us):
    width = plan.batched_width(*_ll(b, m, n, k), row_major, 1)
    assert us[(64, 128, 256, 512).index(width)] <= 1.1 * min(us)
    assert plan.batched_width(*_ll(b, m, n, k), row_major, 0) != 512
    for w, t in zip((64, 128, 256, 512), us):
        assert abs(plan.batched_us(*_ll(b, m, n, k), row_major, w) / t - 1) < 0.45, w


@pytest.mark.parametrize("m,n,k,width", [(829, 6824, 216, 128), (2075, 2816, 160, 128), (8144, 768, 200, 128), (3572, 1808, 128, 128)])
def test_short_k_without_pairs(plan, m, n, k, width):
    """Epilogues without an instantiation of their own: two residuals, measured with every width forced."""
    assert plan.width_of(*_ll(m, n, k), 1, 1) == 512
    assert plan.width_of(*_ll(m, n, k), 1, 0) == width
