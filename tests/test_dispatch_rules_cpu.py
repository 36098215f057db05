"""The rules that pick one form of a kernel or another by size alone (csrc/rules.h), compiled for the host and checked at
the sizes where each form was measured to be the faster one. 148 SMs throughout."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SMS = 148

_WRAPPERS = """
#include "rules.h"
extern "C" bool attn_lone(long long items, int sms) { return b200ait::attn_lone(items, sms); }
extern "C" bool attn_item_per_cta(long long heads, long long seqs, long long bound, long long mean, int causal, int lengths,
                                  int d, int sms) {
  const int q_blocks = static_cast<int>((bound + 127) / 128), kv_blocks = static_cast<int>((bound + 63) / 64);
  return b200ait::attn_item_per_cta({heads * seqs * q_blocks, q_blocks, kv_blocks, causal != 0, lengths != 0, mean, bound, d}, sms);
}
extern "C" long long attn_longest_share(long long items, int q_blocks, int kv_blocks, int slots) {
  return b200ait::attn_longest_share({items, q_blocks, kv_blocks, true, false, 0, 0, 64}, slots);
}
extern "C" bool gemm_rowdot_short(long long m, long long n, long long k, int whole, int bf16) {
  return b200ait::gemm_rowdot_short(m, n, k, whole != 0, bf16 != 0);
}
extern "C" bool blocks_start_early(long long blocks, int threads, int filled, int light, int sms) {
  return b200ait::blocks_start_early(blocks, threads, sms, filled, light != 0);
}
extern "C" bool gemm_rows_output(int n, int tile_n, int residual) { return b200ait::gemm_rows_output(n, tile_n, residual != 0); }
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    work = tmp_path_factory.mktemp("rules")
    src, lib = work / "rules.cpp", work / "rules.so"
    src.write_text(_WRAPPERS)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-Wall", "-Werror", "-I",
                    os.path.join(ROOT, "aitemplate_b200", "csrc"), str(src), "-o", str(lib)], check=True)
    lib = ctypes.CDLL(str(lib))
    for f in (lib.blocks_start_early, lib.attn_lone, lib.attn_item_per_cta, lib.gemm_rowdot_short, lib.gemm_rows_output):
        f.restype = ctypes.c_bool
    lib.attn_longest_share.restype = ctypes.c_longlong
    return lib


@pytest.mark.parametrize("items,lone", [(1, True), (16, True), (128, True), (148, True), (149, False), (296, False)])
def test_wide_heads_with_an_item_per_sm_keep_four_stages(rules, items, lone):
    assert rules.attn_lone(ctypes.c_longlong(items), SMS) == lone


@pytest.mark.parametrize(
    "heads,seqs,bound,mean,causal,lengths,per_item",
    [
        # lengths on the device: they may be short, whatever the padding
        (16, 8, 4096, 4096, False, True, False),
        (16, 8, 4096, 4096, True, True, False),
        # packed: a bound far above the lengths makes nearly every CTA an empty one
        (12, 64, 4096, 128, True, False, False),
        (12, 16, 16384, 1024, True, False, False),
        (12, 8, 16384, 2048, False, False, False),
        (12, 4, 32768, 4096, True, False, False),
        # packed: short items do not pay for a set-up each
        (16, 8, 2048, 1152, True, False, False),
        (16, 8, 3072, 1728, True, False, False),
        (12, 8, 2560, 2048, False, False, False),
        # packed: long ones of different lengths do, just below 4096 rows as well as at it
        (16, 8, 4096, 2304, True, False, True),
        (16, 8, 4095, 2303, True, False, True),
        (16, 6, 3000, 2225, True, False, True),
        (12, 4, 6144, 3072, False, False, True),
        (16, 8, 4096, 2304, False, False, True),
        (16, 8, 4096, 3276, False, False, True),
        (16, 8, 3072, 1728, False, False, False),
        # equal items without a mask
        (16, 1, 4096, 4096, False, False, False),
        (48, 1, 4096, 4096, False, False, False),
        # causal, all sequences alike: by how uneven the shares are, at any length
        (32, 1, 2048, 2048, True, False, False),
        (32, 1, 4096, 4096, True, False, False),
        (32, 1, 3072, 3072, True, False, False),
        (768, 1, 200, 200, True, False, False),  # uneven shares, but items too short to pay for a set-up each
        (384, 1, 256, 256, True, False, False),
        (256, 1, 512, 512, True, False, False),
        (192, 1, 1024, 1024, True, False, True),
        (16, 1, 2560, 2560, True, False, True),
        (16, 1, 4096, 4096, True, False, True),
        (16, 1, 4095, 4095, True, False, True),
        (8, 1, 6144, 6144, True, False, True),
        (8, 1, 4096, 4096, True, False, False),  # 256 items: a slot for each anyway
    ],
)
def test_attention_items_get_a_cta_each_only_where_that_was_faster(rules, heads, seqs, bound, mean, causal, lengths, per_item):
    got = rules.attn_item_per_cta(*map(ctypes.c_longlong, (heads, seqs, bound, mean)), int(causal), int(lengths), 64, SMS)
    assert got == per_item


@pytest.mark.parametrize("heads,s,d,per_item", [(16, 4096, 40, True), (16, 4095, 24, True), (16, 3072, 40, True), (32, 2048, 40, False),
                                                (10, 4096, 40, False), (48, 4096, 40, False), (16, 4096, 48, False), (16, 4096, 56, False)])
def test_equal_items_stay_in_fixed_shares_but_for_narrow_heads_of_part_sectors(rules, heads, s, d, per_item):
    assert rules.attn_item_per_cta(*map(ctypes.c_longlong, (heads, 1, s, s)), 0, 0, d, SMS) == per_item


@pytest.mark.parametrize("items,q_blocks,kv_blocks,slots", [(320, 20, 40, 296), (1536, 48, 96, 296), (21, 7, 9, 4), (5, 5, 10, 296), (9, 3, 5, 2)])
def test_longest_share_is_the_longest_of_all_shares(rules, items, q_blocks, kv_blocks, slots):
    blocks = [min(kv_blocks, 2 * (q_blocks - i % q_blocks)) for i in range(items)]
    assert rules.attn_longest_share(ctypes.c_longlong(items), q_blocks, kv_blocks, slots) == max(
        sum(blocks[c::slots]) for c in range(slots))


@pytest.mark.parametrize(
    "m,n,k,whole,bf16,row_by_row",
    [
        (1, 256000, 256, True, False, True), (2, 50256, 256, True, False, True), (2, 80000, 256, True, False, False),
        (2, 128256, 384, True, True, True), (2, 128256, 392, True, False, True),
        (3, 8192, 256, True, False, True), (4, 16384, 320, True, False, False), (3, 128256, 256, True, False, False),
        (4, 20480, 320, True, True, True), (4, 30520, 384, True, True, False), (4, 50256, 448, True, False, False),
        (4, 50256, 512, True, False, True), (4, 50256, 576, True, False, False), (4, 24576, 640, True, True, True),
        (3, 128256, 512, True, True, False), (4, 128256, 704, True, True, False), (4, 50256, 768, True, True, False),
        (4, 50256, 768, True, False, True), (4, 128256, 776, True, True, True), (3, 128256, 1016, True, False, True),
        # rows that are not whole 16-byte units cost the tile kernels far more
        (4, 128257, 256, False, False, True), (3, 80001, 640, False, True, True),
        # neither fewer channels nor fewer rows, nor the longer rows of the other row-by-row kernel
        (1, 4096, 248, True, False, False), (1, 63, 512, True, False, False), (1, 4096, 1024, True, False, False),
    ],
)
def test_few_rows_against_short_ones_run_where_they_were_faster(rules, m, n, k, whole, bf16, row_by_row):
    assert rules.gemm_rowdot_short(*map(ctypes.c_longlong, (m, n, k)), int(whole), int(bf16)) == row_by_row


@pytest.mark.parametrize("n,tile_n,residual,row_by_row", [
    (1, 64, 0, False), (17, 64, 1, False), (41, 64, 0, False), (43, 64, 1, False), (44, 64, 0, True), (49, 64, 1, True), (63, 64, 0, True),
    (31, 128, 0, False), (31, 256, 1, False), (33, 128, 1, True), (33, 256, 0, True), (1001, 256, 1, True)])
def test_narrow_outputs_are_written_by_their_threads(rules, n, tile_n, residual, row_by_row):
    assert rules.gemm_rows_output(n, tile_n, residual) == row_by_row


@pytest.mark.parametrize(
    "blocks,threads,filled,light,early",
    [
        # rows: softmax of 365 x 1024, 3521 x 896, 13863 x 512, 520 x 3608 (128 threads), 1455 x 48
        (46, 256, 2048, 0, True), (441, 256, 2048, 0, False), (1733, 256, 2048, 0, True), (130, 128, 2048, 0, False), (182, 256, 2048, 1, True),
        # copies and transposes: 8 x [64 x 64], 172 x [112 x 56] twice, 91 x [862 x 112] twice, 11 x [112 x 758]
        (2, 256, 1024, 0, True), (132, 256, 1024, 0, False), (1074, 256, 1024, 0, True), (264, 256, 1024, 0, False),
        (74, 256, 2048, 0, True), (75, 256, 2048, 0, False), (592, 256, 1024, 0, True), (591, 256, 1024, 0, False),
    ])
def test_a_block_or_a_few_per_sm_wait_for_the_kernel_ahead(rules, blocks, threads, filled, light, early):
    assert rules.blocks_start_early(ctypes.c_longlong(blocks), threads, filled, light, SMS) == early
