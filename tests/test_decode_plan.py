"""Rules that a decode engine plans its token step by, on the CPU."""
import ctypes

import pytest

from pipelinerl_b200 import _lib
from pipelinerl_b200.engine import batch_contexts, short_swiglu_slices, short_swiglu_tiles_pay, swiglu_epilogue_pays


@pytest.mark.parametrize("I,H,split,pays", [(18944, 3584, 1, True), (8192, 2048, 8, True), (4096, 1024, 2, False), (8000, 2048, 8, True),
                                            (7936, 2048, 8, False), (9408, 16384, 4, True), (9472, 2048, 8, False), (64, 320, 2, True),
                                            (64, 384, 2, False)])
def test_swiglu_epilogue_rule(I, H, split, pays):
    """Unsplit always; else while the idle SMs of I / 64 tiles on 148 cost at most 5 k-blocks of 64."""
    assert swiglu_epilogue_pays(I, H, split, 148) is pays


@pytest.mark.parametrize("I,H,rows,pays", [(4096, 1024, 4, True), (4096, 1024, 64, True), (4096, 1024, 65, False), (4736, 2048, 8, True),
                                           (4800, 2048, 8, False), (3264, 1088, 8, False), (3392, 1024, 8, True), (3264, 1024, 8, True), (3200, 1024, 8, False), (64, 320, 2, True)])
def test_short_swiglu_tiles_rule(I, H, rows, pays):
    """Up to 64 rows, tiles of 32 features on at most 148 SMs, and the idle ones cost at most 5 k-blocks of 64."""
    assert short_swiglu_tiles_pay(I, H, rows, 148) is pays


@pytest.mark.parametrize("split,rows,slices", [(2, 1, 2), (2, 8, 2), (2, 9, 1), (2, 64, 1), (1, 4, 1), (3, 4, 1), (7, 8, 1)])
def test_short_swiglu_tiles_keep_the_sums_of_the_split_pair(split, rows, slices):
    """Two slices of up to 8 rows are added in order; more of either are one sum."""
    assert short_swiglu_slices(split, rows) == slices


@pytest.mark.parametrize("lengths,want", [([5], (1, 5)), ([64, 64, 64], (3, 64)), ([64, 65], (2, 65)), ([16384] + [100] * 15, (2, 16384)), ([8192] * 32 + [1] * 32, (33, 8192))])
def test_unequal_contexts_as_a_number_of_equal_ones(lengths, want):
    assert batch_contexts(lengths) == want


def attn_plan(slots, live, n_kv, longest, max_seq_len):
    stages = ctypes.c_int32()
    return _lib.load().prl_paged_attn_plan(slots, live, n_kv, longest, max_seq_len, ctypes.byref(stages)), stages.value


@pytest.mark.parametrize("slots,live,n_kv,longest,plan", [
    (16, 16, 4, 16384, (2, 6)), (16, 8, 4, 16384, (4, 6)), (16, 1, 4, 16384, (8, 6)), (32, 32, 4, 4096, (1, 6)), (32, 4, 4, 4096, (4, 6)),      # a batch that drains
    (64, 64, 4, 8192, (2, 3)), (64, 19, 4, 8192, (2, 3)), (64, 18, 4, 8192, (2, 6)), (128, 128, 4, 4096, (1, 3)), (128, 37, 4, 4096, (1, 6)),
    (74, 74, 2, 6080, (1, 6)), (74, 74, 2, 6081, (2, 3)), (185, 185, 1, 8192, (1, 3)), (186, 186, 1, 4032, (1, 3)), (186, 186, 1, 4033, (2, 3)), (297, 297, 1, 8192, (1, 3)),
    (1, 1, 1, 512, (1, 6)), (1, 1, 1, 513, (2, 6)), (1, 1, 1, 5056, (16, 6)), (1, 1, 1, 5057, (32, 6)), (1, 1, 2, 8192, (16, 6)), (1, 1, 2, 8193, (32, 6)),
    (1, 1, 1, 16384, (32, 6)), (1, 1, 1, 16385, (64, 6)), (1, 1, 4, 131072, (32, 6)), (1, 1, 1, 1 << 23, (128, 6))])
def test_shares_of_decode_attention(slots, live, n_kv, longest, plan):
    """Both sides of the rule's lines on 148 SMs; full slots have what prl_paged_attn_splits says."""
    assert attn_plan(slots, live, n_kv, longest, longest) == plan
    if live == slots:
        assert _lib.load().prl_paged_attn_splits(slots, n_kv, longest) == plan[0]


@pytest.mark.parametrize("slots,live,longest,splits", [(32, 8, 512, 1), (32, 8, 513, 2), (32, 8, 1472, 2), (32, 8, 1473, 4), (32, 16, 1984, 1), (32, 16, 1985, 2), (64, 4, 832, 1),
                                                        (64, 4, 833, 2), (16, 4, 640, 4), (16, 4, 3008, 4), (16, 4, 3009, 8), (16, 1, 1216, 4), (16, 1, 1217, 8)])
def test_shares_beside_empty_slots(slots, live, longest, splits):
    """Both sides of the lines for batches with slots that have no token (four key heads)."""
    assert attn_plan(slots, live, 4, longest, 16384)[0] == splits


@pytest.mark.parametrize("slots", [1, 3, 16, 40, 64, 130])
@pytest.mark.parametrize("n_kv,max_seq_len", [(1, 640), (2, 2048), (4, 16384), (8, 131072)])
def test_workspace_of_the_longest_contexts_is_enough(slots, n_kv, max_seq_len):
    """What an engine allocates for (the longest contexts, any number of them) covers every plan of shorter ones."""
    most = max(attn_plan(slots, live, n_kv, max_seq_len, max_seq_len)[0] for live in range(1, slots + 1))
    for live in range(1, slots + 1):
        for longest in (1, 64, 513, 700, 4033, 6081, 10000, max_seq_len):
            splits, _ = attn_plan(slots, live, n_kv, min(longest, max_seq_len), max_seq_len)
            assert splits <= most and -(-max_seq_len // 64) <= 1024 * splits


def test_ring_budget_goes_back_to_the_rule():
    """A set budget is taken back by 0, the default; what no ring fits in stays refused."""
    lib = _lib.load()
    assert [lib.prl_gemm_set_smem_budget_kb(kb) for kb in (100, 220, 48, 0)] == [0] * 4
    assert all(lib.prl_gemm_set_smem_budget_kb(kb) != 0 for kb in (-1, 1, 47, 221))
