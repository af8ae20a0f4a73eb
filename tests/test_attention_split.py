"""The rule that lets several CTAs share a key tile in the attention backward, on the CPU."""
import pytest


@pytest.mark.parametrize("lens,n_q,n_kv,split", [
    ([1], 4, 4, 1), ([20], 28, 4, 1), ([40], 28, 4, 1), ([80], 4, 4, 1), ([80], 28, 4, 1), ([40], 5, 1, 1), ([20] * 20, 14, 2, 1),
    ([300], 28, 4, 4), ([2049, 1500, 547], 28, 4, 2), ([1024, 1001, 1047], 28, 4, 2), ([1531, 977, 64, 2300, 1, 411], 14, 2, 4),
    ([5000, 300], 16, 1, 8), ([16384], 28, 4, 1), ([2048] * 8, 28, 4, 1),
])
def test_split_pays_for_its_cluster(lens, n_q, n_kv, split):
    """Short samples keep one CTA per key tile: a cluster's start and sums cost more there than the steps it shares.  The counts of
    longer rows are for 148 SMs, which the library takes where there is no GPU."""
    from pipelinerl_b200 import _build, _lib
    _build.build(verbose=False)
    assert _lib.load().prl_attn_bwd_split(sum(lens), max(lens), len(lens), n_q, n_kv) == split


@pytest.mark.parametrize("lens,n_q,n_kv,listed", [
    ([1531, 977, 64, 2300, 1, 411], 14, 2, True), ([512, 1024, 300, 2000, 1500, 700, 900, 1100], 28, 4, True), ([3000] + [11] * 300, 14, 2, True),
    ([0, 128, 129, 1, 0, 1500, 3], 4, 4, True), ([1700] * 3, 14, 2, False), ([1024] * 8, 28, 4, False), ([40] * 200, 14, 2, False), ([16] * 800, 14, 2, False),
    ([2 + i * 7 % 29 for i in range(800)], 14, 2, False), ([10 + i * 13 % 51 for i in range(400)], 28, 4, False), ([100, 30], 14, 2, False),
    ([128] * 64, 14, 2, False), ([5000], 14, 2, False),
])
def test_tiles_are_listed_where_that_pays(lens, n_q, n_kv, listed):
    """A tile that looks itself up in the list of the samples pays for the search: the list is for rows whose plain grid is mostly empty.
    Many short samples took up to twice the time with it (800 of 2 to 30 tokens: forward 97 us plain, 206 listed)."""
    from pipelinerl_b200 import _build, _lib
    _build.build(verbose=False)
    tiles = _lib.load().prl_attn_listed_tiles(sum(lens), max(lens), len(lens), n_q, n_kv)
    per = 128 // (n_q // n_kv)
    assert (tiles > 0) == listed
    assert not listed or sum(-(-n // per) for n in lens) <= tiles < len(lens) * -(-max(lens) // per)
