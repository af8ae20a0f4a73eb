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
