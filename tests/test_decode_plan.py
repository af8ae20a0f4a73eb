"""Rules that a decode engine plans its token step by, on the CPU."""
import pytest

from pipelinerl_b200.engine import short_swiglu_tiles_pay, swiglu_epilogue_pays


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


@pytest.mark.parametrize("rows,slices,pays", [(8, 1, True), (8, 2, True), (9, 2, False), (9, 1, True), (64, 1, True), (8, 3, False), (1, 7, False)])
def test_short_swiglu_tiles_keep_the_sums_of_the_split_pair(rows, slices, pays):
    """Two slices of up to 8 rows are added in the epilogue; more of either take the split pair."""
    assert short_swiglu_tiles_pay(4096, 1024, rows, 148, slices) is pays
