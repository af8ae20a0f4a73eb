"""The Modadra decoders on the hybrid engine (pipelinerl_b200/hybrid.py and its kernels) against
oracle/modadra_oracle.py: each mechanism alone, whole prompts against token-by-token decoding, portions down to two
tokens, unequal batches against each request alone, pages and slots that are given back and taken again, window edges and
the constant sink, the carried memory, the choice of experts, the first tokens, long decoding, awkward sizes, the bf16
serving mode, greedy generation through the engine's scheduler, and the trace runner."""
import json
import math
import subprocess
import sys

import pytest
import torch

from oracle import modadra_oracle as mo
from tests import modadra_cases as mc

pytestmark = pytest.mark.gpu

F32_TOL = 2e-4      # fp32 kernels against the float64 oracle
BF16_TOL = 8e-2     # bf16 operands / cache: rounding of activations dominates
P, M = mc.parallel, mc.moe


# ---- each mechanism alone ---------------------------------------------------------------------------------------
def _mechanisms():
    return {
        "both_mixers": mc.model([P()]),
        "every_head_its_own_keys_all_channels_rotated": mc.model([P(heads=4, kv_heads=4, dim=8, vdim=8, rot_dims=8, r_heads=3, r_kv_heads=3)]),
        "one_key_head_two_rotated_channels": mc.model([P(heads=5, kv_heads=1, dim=14, vdim=6, rot_dims=2, r_heads=4, r_kv_heads=1)]),
        "no_rotation_no_window": mc.model([P(rot_dims=0, window=0)]),
        "window_of_one": mc.model([P(window=1)]),
        "one_head_one_channel": mc.model([P(heads=1, kv_heads=1, dim=2, vdim=1, rot_dims=2, r_heads=1, r_kv_heads=1, r_dim=1, r_vdim=1)]),
        "wide_heads": mc.model([P(heads=2, kv_heads=1, dim=80, vdim=136, rot_dims=80, r_heads=2, r_kv_heads=1, r_dim=130, r_vdim=96)], width=40),
        "one_tap": mc.model([P(conv=1)]),
        "many_taps": mc.model([P(conv=7)]),
        "many_small_delta_heads": mc.model([P(r_heads=12, r_kv_heads=3, r_dim=4, r_vdim=8, conv=2)]),
        "routed": mc.model([P(mlp=M())]),
        "routed_one_expert": mc.model([P(mlp=M(experts=1, top=1, ff=9, groups=None))]),
        "routed_no_groups": mc.model([P(mlp=M(experts=7, top=2, ff=10, groups=None, scale=1.0))]),
        "routed_one_group_kept": mc.model([P(mlp=M(experts=12, top=3, ff=9, groups=(4, 1)))]),
        "routed_groups_of_one": mc.model([P(mlp=M(experts=6, top=2, ff=8, groups=(6, 3)))]),
        "routed_groups_of_four": mc.model([P(mlp=M(experts=12, top=5, ff=8, groups=(3, 2), scale=2.5))]),
        "routed_everything": mc.model([P(mlp=M(experts=5, top=5, ff=9, groups=(5, 5)))]),
        "routed_many": mc.model([P(mlp=M(experts=80, top=8, ff=6, groups=(8, 4)))]),
        "odd_width": mc.model([P(mlp=M()), P(heads=3, kv_heads=1)], vocab=61, width=50),
        "no_cap_whole_residual": mc.model([P(mlp=M()), P()], cap=0.0, mult=1.0),
        "three_layers": mc.model([P(mlp=M()), P(heads=3, kv_heads=3, window=9, conv=4), P(r_dim=16, r_vdim=16, mlp=M(experts=4, groups=(2, 1), top=2))]),
    }


@pytest.mark.parametrize("name", sorted(_mechanisms()))
def test_each_mechanism_matches_the_oracle_fp32(cuda_device, name):
    config = _mechanisms()[name]
    wt = mc.weights(config, seed=len(name))
    toks = mc.tokens_for(config, 150)
    res = []
    ref = mc.oracle_logits(config, wt, toks, residuals=res)
    eng = mc.build_engine(config, wt, torch.float32, cuda_device)
    assert mc.rel_err(mc.stream_logits(eng, toks, [150]), ref) < F32_TOL
    assert mc.rel_err(mc.stream_logits(eng, toks, [2, 3, 61, 2, 7, 64, 2]), ref) < F32_TOL     # then one by one
    # the residual stream after every layer of a whole prompt
    s = mc.stage_stream(eng, toks[:20])
    got = []
    eng._forward_rows([(s, 0, 20)], [], trace=got)
    eng.close_stream(s)
    assert len(got) == len(res)
    for a, b in zip(got, res):
        assert (a.double().cpu() - b[:20]).abs().max().item() < 1e-4 * max(1.0, b.abs().max().item())


FULL = mc.model([P(mlp=M()), P(heads=4, kv_heads=2, dim=16, vdim=20, rot_dims=16, window=70, r_heads=4, r_kv_heads=4, r_dim=12, r_vdim=9, conv=4),
                 P(heads=3, kv_heads=1, window=65, r_heads=2, r_kv_heads=1, r_dim=24, r_vdim=16, mlp=M(experts=6, top=2, groups=(3, 2), ff=16))],
                vocab=80, width=64)


def test_prefill_against_token_by_token_decoding(cuda_device):
    wt = mc.weights(FULL, 3)
    toks = mc.tokens_for(FULL, 140, seed=5)
    ref = mc.oracle_logits(FULL, wt, toks)
    eng = mc.build_engine(FULL, wt, torch.float32, cuda_device)
    whole = mc.stream_logits(eng, toks, [140])
    single = mc.stream_logits(eng, toks, [])                                 # every token alone, through the cache / state
    assert mc.rel_err(whole, ref) < F32_TOL and mc.rel_err(single, ref) < F32_TOL
    assert mc.rel_err(whole, single) < 2e-5


@pytest.mark.parametrize("portions", [[2] * 40, [63, 2, 63, 2], [64, 64], [1, 65, 1, 2, 59], [129, 2], [39, 1, 41, 9]])
def test_portions_of_several_sizes(cuda_device, portions):
    wt = mc.weights(FULL, 4)
    toks = mc.tokens_for(FULL, 140, seed=6)
    ref = mc.oracle_logits(FULL, wt, toks)
    eng = mc.build_engine(FULL, wt, torch.float32, cuda_device, prefill_chunk=96)   # 129 is cut by the engine too
    assert mc.rel_err(mc.stream_logits(eng, toks, portions), ref) < F32_TOL


def test_unequal_batches_equal_each_request_alone(cuda_device):
    wt = mc.weights(FULL, 7)
    seqs = [mc.tokens_for(FULL, n, seed=10 + n) for n in (1, 37, 130, 66)]
    eng = mc.build_engine(FULL, wt, torch.float32, cuda_device)
    alone = [mc.stream_logits(eng, s, [len(s)]) for s in seqs]
    # together: every step brings a different mix of portion sizes; request 0 joins late, request 2 skips a step
    streams = [eng.open_stream() for _ in seqs]
    got = [[] for _ in seqs]
    at = [0] * len(seqs)
    plan = [{1: 5, 2: 64}, {0: 1, 1: 1, 2: 2, 3: 30}, {1: 31, 3: 36}, {2: 64, 3: 0}]
    for step in plan:
        entries, who = [], []
        for i, k in step.items():
            if k:
                entries.append((streams[i], seqs[i][at[i]:at[i] + k], list(range(k))))
                who.append((i, k))
                at[i] += k
        lg = eng.feed(entries).double().cpu()
        r = 0
        for i, k in who:
            got[i].append(lg[r:r + k])
            r += k
    assert at == [len(s) for s in seqs]
    for i, s in enumerate(streams):
        eng.close_stream(s)
        assert mc.rel_err(torch.cat(got[i]), alone[i]) < 2e-5, f"request {i} depends on its batch"
    assert mc.rel_err(alone[2], mc.oracle_logits(FULL, wt, seqs[2])) < F32_TOL


def test_pages_and_slots_are_reused(cuda_device):
    """Two slots and five pages for eight sequences: every later sequence runs in a slot whose memory and convolution inputs
    another one left, and on pages that held other keys and values."""
    wt = mc.weights(FULL, 8)
    eng = mc.build_engine(FULL, wt, torch.float32, cuda_device, max_batch=2, max_seq_len=192, n_pages=1 + 5)
    lens = [100, 70, 5, 128, 64, 1, 150, 65]
    for k, n in enumerate(lens):
        toks = mc.tokens_for(FULL, n, seed=40 + k)
        ref = mc.oracle_logits(FULL, wt, toks)
        held = eng.open_stream()
        eng.feed([(held, mc.tokens_for(FULL, 60 + k, seed=k), [])])          # a neighbour that dirties the other slot
        got = mc.stream_logits(eng, toks, [max(1, n // 2), 2])
        eng.close_stream(held)
        assert mc.rel_err(got, ref) < F32_TOL, f"sequence {k}"
        assert len(eng.free_pages) == 5 and len(eng.free_slots) == 2


# ---- edges made to stand out ------------------------------------------------------------------------------------------
PLANS = ([330], [63, 1, 1, 63, 2, 126], [64, 64, 64, 64], [199, 2, 54, 2], [250])       # the rest one by one


@pytest.mark.parametrize("window", [1, 33, 64, 65, 200])
def test_window_edges_and_the_constant_sink(cuda_device, window):
    """Peaked scores (a large score scale) so that single keys carry a row's weight; the oracle with a window one longer or
    one shorter, or without the one in the denominator, is far outside the tolerance, so a key that is one position off at
    the edge shows, in portions of a prompt and in single decoded tokens, at page borders and inside pages."""
    config = mc.model([P(heads=4, kv_heads=2, dim=12, vdim=10, window=window, scale=0.9)], width=40)
    wt = mc.weights(config, 19)
    wt["l0.mix.right.out"] = mc.bf16_round(wt["l0.mix.right.out"] * 0.1)                  # the attention decides
    toks = mc.tokens_for(config, 330, seed=3)
    ref = mc.oracle_logits(config, wt, toks)
    for other in ([window + 1] if window == 1 else [window - 1, window + 1]):
        wrong = mc.oracle_logits(mc.replaced(config, ["layers", 0, "mixer", "left", "mask", "size"], other), wt, toks)
        assert mc.rel_err(wrong[window:], ref[window:]) > 100 * F32_TOL
        assert ((wrong - ref).abs().amax(-1)[window:] > 1e-3).float().mean() > 0.5        # most positions, not one
    plain = mo.sink_attention
    try:
        mo.sink_attention = lambda *a: plain(*a, sink=0.0)
        assert mc.rel_err(mc.oracle_logits(config, wt, toks), ref) > 100 * F32_TOL
    finally:
        mo.sink_attention = plain
    eng = mc.build_engine(config, wt, torch.float32, cuda_device)
    for portions in PLANS:
        assert mc.rel_err(mc.stream_logits(eng, toks, portions), ref) < F32_TOL
    eng16 = mc.build_engine(config, wt, torch.bfloat16, cuda_device)
    assert mc.rel_err(mc.stream_logits(eng16, toks, [199, 2, 54, 2]), ref) < BF16_TOL


def test_one_far_key_inside_the_window_stands_out(cuda_device):
    """One token whose key is long and whose queries ask for it: the positions up to window - 1 behind it see it, the next
    one does not.  The token sits at several places of a page, and the asking tokens come in portions and one by one."""
    config = mc.model([P(heads=2, kv_heads=1, dim=8, vdim=8, window=100, rot_dims=0, scale=1.0)], width=32, vocab=40)
    wt = mc.weights(config, 5)
    wt["l0.mix.left.q"] *= 0.3
    wt["l0.mix.right.out"] = mc.bf16_round(wt["l0.mix.right.out"] * 0.1)
    # token 7 is what the keys answer to, token 9 what the queries ask with
    h7 = mo.rms_unit(wt["embed"][7], 1e-5) * wt["l0.norm1"]
    h9 = mo.rms_unit(wt["embed"][9], 1e-5) * wt["l0.norm1"]
    c = torch.ones(8, dtype=torch.float64)
    wt["l0.mix.left.k"] = mc.bf16_round(wt["l0.mix.left.k"] * 0.3 + 2.0 * torch.outer(c, h7) / (h7 @ h7))
    wt["l0.mix.left.q"] = mc.bf16_round(wt["l0.mix.left.q"] + 2.0 * torch.outer(torch.cat([c, c]), h9) / (h9 @ h9))
    eng = mc.build_engine(config, wt, torch.float32, cuda_device)
    for place in (0, 1, 62, 63, 64, 65):
        toks = [t if t not in (7, 9) else 3 for t in mc.tokens_for(config, 190, seed=place)]
        toks[place] = 7
        for p in (place + 50, place + 98, place + 99, place + 100, place + 101):
            toks[p] = 9
        ref = mc.oracle_logits(config, wt, toks)
        other = list(toks)
        other[place] = 3
        moved = (mc.oracle_logits(config, wt, other) - ref).abs().amax(-1)
        assert moved[place + 99] > 0.05 and moved[place + 100] < 0.5 * moved[place + 99]
        for portions in ([190], [place + 99, 2], [place + 100, 2], [place + 1], [64, 64]):
            assert mc.rel_err(mc.stream_logits(eng, toks, portions), ref) < F32_TOL


def test_rotation_follows_the_position(cuda_device):
    """Fast rotations on every channel: a key or query turned by a neighbouring position's angle, or pairs taken in another
    layout, move the scores by O(1)."""
    config = mc.model([P(heads=2, kv_heads=1, dim=12, vdim=10, rot_dims=12, base=3.0, window=90, scale=0.8)], width=40)
    wt = mc.weights(config, 23)
    toks = mc.tokens_for(config, 200, seed=2)
    ref = mc.oracle_logits(config, wt, toks)
    for path, value in ((["layers", 0, "mixer", "left", "rot", "base"], 3.3), (["layers", 0, "mixer", "left", "rot", "dims"], 10)):
        assert mc.rel_err(mc.oracle_logits(mc.replaced(config, path, value), wt, toks), ref) > 100 * F32_TOL
    eng = mc.build_engine(config, wt, torch.float32, cuda_device)
    for portions in ([200], [1, 2, 62, 3, 64], [130]):
        assert mc.rel_err(mc.stream_logits(eng, toks, portions), ref) < F32_TOL


@pytest.mark.parametrize("shift,far", [(-6.0, True), (2.0, False)])
def test_far_tokens_in_the_memory(cuda_device, shift, far):
    """Decays close to 1 and keys of 64 channels (later writes hardly erase): the memory at token 300 still holds the first tokens, so a state (or the convolution's last
    inputs) that is lost, reset or not carried across portions shows at every later position.  A second model with strong
    decay exercises the other end."""
    config = mc.model([P(window=5, r_heads=4, r_kv_heads=2, r_dim=64, r_vdim=8, conv=4)], width=40)
    wt = mc.weights(config, 11)
    wt["l0.mix.right.A_log"] = mc.bf16_round(wt["l0.mix.right.A_log"] + shift)
    wt["l0.mix.left.out"] = mc.bf16_round(wt["l0.mix.left.out"] * 0.1)
    toks = mc.tokens_for(config, 300, seed=4)
    ref = mc.oracle_logits(config, wt, toks)
    if far:
        other = [(toks[0] + 1) % config["vocab"]] + toks[1:]
        assert mc.rel_err(mc.oracle_logits(config, wt, other)[250:], ref[250:]) > 20 * F32_TOL
    eng = mc.build_engine(config, wt, torch.float32, cuda_device)
    assert mc.rel_err(mc.stream_logits(eng, toks, [300]), ref) < F32_TOL
    assert mc.rel_err(mc.stream_logits(eng, toks, [7, 2, 120, 2, 9]), ref) < F32_TOL      # then 160 single tokens
    assert mc.rel_err(mc.stream_logits(eng, toks, [1, 1, 1, 2, 3, 100]), ref) < F32_TOL   # portions shorter than the taps


def test_first_tokens_and_one_token_sequences(cuda_device):
    wt = mc.weights(FULL, 12)
    eng = mc.build_engine(FULL, wt, torch.float32, cuda_device)
    for n in (1, 2, 3, 4, 5):
        toks = mc.tokens_for(FULL, n, seed=70 + n)
        ref = mc.oracle_logits(FULL, wt, toks)
        assert mc.rel_err(mc.stream_logits(eng, toks, [n]), ref) < F32_TOL
        assert mc.rel_err(mc.stream_logits(eng, toks, []), ref) < F32_TOL


# ---- the choice of experts --------------------------------------------------------------------------------------------
@pytest.mark.parametrize("shift", [0.0, -4.0])
def test_routing_follows_scores_corrections_and_groups(cuda_device, shift):
    """Scores far apart and corrections large enough to change the choice, also with every choice score negative: a closed
    group that counts as zero, a group ranked by its best output alone, a weight that sees the correction, is not divided by
    the sum or misses the constant shows at once."""
    config = mc.model([P(mlp=M(experts=12, top=3, ff=12, groups=(4, 2), scale=1.7))], width=40)
    wt = mc.weights(config, 17)
    wt["l0.mlp.router"] = mc.bf16_round(wt["l0.mlp.router"] * 2.0)
    wt["l0.mlp.correction"] = mc.bf16_round(wt["l0.mlp.correction"] * 2.0 + shift)
    toks = mc.tokens_for(config, 120, seed=4)
    gaps = []
    ref = mc.oracle_logits(config, wt, toks, margins=gaps)
    clear = torch.tensor(gaps[0]) > 1e-4
    assert clear.float().mean() > 0.9
    other = dict(wt)
    other["l0.mlp.correction"] = torch.zeros(12, dtype=torch.float64)
    assert mc.rel_err(mc.oracle_logits(config, other, toks), ref) > 50 * F32_TOL
    for path, value in ((["layers", 0, "mlp", "router", "groups"], None), (["layers", 0, "mlp", "router", "scale"], 1.6)):
        assert mc.rel_err(mc.oracle_logits(mc.replaced(config, path, value), wt, toks), ref) > 50 * F32_TOL
    eng = mc.build_engine(config, wt, torch.float32, cuda_device)
    assert mc.rel_err(mc.stream_logits(eng, toks, [100, 2])[clear], ref[clear]) < F32_TOL
    eng.unfused_router = True
    assert mc.rel_err(mc.stream_logits(eng, toks, [100, 2])[clear], ref[clear]) < F32_TOL


@pytest.mark.parametrize("experts,top,groups,keep", [(12, 3, 4, 2), (8, 8, 1, 1), (6, 2, 6, 3), (96, 7, 8, 3), (33, 4, 3, 1), (1, 1, 1, 1),
                                                     (260, 5, 4, 2), (80, 40, 2, 2)])
def test_choice_kernels(cuda_device, experts, top, groups, keep):
    """prl_moe_choose and prl_moe_router_choose alone, with sigmoid scores, groups ranked by their two best and weights
    divided by their sum: choices, weights and the grouping by expert."""
    from pipelinerl_b200 import _lib
    lib, n, W = _lib.load(), 70 if experts % 3 else 700, 48
    g = torch.Generator().manual_seed(experts)
    x, wr = torch.randn(n, W, generator=g), torch.randn(experts, W, generator=g) * 0.4
    corr = torch.randn(experts, generator=g) - 2.0
    z = x.double() @ wr.double().T
    want = [mo.choose(torch.sigmoid(z[t]), corr.double(), dict(top=top, groups=dict(count=groups, keep=keep))) for t in range(n)]
    d, i32 = cuda_device, dict(dtype=torch.int32, device=cuda_device)
    xd, wd, cd, zd = x.to(d), wr.to(d), corr.to(d), z.float().to(d)
    st = _lib.stream_ptr()
    for ready in (True, False):
        sel, perm = torch.full((top, n), -1, **i32), torch.full((top * n,), -1, **i32)
        wsel, meta = torch.zeros(top, n, device=d), torch.zeros(4, **i32)
        tiles = torch.zeros(3 * int(lib.prl_moe_max_tiles(top * n, experts)), **i32)
        rule = (top, groups, keep, 2, 1, 1, 1.7, 64, sel.data_ptr(), wsel.data_ptr(), perm.data_ptr(), meta.data_ptr(), tiles.data_ptr(), st)
        if ready:
            _lib.check(lib.prl_moe_choose(zd.data_ptr(), experts, cd.data_ptr(), n, experts, experts, *rule))
        else:
            _lib.check(lib.prl_moe_router_choose(xd.data_ptr(), 1, wd.data_ptr(), 1, cd.data_ptr(), n, W, experts, experts, *rule))
        s, w = sel.cpu(), wsel.double().cpu()
        assert s.T.tolist() == want
        for t in range(n):
            sc = torch.sigmoid(z[t, want[t]])
            assert torch.allclose(w[:, t], sc / sc.sum() * 1.7, atol=1e-5)
        order = [p for e in range(experts) for p in range(top * n) if s.view(-1)[p] == e]
        assert perm.tolist() == order and meta[1].item() == top * n


# ---- the serving mode --------------------------------------------------------------------------------------------------
BIG = mc.model([P(heads=8, kv_heads=2, dim=32, vdim=32, rot_dims=16, window=100, r_heads=4, r_kv_heads=2, r_dim=64, r_vdim=32, conv=4,
                  mlp=M(experts=3, top=3, ff=64, groups=None)),
                P(heads=4, kv_heads=2, dim=48, vdim=64, rot_dims=48, window=120, r_heads=4, r_kv_heads=4, r_dim=32, r_vdim=64, conv=4),
                P(heads=4, kv_heads=4, dim=32, vdim=48, rot_dims=32, window=70, r_heads=2, r_kv_heads=1, r_dim=48, r_vdim=64, conv=3,
                  mlp=M(experts=8, top=2, ff=96, groups=(4, 2)))], vocab=200, width=128)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,W,experts,groups,keep,top", [(1, 8, 4, 1, 1, 4), (33, 2048, 16, 8, 6, 4), (592, 264, 32, 4, 2, 16), (593, 1032, 33, 3, 1, 5),
                                                         (1023, 2056, 16, 8, 8, 1)])
def test_router_rows_equal_the_staged_router(cuda_device, dtype, n, W, experts, groups, keep, top):
    """Rows and weights on 16-byte boundaries take a kernel of their own; rows one element further on, the one that stages them.
    Sums, ranking and weights are the same in both, also for rows with infinities and NaN."""
    from pipelinerl_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(n + W)
    x = torch.randn(n, W, generator=g, device="cuda").to(dtype)
    w = (torch.randn(experts, W, generator=g, device="cuda") * W ** -0.5).to(dtype)
    shifted = torch.empty(n * W + 1, dtype=dtype, device="cuda")[1:]
    shifted.copy_(x.view(-1))
    corr = torch.randn(experts, generator=g, device="cuda")
    lib, st = _lib.load(), _lib.stream_ptr()
    i32 = dict(dtype=torch.int32, device="cuda")
    for sigmoid in (2, 0, 1):                       # 2: prl_moe_router (softmax over the chosen), for finite logits
        if sigmoid == 0 and n > 8:
            x[3, 1], x[5, W // 2], x[7, 0] = float("inf"), float("nan"), -float("inf")
            shifted.copy_(x.view(-1))
        got = []
        for rows in (x, shifted):
            sel, wsel, perm = torch.full((top, n), -7, **i32), torch.full((top, n), -7.0, device="cuda"), torch.zeros(top * n, **i32)
            meta, tiles = torch.zeros(4, **i32), torch.zeros(3 * int(lib.prl_moe_max_tiles(top * n, experts)), **i32)
            f32 = int(dtype == torch.float32)
            tail = (sel.data_ptr(), wsel.data_ptr(), perm.data_ptr(), meta.data_ptr(), tiles.data_ptr(), st)
            if sigmoid == 2:
                _lib.check(lib.prl_moe_router(rows.data_ptr(), f32, w.data_ptr(), f32, corr.data_ptr(), n, W, experts, top, 1, *tail))
            else:
                _lib.check(lib.prl_moe_router_choose(rows.data_ptr(), f32, w.data_ptr(), f32, corr.data_ptr(), n, W, experts, experts, top,
                                                     groups, keep, 2, sigmoid, 1, 1.25, 64, *tail))
            got.append((sel, wsel.view(torch.int32)))
        assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,W,experts,groups,keep,top", [(149, 264, 16, 4, 2, 3), (297, 136, 128, 8, 4, 8), (450, 136, 128, 8, 4, 8), (450, 1032, 8, 1, 1, 2), (600, 136, 8, 1, 1, 2), (889, 72, 16, 8, 6, 4),
                                                         (1185, 264, 32, 4, 2, 6)])
def test_router_of_every_schedule(cuda_device, dtype, n, W, experts, groups, keep, top):
    """One, two, four and eight rows a block and a block per row: the lines lie at one, two, three, four, six and eight rows per SM (148)."""
    test_router_rows_equal_the_staged_router(cuda_device, dtype, n, W, experts, groups, keep, top)


def ranked_on_the_host(z, corr, top, groups, keep, group_top, sigmoid, renorm, scale):
    """The choice for one row of logits, entry by entry: ties go to the lower index, NaN is never the largest, an entry or a group that
    is minus infinity is never taken in a round, and a group that has not been taken is closed if it is anything but minus infinity."""
    import numpy as np
    with np.errstate(all="ignore"):
        z = z.astype(np.float32)
        e = np.exp(z - np.fmax.reduce(z))
        score = (1 / (1 + np.exp(-z)) if sigmoid else e * (np.float32(1) / e.sum(dtype=np.float32))).astype(np.float32)
        c, size = score + corr, len(z) // groups

        def largest(v):
            best, at = -np.inf, None
            for i, x in enumerate(v):
                if x > best:
                    best, at = x, i
            return at
        if keep < groups:
            gs = []
            for g in range(groups):
                m = m2 = np.float32(-np.inf)
                for x in c[g * size:(g + 1) * size]:
                    m2, m = np.fmax(m2, np.fmin(m, x)), np.fmax(m, x)
                gs.append(m + m2 if group_top > 1 and size > 1 else m)
            for _ in range(keep):
                g = largest(gs)
                if g is not None:
                    gs[g] = -np.inf
            c = np.array([-np.inf if gs[i // size] != -np.inf else x for i, x in enumerate(c)], dtype=np.float32)
        sel, w = [], []
        for _ in range(top):
            i = largest(c)
            sel.append(0 if i is None else i)
            w.append(np.float32(0) if i is None else score[i])
            if i is not None:
                c[i] = -np.inf
        w = np.array(w, dtype=np.float32)
        return sel, w * np.float32(scale) / ((w.sum() + np.float32(1e-20)) if renorm else np.float32(1))


@pytest.mark.parametrize("E,groups,keep,top", [(1, 1, 1, 1), (4, 1, 1, 4), (16, 8, 6, 4), (16, 8, 8, 5), (24, 3, 1, 8), (32, 32, 5, 3), (32, 4, 2, 16), (31, 1, 1, 31),
                                               (32, 1, 1, 32), (33, 3, 1, 5), (64, 8, 3, 7)])
def test_choice_of_outputs_against_the_host(cuda_device, E, groups, keep, top):
    """Up to 32 outputs are ranked in registers, more in shared memory: both against a plain restatement, for equal logits, zeros of both
    signs, infinities and NaN in logits and corrections.  The logits are those whose scores are exact on both sides (sigmoids 0, 1/2 and 1,
    softmax shares 0 and 1 / k), so that every comparison falls the same way."""
    import numpy as np
    from pipelinerl_b200 import _lib
    lib, st, rng, n = _lib.load(), _lib.stream_ptr(), np.random.default_rng(E + groups), 96
    i32 = dict(dtype=torch.int32, device="cuda")
    for trial in range(8):
        z = rng.choice(np.array([-200.0, -0.0, 0.0, 0.0, 200.0, 200.0], dtype=np.float32), (n, E))
        odd = rng.random((n, E)) < 0.2 * (rng.random((n, 1)) < 0.6)
        z[odd] = rng.choice(np.array([np.inf, -np.inf, np.nan, -np.inf], dtype=np.float32), int(odd.sum()))
        corr = (rng.integers(-24, 25, E) / (8 if trial < 4 else 64)).astype(np.float32)
        corr[rng.random(E) < 0.15] = (0.0, -np.inf, -0.0, np.nan)[trial % 4]
        sigmoid, renorm, group_top = trial & 1, trial >> 1 & 1, 1 + (trial >> 2 & 1)
        sel, wsel, perm = torch.full((top, n), -7, **i32), torch.full((top, n), -7.0, device="cuda"), torch.zeros(top * n, **i32)
        meta, tiles = torch.zeros(4, **i32), torch.zeros(3 * int(lib.prl_moe_max_tiles(top * n, E)), **i32)
        zd, cd = torch.from_numpy(z).cuda(), torch.from_numpy(corr).cuda()
        _lib.check(lib.prl_moe_choose(zd.data_ptr(), E, cd.data_ptr(), n, E, E, top, groups, keep, group_top, sigmoid, renorm, 1.25, 64, sel.data_ptr(),
                                      wsel.data_ptr(), perm.data_ptr(), meta.data_ptr(), tiles.data_ptr(), st))
        for t in range(n):
            want, w = ranked_on_the_host(z[t], corr, top, groups, keep, group_top, sigmoid, renorm, 1.25)
            assert sel[:, t].tolist() == want, (trial, t)
            # the scores are exact or one rounding away (1 / k); the sum of up to 32 of them and the division add 2^-24 each at most
            np.testing.assert_allclose(wsel[:, t].cpu().numpy(), w, rtol=5e-6, atol=1e-30, equal_nan=True)


@pytest.mark.parametrize("plain_gemm", [False, True])
def test_bf16_serving_mode(cuda_device, plain_gemm):
    """bf16 operands and cache with the tensor-core GEMMs (and with the CUDA-core GEMM) against the float64 oracle.  Only the
    last layer's router has a choice to make, so a token whose choice is closer than bf16 rounding can tell apart touches
    only its own logits; the oracle reports the gaps and those positions are left out."""
    wt = mc.weights(BIG, 13)
    toks = mc.tokens_for(BIG, 300, seed=8)
    gaps = []
    ref = mc.oracle_logits(BIG, wt, toks, margins=gaps)
    assert min(gaps[0]) == math.inf
    clear = torch.tensor(gaps[-1]) > 0.03
    assert clear.float().mean().item() > 0.7
    eng = mc.build_engine(BIG, wt, torch.bfloat16, cuda_device, prefill_chunk=512)
    eng.force_plain_gemm = plain_gemm
    whole = mc.stream_logits(eng, toks, [300])
    assert mc.rel_err(whole[clear], ref[clear]) < BF16_TOL
    assert mc.rel_err(mc.stream_logits(eng, toks, [100, 2, 30])[clear], ref[clear]) < BF16_TOL
    # the bf16 engine is about as close to the oracle as the oracle with only its matrix products' inputs rounded
    least = mc.rel_err(mc.oracle_logits(BIG, wt, toks, round_in=mc.bf16_round)[clear], ref[clear])
    assert mc.rel_err(whole[clear], ref[clear]) < 3 * least + 1e-3


@pytest.mark.parametrize("graph", [False, True])
def test_branches_on_two_streams_equal_one_after_the_other(cuda_device, graph):
    """The attention and delta-rule branches of a layer run beside each other, in prompts and in the (captured) token step: the same
    tokens and log-probabilities as one after the other, also from a stream of the caller's."""
    from pipelinerl_b200.engine import SamplingParams
    wt = mc.weights(BIG, 5)
    prompts, got = [mc.tokens_for(BIG, n, seed=n) for n in (400, 300, 5)], []
    for side, own in ((True, False), (False, False), (True, True)):
        eng = mc.build_engine(BIG, wt, torch.bfloat16, cuda_device, max_batch=3, max_seq_len=700, use_cuda_graph=graph)
        eng.side_branches = side
        s = torch.cuda.Stream() if own else torch.cuda.current_stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            outs = eng.generate(prompts, SamplingParams(max_tokens=9, greedy=True, ignore_eos=True))
        torch.cuda.synchronize()
        assert (eng._side is not None) == side
        got.append([(list(r.output_ids), list(r.output_logprobs)) for r in outs])
    assert got[0] == got[1] == got[2]


@pytest.mark.parametrize("graph", [False, True])
def test_narrow_prompts_keep_one_stream(cuda_device, graph):
    """Where nothing else is asked for, a narrow decoder's prompts and its uncaptured token steps run on one stream, captured steps on two."""
    from pipelinerl_b200.engine import SamplingParams
    eng = mc.build_engine(BIG, mc.weights(BIG, 5), torch.bfloat16, cuda_device, max_batch=2, max_seq_len=400, use_cuda_graph=graph)
    s = eng.open_stream()
    eng.feed([(s, mc.tokens_for(BIG, 300, seed=1), [299])])
    eng.close_stream(s)
    assert eng._side is None
    eng.generate([mc.tokens_for(BIG, 9, seed=2)], SamplingParams(max_tokens=3, greedy=True, ignore_eos=True))
    assert (eng._side is not None) == graph


def test_grouped_tensor_core_experts_in_long_prompts(cuda_device):
    """More routed pairs per expert than the few-row grouped GEMM is for: the tcgen05 grouped GEMM with the gelu epilogue
    against the few-row kernel on the same weights."""
    config = mc.model([P(mlp=M(experts=4, top=2, ff=128, groups=(2, 2)))], width=128)
    wt = mc.weights(config, 6)
    toks = mc.tokens_for(config, 300, seed=5)
    eng = mc.build_engine(config, wt, torch.bfloat16, cuda_device, prefill_chunk=512)
    eng.moe_tc_rows = 1 << 30
    few = mc.stream_logits(eng, toks, [300])
    eng.moe_tc_rows = 1
    many = mc.stream_logits(eng, toks, [300])
    assert mc.rel_err(many, few) < 5e-3
    gaps = []
    ref = mc.oracle_logits(config, wt, toks, margins=gaps)
    clear = torch.tensor(gaps[0]) > 0.03
    assert mc.rel_err(many[clear], ref[clear]) < BF16_TOL


@pytest.mark.parametrize("dim,vdim,window", [(32, 32, 100), (64, 64, 64), (128, 128, 37), (80, 48, 90), (48, 96, 33), (16, 16, 200)])
def test_tensor_core_prompt_attention(cuda_device, dim, vdim, window):
    """bf16 with head sizes the tensor-core prompt kernel is built for, peaked scores over five page borders, against the
    CUDA-core kernel on the same cache (they differ by the bf16 rounding of the softmax weights) and against the oracle."""
    config = mc.model([P(heads=4, kv_heads=2, dim=dim, vdim=vdim, rot_dims=dim // 2, window=window, scale=1.5 * dim ** -0.5)], width=64)
    wt = mc.weights(config, 9)
    toks = mc.tokens_for(config, 330, seed=3)
    ref = mc.oracle_logits(config, wt, toks)
    eng = mc.build_engine(config, wt, torch.bfloat16, cuda_device, prefill_chunk=512)
    plans = ([330], [63, 17, 16, 130, 65, 20, 3, 2], [300])                 # the rest one by one
    eng.tc_prompt[0] = False                                                # heads of 128 have another test
    fast = [mc.stream_logits(eng, toks, p) for p in plans]
    eng.lib.prl_attn_any_tensor_cores(0)
    try:
        plain = [mc.stream_logits(eng, toks, p) for p in plans]
    finally:
        eng.lib.prl_attn_any_tensor_cores(1)
    for f, p in zip(fast, plain):
        assert 0 < mc.rel_err(f, p) < 0.25 * BF16_TOL                        # two kernels, the same result
        assert mc.rel_err(f, ref) < BF16_TOL and mc.rel_err(p, ref) < BF16_TOL


CELLS = [(4, 2, 12, 8, 3), (3, 1, 10, 13, 4), (2, 2, 32, 48, 2), (4, 2, 64, 64, 4), (2, 1, 128, 128, 4), (2, 1, 40, 132, 1), (1, 1, 200, 20, 4),
         (6, 2, 5, 40, 6)]       # heads, q / k heads, key size, value size, taps


@pytest.mark.parametrize("heads,kv,dk,dv,taps", CELLS)
def test_pieces_of_the_gated_delta_rule(cuda_device, heads, kv, dk, dv, taps):
    """Long portions as side-by-side pieces (off in fp32 unless asked for) against the oracle and the token-by-token walk: one
    piece that is not full, several, pieces of other lengths, portions that continue a state, and single tokens of another
    sequence beside them.  Memories that last (decays near one) make a wrong state at a piece's border show in every row
    behind it."""
    config = mc.model([P(window=5, r_heads=heads, r_kv_heads=kv, r_dim=dk, r_vdim=dv, conv=taps)], width=40)
    for shift in (-3.0, 1.0):
        wt = mc.weights(config, 27)
        wt["l0.mix.right.A_log"] = mc.bf16_round(wt["l0.mix.right.A_log"] + shift)
        wt["l0.mix.left.out"] = mc.bf16_round(wt["l0.mix.left.out"] * 0.1)
        toks, other = mc.tokens_for(config, 300, seed=21), mc.tokens_for(config, 20, seed=22)
        ref, oref = mc.oracle_logits(config, wt, toks), mc.oracle_logits(config, wt, other)
        eng = mc.build_engine(config, wt, torch.float32, cuda_device, prefill_chunk=320)
        walked = mc.stream_logits(eng, toks, [300])
        eng.split_scan, eng.split_min_rows = True, 2
        for step in (64, 23):
            eng.piece_tokens = step
            for portions in ([300], [64, 65, 2, 100], [130, 1, 2, 3]):
                got = mc.stream_logits(eng, toks, portions)
                assert mc.rel_err(got, ref) < F32_TOL and mc.rel_err(got, walked) < 2e-5
        a, b = eng.open_stream(), eng.open_stream()
        rows = [[], []]
        for k, (na, nb) in enumerate([(100, 5), (70, 1), (2, 1), (128, 13)]):
            at, bt = sum(x.shape[0] for x in rows[0]), sum(x.shape[0] for x in rows[1])
            lg = eng.feed([(a, toks[at:at + na], list(range(na))), (b, other[bt:bt + nb], list(range(nb)))]).double().cpu()
            rows[0].append(lg[:na]); rows[1].append(lg[na:])
        eng.close_stream(a); eng.close_stream(b)
        assert mc.rel_err(torch.cat(rows[0]), ref) < F32_TOL and mc.rel_err(torch.cat(rows[1]), oref) < F32_TOL


@pytest.mark.parametrize("heads,kv,dk,dv,taps", CELLS)
def test_token_step_of_the_gated_delta_rule(cuda_device, heads, kv, dk, dv, taps):
    """The one-kernel token step against the separate kernels and the oracle, behind a prompt, with an idle slot beside it, and
    with the state handed from one path to the other in the middle."""
    config = mc.model([P(window=5, r_heads=heads, r_kv_heads=kv, r_dim=dk, r_vdim=dv, conv=taps)], width=40)
    wt = mc.weights(config, 28)
    wt["l0.mix.left.out"] = mc.bf16_round(wt["l0.mix.left.out"] * 0.1)
    toks = mc.tokens_for(config, 60, seed=23)
    ref = mc.oracle_logits(config, wt, toks)
    eng = mc.build_engine(config, wt, torch.float32, cuda_device)
    assert eng.lib.prl_gated_delta_step_fits(heads, kv, dk, dv, taps)
    assert mc.rel_err(mc.stream_logits(eng, toks, []), ref) < F32_TOL
    eng.unfused_cell = True
    separate = mc.stream_logits(eng, toks, [])
    eng.unfused_cell = False
    assert mc.rel_err(mc.stream_logits(eng, toks, []), separate) < 2e-5
    s, out, at = eng.open_stream(), [], 0
    for k in (7, 1, 1, 1, 2, 1, 1, 20):
        eng.unfused_cell = at % 2 == 0
        out.append(eng.feed([(s, toks[at:at + k], list(range(k)))]))
        at += k
    eng.close_stream(s)
    assert mc.rel_err(torch.cat(out).double().cpu(), ref[:at]) < F32_TOL


@pytest.mark.parametrize("graph", [False, True])
def test_delta_step_of_a_draining_batch(cuda_device, graph):
    """The split of the delta rule's token step goes by the rows that have a token, not by the slots: a batch that drains passes to two
    value heads per CTA (148 SMs: at most 37 rows on 4 q / k heads), its captured step with it, and keeps its bits."""
    from pipelinerl_b200.engine import SamplingParams
    config = mc.model([P(heads=4, kv_heads=2, dim=32, vdim=32, rot_dims=32, window=50, r_heads=8, r_kv_heads=4, r_dim=32, r_vdim=32, conv=4)], width=64)
    wt, got = mc.weights(config, 3), []
    prompts = [mc.tokens_for(config, 3 + i % 5, seed=i) for i in range(44)]
    for all_slots in (False, True):
        eng = mc.build_engine(config, wt, torch.bfloat16, cuda_device, max_batch=44, max_seq_len=64, use_cuda_graph=graph)
        seen, rule = set(), eng._step_plan
        if all_slots:
            eng._live_rows = lambda eng=eng: eng.B
        eng._step_plan = lambda rule=rule, seen=seen: seen.add(rule()) or rule()
        lone = [eng.add_request(p, SamplingParams(max_tokens=3 + 9 * (i % 4 == 0), greedy=True, ignore_eos=True)) for i, p in enumerate(prompts)]
        for _ in range(12):
            eng.step()
            eng.harvest()
        assert not eng.slot_req and (not graph or seen == ({(1,)} if all_slots else {(1,), (2,)}))
        got.append([(list(r.output_ids), list(r.output_logprobs)) for r in lone])
    assert got[0] == got[1] and all(len(ids) == 3 + 9 * (i % 4 == 0) for i, (ids, _) in enumerate(got[0]))


@pytest.mark.parametrize("n,W,F,experts,top", [(1, 64, 72, 4, 2), (33, 200, 136, 5, 3), (300, 96, 128, 16, 4), (7, 20, 12, 3, 1)])
@pytest.mark.parametrize("dtype,act", [(torch.bfloat16, 2), (torch.bfloat16, 1), (torch.float32, 2)])
def test_both_expert_products_in_one_call(cuda_device, dtype, act, n, W, F, experts, top):
    """prl_moe_mlp_act: the bits of prl_moe_gemm_act and prl_moe_gemm, back to back with the grouping that feeds them (several times, so
    that a product that reads its tiles too early would see the former batch's)."""
    from pipelinerl_b200 import _lib
    lib, st, g = _lib.load(), _lib.stream_ptr(), torch.Generator(device="cuda").manual_seed(n + W)
    f32, pairs, i32, ptr = int(dtype == torch.float32), n * top, dict(dtype=torch.int32, device="cuda"), lambda t: t.data_ptr()  # noqa: E731
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    up, down = (rnd(experts * F, W) * W ** -0.5).to(dtype), (rnd(experts * W, F) * F ** -0.5).to(dtype)
    sel, wsel, perm, meta = torch.zeros(pairs, **i32), torch.zeros(pairs, device="cuda"), torch.zeros(pairs, **i32), torch.zeros(4, **i32)
    most = int(lib.prl_moe_max_tiles(pairs, experts))
    tiles, act_out = torch.zeros(3 * most, **i32), torch.zeros(pairs, F, dtype=dtype, device="cuda")
    zs, xs, got = [rnd(n, experts) for _ in range(6)], [rnd(n, W).to(dtype) for _ in range(6)], []
    for together in (False, True):
        outs = [torch.full((pairs, W), float("nan"), device="cuda") for _ in zs]
        for z, x, out in zip(zs, xs, outs):
            _lib.check(lib.prl_moe_choose(ptr(z), experts, None, n, experts, experts, top, 1, 1, 1, 1, 1, 1.3, 64, ptr(sel), ptr(wsel), ptr(perm), ptr(meta),
                                          ptr(tiles), st))
            table = (ptr(perm), ptr(meta), ptr(tiles), most)
            if together:
                _lib.check(lib.prl_moe_mlp_act(ptr(x), f32, n, ptr(up), ptr(down), W, F, *table, act, ptr(wsel), ptr(act_out), ptr(out), st))
            else:
                _lib.check(lib.prl_moe_gemm_act(ptr(x), f32, W, n, ptr(up), f32, F * W, W, *table, F, W, act, ptr(wsel), ptr(act_out), F, st))
                _lib.check(lib.prl_moe_gemm(ptr(act_out), f32, F, 0, ptr(down), f32, W * F, F, *table, W, F, ptr(out), W, 1, st))
        got.append(outs)
    assert all(torch.equal(a, b) and torch.isfinite(a).all() for a, b in zip(*got))


@pytest.mark.parametrize("counts,N,K", [((1,), 8, 8), ((16, 0, 17), 72, 64), ((64, 33, 1, 48), 136, 328), ((5, 64) * 12, 64, 72),
                                        ((2, 3, 9, 16) * 4, 2048, 1000)])
def test_few_rows_per_expert_equal_many(cuda_device, counts, N, K):
    """The grouped product of few rows per expert (tokens given) has the bits of the one of many (gathered rows): tiles of one to 64 rows, remainders
    of its 64 features and 64 channels, more steps than its ring holds."""
    from pipelinerl_b200 import _lib
    lib, st, g = _lib.load(), _lib.stream_ptr(), torch.Generator(device="cuda").manual_seed(N + K)
    i32, ptr, bf16 = dict(dtype=torch.int32, device="cuda"), lambda t: t.data_ptr(), torch.bfloat16  # noqa: E731
    pairs, experts = sum(counts), len(counts)
    n = min(pairs, 3 * experts)
    x, W = torch.randn(n, K, generator=g, device="cuda").to(bf16), torch.randn(experts * N, K, generator=g, device="cuda").to(bf16)
    perm = torch.randperm(pairs, generator=g, device="cuda").to(torch.int32)
    starts = [sum(counts[:e]) for e in range(experts)]
    tiles = torch.tensor([(e, starts[e], c) for e, c in enumerate(counts) if c], **i32)
    meta, wsel = torch.tensor([tiles.shape[0], 0, 0, 0], **i32), torch.rand(pairs, generator=g, device="cuda")
    few, many = (torch.full((pairs, N), float("nan"), device="cuda") for _ in range(2))
    few_act, many_act = (torch.zeros(pairs, N, dtype=bf16, device="cuda") for _ in range(2))
    rows = x[perm.long() % n].contiguous()
    for a, mod, out, act in ((x, n, few, few_act), (rows, 0, many, many_act)):
        table = (ptr(perm), ptr(meta), ptr(tiles), experts)
        _lib.check(lib.prl_moe_gemm(ptr(a), 0, K, mod, ptr(W), 0, N * K, K, *table, N, K, ptr(out), N, 1, st))
        _lib.check(lib.prl_moe_gemm_act(ptr(a), 0, K, mod, ptr(W), 0, N * K, K, *table, N, K, 2, ptr(wsel), ptr(act), N, st))
    assert torch.equal(few, many) and torch.equal(few_act, many_act)
    expert = torch.repeat_interleave(torch.arange(experts, device="cuda"), torch.tensor(counts, device="cuda"))
    want = torch.einsum("sk,snk->sn", rows.double(), W.double().view(experts, N, K)[expert])
    got = few[perm.long()].double()
    assert ((got - want).abs() <= K * 2.0 ** -24 * torch.einsum("sk,snk->sn", rows.double().abs(), W.double().abs().view(experts, N, K)[expert])).all()


@pytest.mark.parametrize("heads,kh,dk,dv", [(16, 8, 128, 128), (4, 2, 64, 48), (6, 2, 20, 36), (4, 4, 32, 64)])
def test_token_step_of_many_rows_equals_few(cuda_device, heads, kh, dk, dv):
    """One value head at a time in a CTA (more than 148 CTAs) or two: the same bits, for outputs, states and convolution inputs."""
    from pipelinerl_b200 import _lib
    lib, g = _lib.load(), torch.Generator(device="cuda").manual_seed(heads)
    n = 148 // kh + 3
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    ch, ptr = 2 * kh * dk + heads * dv, lambda t: t.data_ptr()  # noqa: E731
    P, conv_w, A, dt, gain = rnd(n, ch + heads * dv + 2 * heads), rnd(ch, 4), rnd(heads) * 0.1, rnd(heads), rnd(dv)
    conv0, state0 = rnd(n, ch, 3), rnd(n, heads, dv, dk)
    got = []
    for part in (n, 3):
        conv, state, out = conv0.clone(), state0.clone(), torch.full((n, heads * dv), float("nan"), device="cuda")
        for a in range(0, n, part):
            k = min(part, n - a)
            rows, one = torch.arange(a, a + k, dtype=torch.int32, device="cuda"), torch.ones(k, dtype=torch.int32, device="cuda")
            _lib.check(lib.prl_gated_delta_step(ptr(P), P.shape[1], 0, ch, ch + heads, ch + 2 * heads, ptr(conv_w), 4, ptr(A), ptr(dt), 1e-6, ptr(gain),
                                                1e-5, heads, kh, dk, dv, ptr(rows), ptr(one), ptr(rows), k, ptr(conv), ptr(state), ptr(out), 1,
                                                _lib.stream_ptr()))
        got.append((out, state, conv))
    assert all(torch.equal(a, b) for a, b in zip(*got)) and torch.isfinite(got[0][0]).all()


@pytest.mark.parametrize("heads,kv_heads,window", [(2, 1, 37), (4, 1, 64), (8, 1, 129), (3, 3, 200), (16, 1, 90), (4, 2, 0), (4, 2, 1), (2, 2, 128)])
def test_tcgen05_prompt_attention(cuda_device, heads, kv_heads, window):
    """Heads of 128 in bf16: the tcgen05 prompt kernel with its window, the constant sink and the head gates, against the
    CUDA-core kernel on the same cache and against the oracle.  Portions start inside a page and a key step, rows of a tile
    lose keys of the first step to the window, and steps of a tile may be hidden from some of its rows altogether."""
    config = mc.model([P(heads=heads, kv_heads=kv_heads, dim=128, vdim=128, rot_dims=32, window=window, scale=1.5 * 128 ** -0.5)], width=64)
    wt = mc.weights(config, 9)
    toks = mc.tokens_for(config, 520, seed=3)
    ref = mc.oracle_logits(config, wt, toks)
    eng = mc.build_engine(config, wt, torch.bfloat16, cuda_device, prefill_chunk=520, max_seq_len=576)
    assert eng.tc_prompt[0]
    plans = ([520], [63, 130, 257, 3, 60], [300, 200])                     # the rest one by one
    fast = [mc.stream_logits(eng, toks, p) for p in plans]
    eng.force_plain_attn = True
    eng.lib.prl_attn_any_tensor_cores(0)
    try:
        plain = mc.stream_logits(eng, toks, [520])
    finally:
        eng.lib.prl_attn_any_tensor_cores(1)
    for f in fast:
        assert mc.rel_err(f, plain) < 0.5 * BF16_TOL and mc.rel_err(f, ref) < BF16_TOL
    assert (fast[0] != plain).any()


@pytest.mark.parametrize("shift", [0.0, -150.0, 150.0])
@pytest.mark.parametrize("heads,kv_heads,pos0,rows,window", [(4, 2, 0, 200, 37), (2, 2, 130, 300, 64), (8, 1, 77, 40, 129), (4, 4, 500, 150, 0)])
def test_tcgen05_prompt_attention_alone(cuda_device, shift, heads, kv_heads, pos0, rows, window):
    """The tcgen05 prompt kernel alone, with and without a sink and gates, on scores that are all far below (or far above) zero:
    rows of a tile that see nothing in its first steps must take their reference from the first step they do see."""
    from pipelinerl_b200 import _lib
    lib, d = _lib.load(), cuda_device
    g = torch.Generator().manual_seed(rows)
    S, R = pos0 + rows, heads // kv_heads
    c = torch.sign(torch.randn(128, generator=g))
    q = mc.bf16_round(torch.randn(rows, heads, 128, generator=g) * 0.3 + c * (0.5 if shift else 0.0))
    k = mc.bf16_round(torch.randn(S, kv_heads, 128, generator=g) * 0.3 + c * (shift / 64.0))
    v = mc.bf16_round(torch.randn(S, kv_heads, 128, generator=g))
    sink, gate = torch.randn(heads, generator=g) + shift, torch.randn(rows, heads, generator=g)
    pages = -(-S // 64)
    order = torch.randperm(pages, generator=g) + 1
    kv = torch.zeros(2, pages + 1, kv_heads, 64, 128, dtype=torch.bfloat16)
    for t in range(S):
        kv[0, order[t // 64], :, t % 64], kv[1, order[t // 64], :, t % 64] = k[t].bfloat16(), v[t].bfloat16()
    scale = 1.0                                                             # scores around `shift`
    i32 = dict(dtype=torch.int32, device=d)
    bt = order.int().view(1, -1).to(d)
    one = lambda x: torch.tensor([x], **i32)
    ss, sl, sp, slot = one(0), one(rows), one(pos0), one(0)
    qd, kvd, sd, gd = q.bfloat16().to(d), kv.to(d), sink.to(d), gate.to(d)
    for use in (False, True):
        out = torch.zeros(rows, heads, 128, dtype=torch.bfloat16, device=d)
        _lib.check(lib.prl_paged_attn_prefill_tc_gated(qd.data_ptr(), rows, kvd.data_ptr(), pages + 1, 1, 0, bt.data_ptr(), pages, ss.data_ptr(),
                                                       sl.data_ptr(), sp.data_ptr(), slot.data_ptr(), 1, rows, heads, kv_heads, 128, 64, scale,
                                                       window, sd.data_ptr() if use else None, gd.data_ptr() if use else None, heads,
                                                       out.data_ptr(), _lib.stream_ptr()))
        back = (pos0 + torch.arange(rows))[:, None] - torch.arange(S)[None, :]
        see = (back >= 0) & ((back < window) if window else torch.ones_like(back, dtype=torch.bool))
        ref = torch.zeros(rows, heads, 128, dtype=torch.float64)
        for h in range(heads):
            s = (q[:, h].double() @ k[:, h // R].double().T * scale).masked_fill(~see, -math.inf)
            if use:
                s = torch.cat([s, sink[h].double().expand(rows, 1)], 1)
            w = torch.softmax(s, 1)[:, :S]
            ref[:, h] = w @ v[:, h // R].double() * (torch.sigmoid(gate[:, h].double())[:, None] if use else 1.0)
        err = (out.double().cpu() - ref).abs().max().item()
        assert err < 0.03, (use, err)


def test_long_decoding(cuda_device):
    """A short prompt and 400 single tokens over six page borders and several windows, in fp32 against the oracle."""
    config = mc.model([P(mlp=M(), window=150), P(window=64)])
    wt = mc.weights(config, 31)
    toks = mc.tokens_for(config, 420, seed=12)
    eng = mc.build_engine(config, wt, torch.float32, cuda_device)
    assert mc.rel_err(mc.stream_logits(eng, toks, [20]), mc.oracle_logits(config, wt, toks)) < F32_TOL


def test_greedy_generation_through_the_scheduler(cuda_device):
    """add_request / run_prefill / CUDA-graph token steps / harvest, five prompts on two slots (slots and pages are reused,
    idle slots ride along in the step), greedy ids and log-probabilities of the capped logits against the oracle wherever
    its top-2 margin is not a rounding matter."""
    from pipelinerl_b200.engine import SamplingParams
    wt = mc.weights(FULL, 14)
    eng = mc.build_engine(FULL, wt, torch.float32, cuda_device, max_batch=2, max_seq_len=256, use_cuda_graph=True, prefill_chunk=64)
    prompts = [mc.tokens_for(FULL, n, seed=90 + n) for n in (1, 5, 70, 130, 64)]
    outs = eng.generate(prompts, SamplingParams(max_tokens=6, greedy=True, ignore_eos=True))
    assert len(eng.free_slots) == 2 and len(eng.free_pages) == eng.n_pages - 1
    for p, r in zip(prompts, outs):
        assert len(r.output_ids) == 6 and r.finish_reason == "length"
        seq = list(p)
        for tok, lp in zip(r.output_ids, r.output_logprobs):
            lg = mc.oracle_logits(FULL, wt, seq)[-1]
            top = torch.topk(lg, 2)
            if (top.values[0] - top.values[1]).item() > 1e-3:
                assert tok == top.indices[0].item()
            assert abs(lp - torch.log_softmax(lg, -1)[tok].item()) < 1e-3
            seq.append(tok)


def test_trace_runner_command_line(cuda_device, tmp_path):
    """bin/trace_run on a checkpoint folder: registry, safetensors loader, streams, output files, in both dtypes."""
    config = mc.model([P(mlp=M(experts=4, top=1, ff=8, groups=(2, 1))), P(window=33)], vocab=64, width=40)
    wt = mc.weights(config, 15)
    mc.write_checkpoint(tmp_path, config, wt)
    a, b = mc.tokens_for(config, 90, seed=1), mc.tokens_for(config, 20, seed=2)
    steps = [
        dict(step=0, entries=[dict(id="a", tokens=a[:50], want=[0, 49])], end=[]),
        dict(step=1, entries=[dict(id="a", tokens=a[50:52], want=[]), dict(id="b", tokens=b[:19], want=[3])], end=[]),
        dict(step=2, entries=[dict(id="b", tokens=b[19:], want=[0]), dict(id="a", tokens=a[52:], want=[37])], end=["a", "b"]),
        dict(step=3, entries=[dict(id="c", tokens=b, want=[19])], end=["c"]),
    ]
    gaps = [[], []]
    ra, rb = (mc.oracle_logits(config, wt, t, margins=m) for t, m in zip((a, b), gaps))
    expect = {0: torch.stack([ra[0], ra[49]]), 1: rb[3:4], 2: torch.stack([rb[19], ra[89]]), 3: rb[19:20]}
    root = __import__("pathlib").Path(__file__).resolve().parent.parent
    for dtype, tol in (("float32", F32_TOL), ("bfloat16", BF16_TOL)):
        out = tmp_path / dtype
        p = subprocess.run([sys.executable, str(root / "bin" / "trace_run"), "--model", str(tmp_path), "--dtype", dtype,
                            "--out", str(out), "--max-tokens", "192"], input="\n".join(json.dumps(s) for s in steps) + "\n",
                           capture_output=True, text=True, timeout=900)
        assert p.returncode == 0, p.stderr[-2000:]
        assert [l for l in p.stdout.split("\n") if l.startswith("done")] == [f"done {i}" for i in range(4)]
        import numpy as np
        for i, ref in expect.items():
            got = torch.from_numpy(np.fromfile(out / f"{i}.f32", dtype="<f4")).view(-1, config["vocab"])
            assert got.shape == ref.shape and mc.rel_err(got, ref) < tol


@pytest.mark.parametrize("segs,heads,kh,dk,dv,taps", [((1,), 2, 1, 4, 4, 2), ((5, 1, 2, 9), 4, 2, 128, 128, 4), ((3, 70), 2, 2, 124, 132, 3), ((66,), 2, 1, 256, 260, 4),
                                                       ((7, 2, 30), 3, 3, 20, 300, 2), ((2, 3, 4), 6, 2, 36, 8, 4), ((130,), 16, 8, 128, 128, 3)])
def test_front_rows_of_the_gated_delta_rule(cuda_device, segs, heads, kh, dk, dv, taps):
    """Convolution with carried inputs, SiLU and unit length against 64 bits.  Bound: `taps` products and sums of 2^-24 each relative to
    the sum of magnitudes, a SiLU of a few units of 2^-24 of a slope of at most 1.1, and the same again for the length."""
    from pipelinerl_b200 import _lib
    lib, dev, g = _lib.load(), cuda_device, torch.Generator().manual_seed(sum(segs) + dv)
    n, ns, ch = sum(segs), len(segs), 2 * kh * dk + heads * dv
    ld = (ch + heads * dv + 2 * heads + 3) // 4 * 4
    rnd = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    P, w, conv0 = rnd(n, ld), rnd(ch, taps), rnd(ns, ch, taps - 1)
    starts = [sum(segs[:i]) for i in range(ns)]
    subs = [(i, s + a, min(64, l - a)) for i, (s, l) in enumerate(zip(starts, segs)) for a in range(0, l, 64)]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)  # noqa: E731
    tabs = [i32([i for i, l in enumerate(segs) for _ in range(l)]), i32([t for l in segs for t in range(l)]), i32(starts), i32(list(segs)), i32(list(range(ns))),
            i32([sum(1 for j, _, _ in subs if j < i) for i in range(ns)]), i32([sum(1 for j, _, _ in subs if j == i) for i in range(ns)]),
            i32([s for _, s, _ in subs]), i32([l for _, _, l in subs])]
    f = lambda *s: torch.zeros(*s, device=dev)  # noqa: E731
    on = lambda t: t.to(dev)  # noqa: E731
    Pd, wd, conv, A, dt, gain = on(P), on(w), on(conv0.clone()), on(0.1 * rnd(heads)), on(rnd(heads)), on(rnd(dv))
    C, scr = f(n, ch), f(n * int(lib.prl_gated_delta_split_floats(heads, dk)))
    S0, D, state, out = f(len(subs), heads, dk, dv), f(n, heads * dv), f(ns, heads, dv, dk), f(n, heads * dv)
    p = lambda t: t.data_ptr()  # noqa: E731
    _lib.check(lib.prl_gated_delta_split(p(Pd), ld, 0, ch, ch + heads, ch + 2 * heads, p(wd), taps, p(A), p(dt), 1e-6, p(gain), 1e-5, heads, kh, dk, dv, n,
                                         p(tabs[0]), p(tabs[1]), p(tabs[2]), p(tabs[3]), p(tabs[4]), ns, p(tabs[5]), p(tabs[6]), p(tabs[7]), p(tabs[8]),
                                         len(subs), p(C), p(scr), p(S0), p(D), p(conv), p(state), p(out), 1, _lib.stream_ptr()))
    want, size = torch.empty(n, ch, dtype=torch.float64), torch.empty(n, ch, dtype=torch.float64)
    for i, (s, l) in enumerate(zip(starts, segs)):
        x = torch.cat([conv0[i].double(), P[s:s + l, :ch].double().T], 1)          # [ch, taps - 1 + l]
        t = x.unfold(1, taps, 1) * w.double()[:, None]
        want[s:s + l], size[s:s + l] = torch.nn.functional.silu(t.sum(-1)).T, t.abs().sum(-1).T
    bound = 2.0 ** -24 * ((taps + 2) * size + 8 * want.abs())
    for h in range(2 * kh):
        c = slice(h * dk, (h + 1) * dk)
        length = (want[:, c].square().sum(-1, keepdim=True) + 1e-6).sqrt()
        by = (dk ** -0.5 if h < kh else 1.0) / length
        worst = bound[:, c].norm(dim=-1, keepdim=True) / length                    # of the length, relative
        bound[:, c] = by * (bound[:, c] + want[:, c].abs() * (worst + 2.0 ** -24 * (dk / 16 + 8)))
        want[:, c] *= by
    assert bool(((C.cpu().double() - want).abs() <= bound).all())


@pytest.mark.parametrize("segs,dk", [((640,), 128), ((300, 340), 128), ((640,), 64), ((610, 5), 64)])
def test_gated_delta_rule_of_heads_that_fill_the_chip(cuda_device, segs, dk):
    """16 value heads of ten pieces (more blocks than SMs, so that the next kernels start early) against the first 8 of them by themselves: a head's outputs and
    state depend on its own inputs only, bit for bit, several times over."""
    from pipelinerl_b200 import _lib
    lib, dev, dv, taps, g = _lib.load(), cuda_device, 128, 4, torch.Generator().manual_seed(sum(segs) + dk)
    n, ns = sum(segs), len(segs)
    on = lambda *s: torch.randn(*s, generator=g).to(dev)  # noqa: E731
    q, k, v, gate, b, a = on(n, 8, dk), on(n, 8, dk), on(n, 16, dv), on(n, 16, dv), on(n, 16), on(n, 16)
    wq, wk, wv, A, dt, gain = on(8, dk, taps), on(8, dk, taps), on(16, dv, taps), 0.1 * on(16), on(16), on(dv)
    starts = [sum(segs[:i]) for i in range(ns)]
    subs = [(i, s + c, min(64, l - c)) for i, (s, l) in enumerate(zip(starts, segs)) for c in range(0, l, 64)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)  # noqa: E731
    tabs = [i32([i for i, l in enumerate(segs) for _ in range(l)]), i32([t for l in segs for t in range(l)]), i32(starts), i32(list(segs)), i32(list(range(ns))),
            i32([sum(1 for j, _, _ in subs if j < i) for i in range(ns)]), i32([sum(1 for j, _, _ in subs if j == i) for i in range(ns)]),
            i32([s for _, s, _ in subs]), i32([l for _, _, l in subs])]
    p = lambda t: t.data_ptr()  # noqa: E731

    def run(H):
        kh, ch = H // 2, H * dk + H * dv
        P = torch.cat([q[:, :kh].reshape(n, -1), k[:, :kh].reshape(n, -1), v[:, :H].reshape(n, -1), b[:, :H], a[:, :H], gate[:, :H].reshape(n, -1)], 1).contiguous()
        w = torch.cat([wq[:kh].reshape(-1, taps), wk[:kh].reshape(-1, taps), wv[:H].reshape(-1, taps)]).contiguous()
        f = lambda *s: torch.zeros(*s, device=dev)  # noqa: E731
        C, scr = f(n, ch), f(n * int(lib.prl_gated_delta_split_floats(H, dk)))
        S0, D, conv, state, out = f(len(subs), H, dk, dv), f(n, H * dv), f(ns, ch, taps - 1), f(ns, H, dv, dk), f(n, H * dv)
        _lib.check(lib.prl_gated_delta_split(p(P), P.shape[1], 0, ch, ch + H, ch + 2 * H, p(w), taps, p(A), p(dt), 1e-6, p(gain), 1e-5, H, kh, dk, dv, n,
                                             *(p(t) for t in tabs[:5]), ns, *(p(t) for t in tabs[5:]), len(subs), p(C), p(scr), p(S0), p(D), p(conv), p(state),
                                             p(out), 1, _lib.stream_ptr()))
        return out.view(n, H, dv), state

    want, want_state = run(8)
    assert want.isfinite().all() and want.abs().max() > 0
    for _ in range(4):
        out, state = run(16)
        assert torch.equal(out[:, :8], want) and torch.equal(state[:, :8], want_state)
