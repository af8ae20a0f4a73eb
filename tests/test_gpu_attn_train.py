"""Learner attention on sm_100a (csrc/attn_tc.cu forward, csrc/attn_train.cu backward) against an fp32 reference.

The op: block-diagonal causal attention over one packed row -- what the reference gets from flash-attn varlen
through HF when `position_ids` restart per packed sample (pipelinerl/finetune/rl/__init__.py:204,
conf/finetune/base.yaml:12-13,64).  Reference here: plain fp32 softmax(Q K^T / sqrt(d) + causal mask) V per segment and
head with torch autograd, on the same bf16-representable inputs.  Bar: every output / gradient
element within 2^-7 of the tensor's scale (bf16 P / dS operands + bf16 result rounding); the measured maxima are printed.
The backward must also be bitwise reproducible (fixed-order GQA reduction, no atomics)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

D = 128


def _ops():
    from pipelinerl_b200.learner_body import Ops
    return Ops()


def _reference(qkv, d_out, bounds, n_q, n_kv):
    """fp32 attention + autograd, one (segment, kv head) at a time to bound memory.  Returns out, dqkv (fp32)."""
    T = qkv.shape[0]
    R = n_q // n_kv
    x = qkv.float()
    out = torch.empty(T, n_q * D, device=qkv.device)
    dqkv = torch.zeros_like(x)
    scale = 1.0 / math.sqrt(D)
    for s, e in bounds:
        L = e - s
        mask = torch.ones(L, L, dtype=torch.bool, device=qkv.device).tril()
        for g in range(n_kv):
            kc, vc = (n_q + g) * D, (n_q + n_kv + g) * D
            k = x[s:e, kc:kc + D].clone().requires_grad_(True)
            v = x[s:e, vc:vc + D].clone().requires_grad_(True)
            for r in range(R):
                hq = (g * R + r) * D
                q = x[s:e, hq:hq + D].clone().requires_grad_(True)
                sc = (q @ k.t()) * scale
                p = torch.softmax(sc.masked_fill(~mask, float("-inf")), -1)
                o = p @ v
                out[s:e, hq:hq + D] = o.detach()
                gq, gk, gv = torch.autograd.grad(o, (q, k, v), d_out[s:e, hq:hq + D].float())
                dqkv[s:e, hq:hq + D] = gq
                dqkv[s:e, kc:kc + D] += gk
                dqkv[s:e, vc:vc + D] += gv
                del sc, p, o, gq, gk, gv
    return out, dqkv


def _run(dev, n_q, n_kv, lens, seed=0, pad_cols=0, fwd_gen=2, bwd_gen=None):
    """fwd_gen / bwd_gen: 1 = operands through shared memory, 2 = P / dS handed to the tensor core through TMEM (default);
    bwd_gen 3 = 2 + Q / dO resident in TMEM, 4 = 16 decoupled softmax warps"""
    from pipelinerl_b200 import _lib
    o = _ops()
    bwd_gen = fwd_gen if bwd_gen is None else bwd_gen
    _lib.check(o.lib.prl_attn_set_fwd_generation(fwd_gen))
    _lib.check(o.lib.prl_attn_set_bwd_generation(bwd_gen))
    T = sum(lens)
    g = torch.Generator(device=dev).manual_seed(seed)
    width = (n_q + 2 * n_kv) * D
    buf = torch.randn(T, width + pad_cols, generator=g, device=dev).to(torch.bfloat16)
    qkv = buf[:, :width]                                  # row stride may exceed the logical width
    d_out = torch.randn(T, n_q * D, generator=g, device=dev).to(torch.bfloat16)
    bounds, s = [], 0
    for L in lens:
        bounds.append((s, s + L))
        s += L
    st = torch.tensor([b[0] for b in bounds], dtype=torch.int32, device=dev)
    ln = torch.tensor(lens, dtype=torch.int32, device=dev)
    out, lse = o.attn_fwd(qkv, st, ln, max(lens), n_q, n_kv, D)
    dqkv = o.attn_bwd(qkv, out, d_out, lse, st, ln, max(lens), n_q, n_kv, D)
    dqkv2 = o.attn_bwd(qkv, out, d_out, lse, st, ln, max(lens), n_q, n_kv, D)
    torch.cuda.synchronize()
    assert torch.equal(dqkv, dqkv2), "attention backward is not bitwise reproducible"
    want_out, want_d = _reference(qkv, d_out, bounds, n_q, n_kv)
    res = {}
    err = (out.float() - want_out).abs().max().item() / want_out.abs().max().item()
    res["out"] = err
    # log-sum-exp (log2 domain of the scaled scores) against fp32, spot-checked on the first kv group
    qc, kc = 0, n_q * D
    s0, e0 = bounds[-1]
    sc = (qkv[s0:e0, qc:qc + D].float() @ qkv[s0:e0, kc:kc + D].float().t()) / math.sqrt(D)
    sc = sc.masked_fill(~torch.ones(e0 - s0, e0 - s0, dtype=torch.bool, device=dev).tril(), float("-inf"))
    want_lse = torch.logsumexp(sc, -1) / math.log(2.0)
    res["lse"] = (lse[s0:e0, 0] - want_lse).abs().max().item()
    qe, ke = n_q * D, (n_q + n_kv) * D
    for name, a, b in (("dq", 0, qe), ("dk", qe, ke), ("dv", ke, width)):
        scale = max(want_d[:, a:b].abs().max().item(), 1e-3)      # a single-token segment has dq = dk = 0 exactly
        res[name] = (dqkv[:, a:b].float() - want_d[:, a:b]).abs().max().item() / scale
    _lib.check(o.lib.prl_attn_set_fwd_generation(2))
    _lib.check(o.lib.prl_attn_set_bwd_generation(4))
    print(f"[attn_train fwd gen{fwd_gen} bwd gen{bwd_gen}] n_q={n_q} n_kv={n_kv} lens={lens if len(lens) < 8 else str(lens[:6]) + '...'}: " +
          " ".join(f"{k}={v:.2e}" for k, v in res.items()))
    assert res["out"] <= 2 ** -7, res
    assert res["lse"] <= 2e-3, res
    for k in ("dq", "dk", "dv"):
        assert res[k] <= 2 ** -7, res
    assert torch.isfinite(dqkv.float()).all() and torch.isfinite(out.float()).all()
    return res


@pytest.mark.parametrize("n_q,n_kv,lens", [
    (4, 2, [1]),                       # a single token
    (4, 2, [5, 1, 3]),
    (7, 1, [64]),
    (7, 1, [130, 17, 300, 1, 64]),     # ragged: tiles straddle segment ends
    (2, 2, [257]),                     # R = 1
    (4, 1, [200, 56]),
    (5, 1, [129, 383]),                # Qwen2.5-32B's 5:1 grouping
    (16, 1, [96, 33]),
    (28, 4, [511, 1, 700]),
])
@pytest.mark.parametrize("fwd_gen,bwd_gen", [(1, 1), (2, 2), (2, 3), (2, 4)])
def test_varlen_attention_small(cuda_device, n_q, n_kv, lens, fwd_gen, bwd_gen):
    _run(cuda_device, n_q, n_kv, lens, seed=len(lens) * 131 + n_q, fwd_gen=fwd_gen, bwd_gen=bwd_gen)


def test_varlen_attention_padded_row_stride(cuda_device):
    _run(cuda_device, 7, 1, [100, 250], seed=3, pad_cols=64)


@pytest.mark.parametrize("lens", [[2048, 2048], [4096], [3000, 5, 1091]])
def test_varlen_attention_qwen7b_heads_medium(cuda_device, lens):
    _run(cuda_device, 28, 4, lens, seed=11)


@pytest.mark.parametrize("lens,fwd_gen,bwd_gen", [([16384], 2, 2), ([8192, 8192], 2, 2), ([5000, 11000, 384], 2, 2),
                                                  ([16384], 1, 1), ([16384], 2, 1), ([16384], 1, 2), ([16384], 2, 3),
                                                  ([5000, 11000, 384], 2, 3), ([16384], 2, 4), ([8192, 8192], 2, 4),
                                                  ([5000, 11000, 384], 2, 4)])
def test_varlen_attention_qwen7b_heads_16k(cuda_device, lens, fwd_gen, bwd_gen):
    """the trainer's micro-batch size (16 384 packed tokens) at Qwen2.5-7B's 28 / 4 heads"""
    _run(cuda_device, 28, 4, lens, seed=5, fwd_gen=fwd_gen, bwd_gen=bwd_gen)


def test_attention_output_rows_outside_every_segment_are_untouched(cuda_device):
    """rows not covered by a segment are never written (the body always covers the row; this pins the bounds logic)"""
    o = _ops()
    dev = cuda_device
    n_q, n_kv, T = 4, 2, 300
    width = (n_q + 2 * n_kv) * D
    qkv = torch.randn(T, width, device=dev).to(torch.bfloat16)
    st = torch.tensor([10], dtype=torch.int32, device=dev)
    ln = torch.tensor([200], dtype=torch.int32, device=dev)
    out, lse = o.attn_fwd(qkv, st, ln, 200, n_q, n_kv, D)
    ref, _ = o.attn_fwd(qkv[10:210].contiguous(), torch.zeros(1, dtype=torch.int32, device=dev), ln, 200, n_q, n_kv, D)
    assert torch.equal(out[10:210], ref)


@pytest.mark.parametrize("n_q,n_kv,lens,sp", [
    (4, 2, [5, 1, 3, 7], 2),
    (7, 1, [130, 17, 300, 1, 64], 2),          # slices start in the middle of a sample
    (28, 4, [511, 1, 700, 836], 4),
    (5, 1, [129, 383], 4),
    (28, 4, [16384], 2),                        # one 16 384-token sample over two ranks
    (28, 4, [5000, 11000, 384], 4),
])
def test_sequence_parallel_slices_match_full_attention(cuda_device, n_q, n_kv, lens, sp):
    """prl_attn_varlen_fwd_kv / _bwd_kv (the sequence-parallel learner, reference finetune_loop.py:507-517 + make_slices
    finetune/types.py:145-180): every rank's slice of queries against the gathered K / V reproduces its rows of the
    single-rank result bit for bit (out, lse, dQ), and the ranks' dK / dV contributions sum to the single-rank dK / dV."""
    from pipelinerl_b200.learner_body import NativeBody
    o = _ops()
    dev = cuda_device
    D = 128
    T = sum(lens)
    assert T % sp == 0
    g = torch.Generator(device=dev).manual_seed(7 + T)
    qkv = torch.randn(T, (n_q + 2 * n_kv) * D, generator=g, device=dev).to(torch.bfloat16)
    d_out = torch.randn(T, n_q * D, generator=g, device=dev).to(torch.bfloat16)
    st = torch.tensor([sum(lens[:i]) for i in range(len(lens))], dtype=torch.int32, device=dev)
    ln = torch.tensor(lens, dtype=torch.int32, device=dev)
    out, lse = o.attn_fwd(qkv, st, ln, max(lens), n_q, n_kv, D)
    dqkv = o.attn_bwd(qkv, out, d_out, lse, st, ln, max(lens), n_q, n_kv, D)
    qe = n_q * D
    kv = qkv[:, qe:].contiguous()
    pos = torch.cat([torch.arange(l) for l in lens])
    dkv_sum = torch.zeros(T, 2 * n_kv * D, dtype=torch.float32, device=dev)
    Tl = T // sp
    for r in range(sp):
        a, b = r * Tl, (r + 1) * Tl
        segs = NativeBody.sp_segments(pos[a:b], a, dev)
        out_r, lse_r = o.attn_fwd_kv(qkv[a:b], kv, segs, n_q, n_kv, D)
        assert torch.equal(out_r, out[a:b]), f"rank {r}: forward rows differ from the single-rank result"
        assert torch.equal(lse_r, lse[a:b])
        dq_r = torch.empty(Tl, qe, dtype=torch.bfloat16, device=dev)
        dkv_r = o.attn_bwd_kv(qkv[a:b], kv, out_r, d_out[a:b].contiguous(), lse_r, segs, n_q, n_kv, D, dq_r)
        assert torch.equal(dq_r, dqkv[a:b, :qe]), f"rank {r}: dQ rows differ from the single-rank result"
        assert torch.all(dkv_r[b:] == 0), "keys after the slice's last query must receive no gradient"
        dkv_sum += dkv_r.float()
    want = dqkv[:, qe:].float()
    scale = max(want.abs().max().item(), 1e-3)
    err = (dkv_sum - want).abs().max().item() / scale
    print(f"[attn sp={sp}] n_q={n_q} n_kv={n_kv} lens={lens}: sum of rank dK/dV vs single rank rel {err:.2e}")
    assert err <= 2 ** -7, err


@pytest.mark.parametrize("n_q,n_kv,lens", [
    (16, 1, [1500, 3]),        # eight CTAs per key tile
    (5, 1, [700, 20]),         # four; shares of one or two steps in the short sample, empty ones at the end of the long one
    (14, 2, [900, 130, 129]),  # two to four
    (28, 4, [300]),
    (64, 1, [70, 1]),          # one query token per step
])
def test_varlen_backward_with_shared_key_tiles(cuda_device, n_q, n_kv, lens):
    """Several CTAs share a key tile's queries: gradients against the oracle, and the same bits in every run."""
    _run(cuda_device, n_q, n_kv, lens, seed=17, fwd_gen=2, bwd_gen=4)
    o, T = _ops(), sum(lens)
    g = torch.Generator().manual_seed(1)
    qkv = torch.randn(T, (n_q + 2 * n_kv) * 128, generator=g).to(torch.bfloat16).to(cuda_device)
    d = torch.randn(T, n_q * 128, generator=g).to(torch.bfloat16).to(cuda_device)
    st = torch.tensor([sum(lens[:i]) for i in range(len(lens))], dtype=torch.int32, device=cuda_device)
    ln = torch.tensor(lens, dtype=torch.int32, device=cuda_device)
    shape = (st, ln, max(lens), n_q, n_kv, 128)
    out, lse = o.attn_fwd(qkv, *shape)
    first = o.attn_bwd(qkv, out, d, lse, *shape)
    assert all(torch.equal(first, o.attn_bwd(qkv, out, d, lse, *shape)) for _ in range(3))


@pytest.mark.parametrize("gen", [1, 2, 3, 4])
def test_varlen_backward_keeps_its_bits_with_cold_row_statistics(cuda_device, gen):
    """The first sub-tile's log-sum-exp and delta come from far memory in one run and from L2 in the next: the softmax threads meet
    after they are stored, so none reads an entry before it is there."""
    from pipelinerl_b200 import _lib
    o, lens, n_q, n_kv = _ops(), [700, 129, 64, 1, 300], 14, 2
    T, g = sum(lens), torch.Generator().manual_seed(gen)
    qkv = torch.randn(T, (n_q + 2 * n_kv) * 128, generator=g).to(torch.bfloat16).to(cuda_device)
    d = torch.randn(T, n_q * 128, generator=g).to(torch.bfloat16).to(cuda_device)
    st = torch.tensor([sum(lens[:i]) for i in range(len(lens))], dtype=torch.int32, device=cuda_device)
    shape = (st, torch.tensor(lens, dtype=torch.int32, device=cuda_device), max(lens), n_q, n_kv, 128)
    out, lse = o.attn_fwd(qkv, *shape)
    flush = torch.empty(1 << 28, dtype=torch.uint8, device=cuda_device)
    _lib.check(o.lib.prl_attn_set_bwd_generation(gen))
    try:
        runs = []
        for i in range(8):
            if i % 2:
                flush.zero_()
            runs.append(o.attn_bwd(qkv, out, d, lse, *shape))
        torch.cuda.synchronize()
    finally:
        _lib.check(o.lib.prl_attn_set_bwd_generation(4))
    assert all(torch.equal(runs[0], r) for r in runs[1:])


@pytest.mark.parametrize("n_q,n_kv,lens", [(14, 2, [1, 700, 0, 18, 19, 300]), (4, 4, [0, 128, 129, 1, 0]), (5, 1, [3] * 31 + [40, 0, 26, 1, 77] + [2] * 40),
                                           (8, 2, [64])])
def test_listed_tiles_equal_each_sample_alone(cuda_device, n_q, n_kv, lens):
    """Forward and dQ launch the tiles that are there, found in a list of the samples (where that pays): the bits of each sample by
    itself, for samples of no tokens, of one tile exactly and one more, and for more samples than a warp looks at together."""
    from pipelinerl_b200 import _lib
    lib, st, g = _lib.load(), _lib.stream_ptr(), torch.Generator(device="cuda").manual_seed(sum(lens))
    T, width, ptr = sum(lens), (n_q + 2 * n_kv) * 128, lambda t: t.data_ptr()  # noqa: E731
    qkv = torch.randn(T, width, generator=g, device="cuda").bfloat16()
    d_out = torch.randn(T, n_q * 128, generator=g, device="cuda").bfloat16()
    starts = [sum(lens[:i]) for i in range(len(lens))]

    def run(picked):
        out = torch.zeros(T, n_q * 128, dtype=torch.bfloat16, device="cuda")
        lse, dqkv, ws = torch.zeros(T, n_q, device="cuda"), torch.zeros_like(qkv), torch.empty(T * n_q, device="cuda")
        start, length = (torch.tensor([v[i] for i in picked], dtype=torch.int32, device="cuda") for v in (starts, lens))
        seg = (ptr(start), ptr(length), len(picked), max(max(lens[i] for i in picked), 1), n_q, n_kv, 128, 128 ** -0.5)
        _lib.check(lib.prl_attn_varlen_fwd(ptr(qkv), width, T, *seg, ptr(out), ptr(lse), st))
        _lib.check(lib.prl_attn_varlen_bwd(ptr(qkv), width, T, *seg, ptr(out), ptr(d_out), ptr(lse), ptr(dqkv), width, ptr(ws), ws.numel() * 4, st))
        return out, lse, dqkv[:, :n_q * 128]
    together = run(list(range(len(lens))))
    for i, k in enumerate(lens):
        if k and (len(lens) < 10 or i % 7 == 0 or k > 3):
            rows = slice(starts[i], starts[i] + k)
            assert all(torch.equal(a[rows], b[rows]) for a, b in zip(together, run([i])))
    assert all(torch.isfinite(t.float()).all() for t in together)


@pytest.mark.parametrize("n_q,n_kv,lens,listed", [(14, 2, [1, 700, 0, 18, 19, 300], True), (4, 4, [0, 128, 129, 1, 0, 1500, 3], True),
                                                  (5, 1, [3] * 31 + [40, 0, 26, 1, 77] + [2] * 40, True), (14, 2, [40, 0, 17, 37, 18, 1] * 12, False)])
def test_tiles_of_packed_samples_equal_each_sample_alone(cuda_device, n_q, n_kv, lens, listed):
    """Outputs and all gradients of samples packed together against each sample alone, where the tiles are listed and where they are not.
    dK and dV of a sample alone may be summed in another order (more CTAs share a key tile): fp32 partial sums rounded once to bf16 on
    either side, 2 * 2^-9 of the norm."""
    from pipelinerl_b200 import _lib
    from pipelinerl_b200.learner_body import Ops
    o, g = Ops(), torch.Generator(device="cuda").manual_seed(sum(lens))
    assert (_lib.load().prl_attn_listed_tiles(sum(lens), max(lens), len(lens), n_q, n_kv) > 0) == listed
    qkv = torch.randn(sum(lens), (n_q + 2 * n_kv) * 128, generator=g, device="cuda").bfloat16()
    d_out = torch.randn(sum(lens), n_q * 128, generator=g, device="cuda").bfloat16()
    tables = lambda st, ln: tuple(torch.tensor(v, dtype=torch.int32, device="cuda") for v in (st, ln))  # noqa: E731
    starts, q = [sum(lens[:i]) for i in range(len(lens))], n_q * 128
    shape = (*tables(starts, lens), max(lens), n_q, n_kv, 128)
    out, lse = o.attn_fwd(qkv, *shape)
    dqkv = o.attn_bwd(qkv, out, d_out, lse, *shape)
    for i, n in enumerate(lens):
        if n == 0 or (len(lens) > 10 and i % 7 and n <= 3):
            continue
        rows = slice(starts[i], starts[i] + n)
        shape = (*tables([0], [n]), n, n_q, n_kv, 128)
        out1, lse1 = o.attn_fwd(qkv[rows], *shape)
        dqkv1 = o.attn_bwd(qkv[rows], out1, d_out[rows].contiguous(), lse1, *shape)
        assert torch.equal(out[rows], out1) and torch.equal(lse[rows], lse1) and torch.equal(dqkv[rows, :q], dqkv1[:, :q])
        both = [t[:, q:].float() for t in (dqkv[rows], dqkv1)]
        assert (both[0] - both[1]).norm() <= 2.0 ** -8 * both[1].norm() + 1e-6
