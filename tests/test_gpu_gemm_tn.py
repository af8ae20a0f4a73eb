"""CTA-pair persistent tcgen05 GEMM of the learner body (csrc/gemm_tn.cu) against fp32 torch matmuls of the
same bf16 operands.  Tolerance: fp32 accumulation of bf16 products (1e-4 of the output scale) plus one bf16
rounding (2^-8 relative) where the output is bf16."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def gemm_tn(A, B, out_dtype=torch.bfloat16, bias=None, residual=None, acc_into=None, alpha=1.0):
    from pipelinerl_b200 import _lib
    lib = _lib.load()
    M, K = A.shape
    N = B.shape[0]
    if acc_into is not None:
        C = acc_into
    else:
        C = torch.full((M, N), float("nan"), dtype=out_dtype, device=A.device)
    _lib.check(lib.prl_gemm_tn(A.data_ptr(), A.stride(0), B.data_ptr(), B.stride(0), M, N, K, C.data_ptr(), C.stride(0),
                               int(C.dtype == torch.float32), int(acc_into is not None),
                               bias.data_ptr() if bias is not None else None,
                               residual.data_ptr() if residual is not None else None,
                               residual.stride(0) if residual is not None else 0, alpha, _lib.stream_ptr()))
    torch.cuda.synchronize()
    return C


SHAPES = [(1, 8, 8), (256, 256, 64), (129, 130, 72), (300, 777, 200), (1024, 4608, 3584), (2048, 3584, 18944),
          (4608, 3584, 4096), (5000, 1000, 1288), (16, 37888, 512), (777, 24, 136)]


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_gemm_tn_f32_out(cuda_device, M, N, K):
    g = torch.Generator().manual_seed(M * 31 + N * 7 + K)
    A = (torch.randn(M, K, generator=g) * 0.5).to(torch.bfloat16).to(cuda_device)
    B = (torch.randn(N, K, generator=g) * 0.05).to(torch.bfloat16).to(cuda_device)
    got = gemm_tn(A, B, out_dtype=torch.float32)
    want = A.float() @ B.float().t()
    assert torch.isfinite(got).all(), "unwritten output"
    assert (got - want).abs().max().item() <= 2e-4 * want.abs().max().item() + 1e-6


@pytest.mark.parametrize("M,N,K", [(300, 776, 200), (1024, 4608, 3584), (513, 100, 64)])
def test_gemm_tn_bf16_bias_residual(cuda_device, M, N, K):
    g = torch.Generator().manual_seed(5)
    A = (torch.randn(M, K, generator=g) * 0.5).to(torch.bfloat16).to(cuda_device)
    B = (torch.randn(N, K, generator=g) * 0.05).to(torch.bfloat16).to(cuda_device)
    bias = torch.randn(N, generator=g).to(torch.bfloat16).to(cuda_device)
    res = torch.randn(M, N, generator=g).to(torch.bfloat16).to(cuda_device)
    got = gemm_tn(A, B, bias=bias, residual=res)
    want = A.float() @ B.float().t() + bias.float() + res.float()
    scale = want.abs().max().item()
    assert (got.float() - want).abs().max().item() <= (2e-4 + 2 ** -8) * scale
    plain = gemm_tn(A, B)
    assert torch.equal(plain, (A.float() @ B.float().t()).to(torch.bfloat16)) or \
        (plain.float() - A.float() @ B.float().t()).abs().max().item() <= (2e-4 + 2 ** -8) * scale


def test_gemm_tn_accumulates_and_strided_operands(cuda_device):
    """wgrad form: fp32 C += A * B^T with operands that are column slices of wider buffers."""
    g = torch.Generator().manual_seed(9)
    big_a = torch.randn(640, 1024, generator=g).to(torch.bfloat16).to(cuda_device)
    big_b = torch.randn(384, 1024, generator=g).to(torch.bfloat16).to(cuda_device)
    A, B = big_a[:, 128:128 + 520], big_b[:, 256:256 + 520]
    C = torch.randn(640, 384, generator=g).to(cuda_device)
    want = C + 0.5 * (A.float() @ B.float().t())
    got = gemm_tn(A, B, acc_into=C, alpha=0.5)
    assert (got - want).abs().max().item() <= 2e-4 * want.abs().max().item()


def test_gemm_tn_is_deterministic(cuda_device):
    g = torch.Generator().manual_seed(1)
    A = torch.randn(3000, 2048, generator=g).to(torch.bfloat16).to(cuda_device)
    B = torch.randn(1500, 2048, generator=g).to(torch.bfloat16).to(cuda_device)
    assert torch.equal(gemm_tn(A, B), gemm_tn(A, B))


@pytest.mark.parametrize("R,C", [(1, 1), (64, 64), (100, 37), (4096, 3584), (777, 1288)])
def test_transpose_bf16(cuda_device, R, C):
    from pipelinerl_b200 import _lib
    lib = _lib.load()
    x = torch.randn(R, C, device=cuda_device).to(torch.bfloat16)
    out = torch.empty(C, R, dtype=torch.bfloat16, device=cuda_device)
    _lib.check(lib.prl_transpose_bf16(x.data_ptr(), R, C, x.stride(0), out.data_ptr(), out.stride(0), _lib.stream_ptr()))
    torch.cuda.synchronize()
    assert torch.equal(out, x.t().contiguous())


def test_gemm_tn_rejects_bad_arguments(cuda_device):
    from pipelinerl_b200 import _lib
    lib = _lib.load()
    A = torch.zeros(16, 20, dtype=torch.bfloat16, device=cuda_device)
    C = torch.zeros(16, 16, dtype=torch.bfloat16, device=cuda_device)
    rc = lib.prl_gemm_tn(A.data_ptr(), 20, A.data_ptr(), 20, 16, 16, 20, C.data_ptr(), 16, 0, 0, None, None, 0, 1.0,
                         _lib.stream_ptr())
    assert rc != 0 and b"multiples of 8" in lib.prl_last_error()
    rc = lib.prl_gemm_tn(A.data_ptr(), 24, A.data_ptr(), 24, 16, 16, 16, C.data_ptr(), 16, 0, 1, None, None, 0, 1.0,
                         _lib.stream_ptr())
    assert rc != 0 and b"accumulate" in lib.prl_last_error()


def gemm_ex(A, a_mn, B, b_mn, M, N, K, out_dtype=torch.float32, acc_into=None):
    """A given as [K, M] when a_mn else [M, K]; B as [K, N] when b_mn else [N, K]."""
    from pipelinerl_b200 import _lib
    lib = _lib.load()
    C = acc_into if acc_into is not None else torch.full((M, N), float("nan"), dtype=out_dtype, device=A.device)
    _lib.check(lib.prl_gemm_ex(A.data_ptr(), A.stride(0), int(a_mn), B.data_ptr(), B.stride(0), int(b_mn), M, N, K,
                               C.data_ptr(), C.stride(0), int(C.dtype == torch.float32), int(acc_into is not None), None,
                               None, 0, 1.0, _lib.stream_ptr()))
    torch.cuda.synchronize()
    return C


@pytest.mark.parametrize("a_mn,b_mn", [(False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (304, 776, 200), (1000, 520, 1288), (4608, 3584, 2048), (24, 72, 136)])
def test_gemm_mn_major_operands(cuda_device, M, N, K, a_mn, b_mn):
    """dgrad reads W as stored (B MN-major), wgrad reads dY and X as stored (both MN-major): no transposed copies."""
    g = torch.Generator().manual_seed(M + N + K)
    A = (torch.randn(M, K, generator=g) * 0.5).to(torch.bfloat16).to(cuda_device)
    B = (torch.randn(N, K, generator=g) * 0.05).to(torch.bfloat16).to(cuda_device)
    want = A.float() @ B.float().t()
    got = gemm_ex(A.t().contiguous() if a_mn else A, a_mn, B.t().contiguous() if b_mn else B, b_mn, M, N, K)
    assert torch.isfinite(got).all()
    assert (got - want).abs().max().item() <= 2e-4 * want.abs().max().item() + 1e-6
    ref = gemm_ex(A, False, B, False, M, N, K)
    assert torch.equal(got, ref)    # same products, same k order: bitwise equal to the K-major path


@pytest.mark.parametrize("T,K,I", [(300, 512, 1024), (257, 896, 1152), (1024, 3584, 18944), (5, 256, 128)])
def test_gemm_swiglu_epilogue_is_bit_identical_to_gemm_plus_silu(cuda_device, T, K, I):
    """gate_up GEMM with SiLU(gate) * up in its epilogue (prl_gemm_swiglu: the pair's two CTAs stage the gate rows and the up
    rows of the same 128 features) == prl_gemm_ex followed by prl_silu_mul_fwd, bit for bit, for both outputs."""
    from pipelinerl_b200.learner_body import Ops
    o = Ops()
    g = torch.Generator(device=cuda_device).manual_seed(T + K + I)
    x = (torch.randn(T, K, generator=g, device=cuda_device) * 0.5).to(torch.bfloat16)
    W = (torch.randn(2 * I, K, generator=g, device=cuda_device) * K ** -0.5).to(torch.bfloat16)
    gu_ref = o.gemm(x, W)
    act_ref = o.silu_mul(gu_ref)
    gu, act = o.gemm_swiglu(x, W, need_gate_up=True)
    torch.cuda.synchronize()
    assert torch.equal(gu, gu_ref) and torch.equal(act, act_ref)
    none, act2 = o.gemm_swiglu(x, W, need_gate_up=False)
    assert none is None and torch.equal(act2, act_ref)
    # and against fp32 math
    ref = x.float() @ W.float().t()
    want = torch.nn.functional.silu(ref[:, :I]) * ref[:, I:]
    assert (act.float() - want).abs().max().item() <= 2 ** -6 * want.abs().max().item()


@pytest.mark.parametrize("T,K,I", [(1024, 512, 256), (1000, 896, 1152), (130, 256, 128)])
def test_gemm_swiglu_f32_is_bit_identical_to_fp32_gemm_plus_sampler_silu(cuda_device, T, K, I):
    """The sampler's chunked prefill (engine.py): prl_gemm_swiglu_f32 == prl_gemm_tn with an fp32 output followed by
    prl_silu_mul (the token step's own SiLU(gate) * up of fp32 values), bit for bit -- the fusion removes the [T, 2I] fp32
    round trip, not a rounding point."""
    from pipelinerl_b200 import _lib
    lib = _lib.load()
    dev = cuda_device
    g = torch.Generator(device=dev).manual_seed(T + K + I)
    x = (torch.randn(T, K, generator=g, device=dev) * 0.5).to(torch.bfloat16)
    W = (torch.randn(2 * I, K, generator=g, device=dev) * K ** -0.5).to(torch.bfloat16)
    part = torch.empty(T, 2 * I, dtype=torch.float32, device=dev)
    _lib.check(lib.prl_gemm_tn(x.data_ptr(), K, W.data_ptr(), K, T, 2 * I, K, part.data_ptr(), 2 * I, 1, 0, None, None, 0, 1.0,
                               _lib.stream_ptr()))
    act_ref = torch.empty(T, I, dtype=torch.bfloat16, device=dev)
    _lib.check(lib.prl_silu_mul(part.data_ptr(), 1, T, I, act_ref.data_ptr(), None, 0, _lib.stream_ptr()))
    act = torch.empty(T, I, dtype=torch.bfloat16, device=dev)
    _lib.check(lib.prl_gemm_swiglu_f32(x.data_ptr(), K, W.data_ptr(), K, T, I, K, act.data_ptr(), I, _lib.stream_ptr()))
    torch.cuda.synchronize()
    assert torch.equal(act, act_ref)
    ref = x.float() @ W.float().t()
    want = torch.nn.functional.silu(ref[:, :I]) * ref[:, I:]
    assert (act.float() - want).abs().max().item() <= 2 ** -7 * want.abs().max().item()


@pytest.mark.parametrize("M,V,K,with_lo,with_ent", [(300, 1031, 256, True, True), (2048, 4096, 512, True, False),
                                                     (130, 777, 128, False, True), (1, 520, 64, True, True)])
def test_head_dlogits_without_materialised_logits(cuda_device, M, V, K, with_lo, with_ent):
    """prl_head_dlogits: the head GEMM (hi + lo weight streams in one TMEM accumulation) with the backward of
    log-softmax / entropy in its epilogue, bf16 d logits out.  Against fp32 torch autograd through logits / T ->
    log_softmax -> (target logprob, entropy) on the same bf16 inputs, and the statistics of prl_head_logprob as inputs."""
    from pipelinerl_b200 import _lib
    lib = _lib.load()
    dev = cuda_device
    g = torch.Generator(device=dev).manual_seed(M + V + K)
    T = 0.7
    x = (torch.randn(M, K, generator=g, device=dev) * 0.7).to(torch.bfloat16)
    Wf = torch.randn(V, K, generator=g, device=dev) * K ** -0.5
    W = Wf.to(torch.bfloat16)
    W_lo = (Wf - W.float()).to(torch.bfloat16) if with_lo else None
    tg = torch.randint(0, V, (M,), generator=g, device=dev)
    g_lp = torch.randn(M, generator=g, device=dev)
    g_ent = torch.randn(M, generator=g, device=dev) * 0.3 if with_ent else None
    lp = torch.empty(M, device=dev)
    ent, lse = torch.empty_like(lp), torch.empty_like(lp)
    ws = torch.empty(int(lib.prl_head_workspace_bytes(M, V)), dtype=torch.uint8, device=dev)
    _lib.check(lib.prl_head_logprob(W.data_ptr(), W_lo.data_ptr() if with_lo else None, x.data_ptr(), M, V, K, T, tg.data_ptr(),
                                    1, 0, 0, lp.data_ptr(), ent.data_ptr(), lse.data_ptr(), None, None, ws.data_ptr(), ws.numel(),
                                    _lib.stream_ptr()))
    ld = (V + 7) // 8 * 8
    dz = torch.zeros(M, ld, dtype=torch.bfloat16, device=dev)
    _lib.check(lib.prl_head_dlogits(W.data_ptr(), W_lo.data_ptr() if with_lo else None, x.data_ptr(), M, V, K, T, tg.data_ptr(),
                                    lse.data_ptr(), ent.data_ptr(), g_lp.data_ptr(), g_ent.data_ptr() if with_ent else None,
                                    dz.data_ptr(), ld, _lib.stream_ptr()))
    torch.cuda.synchronize()
    Wsum = W.float() + (W_lo.float() if with_lo else 0.0)
    z = (x.float() @ Wsum.t()).requires_grad_(True)
    ls = torch.log_softmax(z / T, -1)
    obj = (ls.gather(1, tg[:, None])[:, 0] * g_lp).sum()
    if with_ent:
        obj = obj + ((-(ls.exp() * ls).sum(-1)) * g_ent).sum()
    obj.backward()
    want = z.grad
    err = (dz[:, :V].float() - want).abs().max().item() / want.abs().max().item()
    print(f"[head dlogits M={M} V={V} K={K} lo={with_lo} ent={with_ent}] rel max err {err:.2e}")
    assert err <= 2 ** -7
    if ld > V:
        assert torch.count_nonzero(dz[:, V:]) == 0      # padding columns are not touched


@pytest.mark.parametrize("T,H,I", [(300, 512, 1024), (257, 896, 1152), (1024, 3584, 18944), (5, 256, 160)])
def test_dgrad_with_silu_backward_epilogue_is_bit_identical(cuda_device, T, H, I):
    """prl_gemm_dgrad_swiglu (down_proj dgrad whose epilogue applies the backward of SiLU(gate) * up) == prl_gemm_ex with the
    weight read as stored followed by prl_silu_mul_bwd, bit for bit."""
    from pipelinerl_b200.learner_body import Ops
    o = Ops()
    g = torch.Generator(device=cuda_device).manual_seed(T + H + I)
    dY = (torch.randn(T, H, generator=g, device=cuda_device) * 0.5).to(torch.bfloat16)
    W = (torch.randn(H, I, generator=g, device=cuda_device) * H ** -0.5).to(torch.bfloat16)
    gu = torch.randn(T, 2 * I, generator=g, device=cuda_device).to(torch.bfloat16)
    want = o.silu_mul_bwd(gu, o.dgrad(dY, W))
    got = o.dgrad_swiglu(dY, W, gu)
    torch.cuda.synchronize()
    assert torch.equal(got, want)


# one shape per tile width that the width rule takes on 148 SMs (noted), columns that end inside a 32-column chunk and a 4-column
# piece, rows that end inside a tile; the strides of C make its rows 16-byte aligned or not
@pytest.mark.parametrize("M,N,K,b_mn,pad", [
    (4096, 3581, 192, False, 3),    # 208
    (1000, 3578, 72, False, 2),     # 208
    (3070, 2045, 136, False, 0),    # 176, rows of C not 16-byte aligned
    (4000, 2048, 64, False, 8),     # 240
    (1024, 8226, 64, False, 6),     # 224
    (452, 3584, 128, False, 0),     # 112
    (200, 2041, 72, False, 7),      # 64
    (1, 24, 8, False, 0),           # 64
    (2048, 3576, 136, True, 0),     # 224, MN-major B
    (1000, 2040, 64, True, 4),      # 128
    (130, 1016, 72, True, 1),       # 64
    (3072, 2048, 64, True, 0),      # 192
])
def test_gemm_output_widths_and_epilogues(cuda_device, M, N, K, b_mn, pad):
    """plain fp32, fp32 accumulate, bf16 + bias + residual over the widths of the output tiles.  fp32: products of bf16 sum to
    within K * 2^-24 of the sum of their magnitudes; bf16: one more rounding of the result."""
    from pipelinerl_b200 import _lib
    lib = _lib.load()
    g = torch.Generator().manual_seed(M + N + K)
    A = torch.randn(M, K, generator=g).to(torch.bfloat16).to(cuda_device)
    B = torch.randn(N, K, generator=g).to(torch.bfloat16).to(cuda_device)
    Bs = B.T.contiguous() if b_mn else B
    want = A.double() @ B.double().T
    slack = K * 2.0 ** -24 * (A.double().abs() @ B.double().abs().T) + 1e-12
    old = torch.randn(M, N, generator=g).to(cuda_device)
    bias = torch.randn(N, generator=g).to(torch.bfloat16).to(cuda_device)
    res = torch.randn(M, N + pad, generator=g).to(torch.bfloat16).to(cuda_device)[:, :N]

    def run(C, acc=0, bias=None, res=None, alpha=1.0):
        _lib.check(lib.prl_gemm_ex(A.data_ptr(), K, 0, Bs.data_ptr(), Bs.stride(0), int(b_mn), M, N, K, C.data_ptr(), C.stride(0),
                                   int(C.dtype == torch.float32), acc, bias.data_ptr() if bias is not None else None,
                                   res.data_ptr() if res is not None else None, res.stride(0) if res is not None else 0, alpha,
                                   _lib.stream_ptr()))
        return C
    wide = torch.full((M, N + pad), 7.0, device=cuda_device)
    got = run(wide[:, :N])
    assert ((got.double() - want).abs() <= slack).all()
    assert (wide[:, N:] == 7.0).all(), "columns beyond the output were written"
    wide[:, :N] = old
    got = run(wide[:, :N], acc=1, alpha=0.5)
    total = old.double() + 0.5 * want
    assert ((got.double() - total).abs() <= slack + 2.0 ** -23 * (old.abs().double() + total.abs())).all()
    assert (wide[:, N:] == 7.0).all()
    half = torch.full((M, N + pad), 7.0, dtype=torch.bfloat16, device=cuda_device)
    got = run(half[:, :N], bias=bias, res=res)
    total = want + bias.double() + res.double()
    assert ((got.double() - total).abs() <= 2 * slack + 2.0 ** -8 * total.abs() + 1e-6).all()
    assert (half[:, N:] == 7.0).all()


def test_gate_quotient_over_its_range(cuda_device):
    """SiLU in the GEMM's epilogue against the device's own division: gates from far below to far above zero, the overflow of
    exp among them.  One feature per gate value, up = 1; both sides round to bf16, a tie may fall either way (one bf16 ulp)."""
    from pipelinerl_b200.learner_body import Ops
    n, K = 512, 512
    gate = torch.cat([torch.linspace(-130, 130, n - 8), torch.tensor([-1e30, -88.7, -87.4, -1e-30, 0.0, 1e-30, 88.7, 1e30])])
    gate = gate.to(torch.bfloat16).to(cuda_device)
    W = torch.zeros(2 * n, K, dtype=torch.bfloat16, device=cuda_device)
    W[torch.arange(n), torch.arange(n)] = gate
    W[n:, :] = torch.eye(n, dtype=torch.bfloat16, device=cuda_device)
    X = torch.eye(K, dtype=torch.bfloat16, device=cuda_device)       # row i: gate i and up = 1 at feature i
    _, act = Ops().gemm_swiglu(X, W, need_gate_up=False)
    got, g = act.diagonal().float(), gate.float()
    want = (g / (1 + torch.exp(-g))).to(torch.bfloat16).float()
    assert torch.isfinite(got).all()
    assert ((got - want).abs() <= 2.0 ** -7 * want.abs() + 1e-36).all(), (got - want).abs().max()


def _quotient(a, b):
    from pipelinerl_b200 import _lib
    lib, q = _lib.load(), torch.empty_like(a)
    _lib.check(lib.prl_debug_quotient(a.data_ptr(), b.data_ptr(), a.numel(), q.data_ptr(), _lib.stream_ptr()))
    return q


@pytest.mark.parametrize("name", ["plain", "scaled", "silu", "sigmoid", "small", "subnormal", "midpoints"])
def test_quotient_of_the_gates_in_fp32(cuda_device, name):
    """a / b, b >= 1, against the device's own division.  From 2^-100 on: another value than the rounded one only within 2^-21 ulp of
    a midpoint, which one quotient in 2^20 is, and then its neighbour.  Below: one unit in the last place.  "midpoints" are the
    quotients nearest to one: mantissas A, B (B odd) with A 2^24 or A 2^25 = M B + 1, M a 25-bit midpoint, found by inverting B."""
    n, g = 1 << 22, torch.Generator(device=cuda_device).manual_seed(len(name))

    def draw(lo, hi):
        return (1 + torch.rand(n, generator=g, device=cuda_device)) * torch.exp2(torch.randint(lo, hi + 1, (n,), generator=g, device=cuda_device).float())
    gate = torch.linspace(-75, 100, n, device=cuda_device)
    if name == "plain":
        a, b = draw(-30, 100) * torch.where(torch.rand(n, generator=g, device=cuda_device) < 0.5, -1.0, 1.0), draw(0, 60)
    elif name == "scaled":
        a, b = draw(30, 100), draw(60, 126)
    elif name == "silu":
        a, b = gate, 1 + torch.exp(-gate)
    elif name == "sigmoid":
        a, b = torch.ones_like(gate), 1 + torch.exp(-gate.clamp(min=-69))
    elif name == "small":
        a, b = draw(-126, -100), draw(0, 30)
    elif name == "subnormal":
        a, b = draw(-149, -126), draw(0, 20)
    else:
        B = torch.arange((1 << 23) + 1, 1 << 24, 2, device=cuda_device)
        parts = []
        for bits in (24, 25):
            m, inv = (1 << bits) - 1, B.clone()
            for _ in range(5):
                inv = (inv * ((2 - (B * inv & m)) & m)) & m
            M = (-inv & m) + ((1 << 24) if bits == 24 else 0)
            A = (M * B + 1) >> bits
            ok = (M >= 1 << 24) & (M < 1 << 25) & (A >= 1 << 23) & (A < 1 << 24)
            assert ((M * B + 1)[ok] & m == 0).all() and ok.sum() > 1000000
            parts.append((A[ok].float() * 2.0 ** -23, B[ok].float() * 2.0 ** -23))
        a, b = torch.cat([x[0] for x in parts]), torch.cat([x[1] for x in parts])
    got, want = _quotient(a, b), a / b
    off = (got.view(torch.int32).long() - want.view(torch.int32).long()).abs()
    assert off.max().item() <= 1
    if name in ("plain", "scaled", "silu", "sigmoid"):
        assert (want.abs() >= 2.0 ** -100).sum() >= 0.99 * n and (off != 0).sum().item() <= 8 + n / 2 ** 20


def test_quotient_of_the_gates_at_zero_and_infinity(cuda_device):
    inf, nan = float("inf"), float("nan")
    a = torch.tensor([0.0, -0.0, 1.0, -1.0, inf, -inf, nan, 3.4e38, -3.4e38, 88.0, -104.0], device=cuda_device)
    b = torch.tensor([1.0, 2.0, 3.0, inf, 3.4e38, 1.8446744e19, 2.0e19, nan, 1.0000001], device=cuda_device)
    a, b = (t.contiguous() for t in torch.cartesian_prod(a, b).T)
    got, want = _quotient(a, b), a / b
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    ok = ~torch.isnan(want)
    assert torch.equal(got[ok], want[ok]) and torch.equal(torch.signbit(got[ok]), torch.signbit(want[ok]))


@pytest.mark.parametrize("M,N,pad", [(256, 256, 0), (300, 516, 0), (129, 66, 1)])
def test_fp32_accumulation_keeps_subnormal_numbers(cuda_device, M, N, pad):
    """A sum below 2^-126, a product below it and an old value below it: all exact in fp32, none is a zero."""
    from pipelinerl_b200 import _lib
    lib, K = _lib.load(), 64
    A = torch.full((M, K), 2.0 ** -70, dtype=torch.bfloat16, device=cuda_device)
    for b, old in ((2.0 ** -70, 2.0 ** -133), (2.0 ** -63, -2.0 ** -126), (2.0 ** -70, -2.0 ** -134), (2.0 ** -62, 2.0 ** -140)):
        B = torch.full((N, K), b, dtype=torch.bfloat16, device=cuda_device)
        wide = torch.full((M, N + pad), old, device=cuda_device)
        _lib.check(lib.prl_gemm_ex(A.data_ptr(), K, 0, B.data_ptr(), K, 0, M, N, K, wide.data_ptr(), N + pad, 1, 1, None, None, 0, 1.0,
                                   _lib.stream_ptr()))
        want = torch.tensor(K * 2.0 ** -70 * b + old, dtype=torch.float64).float().item()
        assert want != 0.0 or old == -2.0 ** -134
        assert (wide[:, :N] == want).all() and (wide[:, N:] == old).all(), (b, old)


@pytest.mark.parametrize("pad", [0, 1])
def test_fp32_accumulation_rounds_as_the_cpu_does(cuda_device, pad):
    """Products around 2^-100, where adding in L2 begins, and at zero, infinity and NaN; old values from zero to far above them, their
    negatives and neighbours (cancellation) among them.  One term per sum, so the product is exact and the sum has one rounding."""
    from pipelinerl_b200 import _lib
    lib, g, N, K = _lib.load(), torch.Generator().manual_seed(pad), 320, 64
    e = torch.tensor([0, -60, -99, -100, -101, -102, -110, -125, -126, -130, -140, -149, 3, 40])
    M = 2 * len(e)
    A, B = torch.zeros(M, K), torch.zeros(N, K)
    A[:, 0] = torch.cat([torch.exp2((e // 2).float()), -torch.exp2((e // 2).float())])
    A[-1, 0] = 0.0
    scale = torch.exp2((e - e // 2).float()).repeat(2)                    # the rest of the exponent, row by row, in a second operand
    B[:, 0] = 1 + torch.randint(0, 128, (N,), generator=g).float() / 128
    B[0, 0], B[1, 0], B[2, 0] = 0.0, torch.inf, torch.nan
    prod = A[:, :1] * B[:, 0]
    olds = []
    for row in range(M):
        m = prod[row] * scale[row]
        old = torch.randn(N, generator=g) * torch.exp2(torch.randint(-149, 20, (N,), generator=g).float())
        old[64:128] = -m[64:128]
        old[128:192] = torch.nextafter(-m[128:192], torch.tensor(0.0))
        old[192:256] = torch.exp2(torch.randint(-149, -120, (64,), generator=g).float())
        old[256:264] = 0.0
        olds.append(old)
    old = torch.stack(olds)
    for row in range(0, M):                                               # a launch per row: its own scale in alpha
        wide = torch.full((M, N + pad), 7.0)
        wide[:, :N] = old
        wide = wide.to(cuda_device)
        a, b = A.to(torch.bfloat16).to(cuda_device), B.to(torch.bfloat16).to(cuda_device)
        _lib.check(lib.prl_gemm_ex(a.data_ptr(), K, 0, b.data_ptr(), K, 0, M, N, K, wide.data_ptr(), N + pad, 1, 1, None, None, 0,
                                   float(scale[row]), _lib.stream_ptr()))
        want = prod[row].double().float() * scale[row] + old[row]         # exact product and scale (a power of two), one rounded sum
        got = wide[row, :N].cpu()
        nan = torch.isnan(want)
        assert torch.equal(torch.isnan(got), nan) and torch.equal(got[~nan], want[~nan]), row
        assert (wide[:, N:] == 7.0).all()


def test_fp32_accumulation_over_many_tiles_of_a_pair(cuda_device):
    """More tiles than CTA pairs, ragged on both sides."""
    from pipelinerl_b200 import _lib
    lib, g = _lib.load(), torch.Generator().manual_seed(3)
    M, N, K = 4000, 9220, 72
    At = torch.randn(K, M, generator=g).to(torch.bfloat16).to(cuda_device)
    Bt = torch.randn(K, 9224, generator=g).to(torch.bfloat16).to(cuda_device)
    old = torch.randn(M, N, generator=g).to(cuda_device)
    C = old.clone()
    for _ in range(2):
        _lib.check(lib.prl_gemm_ex(At.data_ptr(), M, 1, Bt.data_ptr(), 9224, 1, M, N, K, C.data_ptr(), N, 1, 1, None, None, 0, 1.0,
                                   _lib.stream_ptr()))
    plain = torch.empty(M, N, device=cuda_device)
    _lib.check(lib.prl_gemm_ex(At.data_ptr(), M, 1, Bt.data_ptr(), 9224, 1, M, N, K, plain.data_ptr(), N, 1, 0, None, None, 0, 1.0,
                               _lib.stream_ptr()))
    assert torch.equal(C, old + plain + plain)


def _at(t, offset):
    """A copy of `t` whose storage starts `offset` elements into a buffer (for bf16 one element is two bytes off 16)."""
    buf = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)
    out = buf[offset:offset + t.numel()].view(t.shape)
    out.copy_(t)
    return out


@pytest.mark.parametrize("M,K,I,offset", [(130, 72, 128, 1), (300, 264, 384, 4)])
def test_silu_epilogue_into_unaligned_rows(cuda_device, M, K, I, offset):
    """act and gate_up that start off 16 bytes leave the staged chunk element by element: the same bits, nothing beside them."""
    from pipelinerl_b200 import _lib
    from pipelinerl_b200.learner_body import Ops
    lib, g = _lib.load(), torch.Generator().manual_seed(M)
    X = torch.randn(M, K, generator=g).to(torch.bfloat16).to(cuda_device)
    W = (0.2 * torch.randn(2 * I, K, generator=g)).to(torch.bfloat16).to(cuda_device)
    want_gu, want = Ops().gemm_swiglu(X, W)
    act = torch.full((M * I + 8,), 7.0, dtype=torch.bfloat16, device=cuda_device)
    gu = torch.full((M * 2 * I + 8,), 7.0, dtype=torch.bfloat16, device=cuda_device)
    _lib.check(lib.prl_gemm_swiglu(X.data_ptr(), K, W.data_ptr(), K, M, I, K, act[offset:].data_ptr(), I, gu[offset:].data_ptr(), 2 * I,
                                   _lib.stream_ptr()))
    assert torch.equal(act[offset:offset + M * I].view(M, I), want) and torch.equal(gu[offset:offset + 2 * M * I].view(M, 2 * I), want_gu)
    for t, n in ((act, M * I), (gu, 2 * M * I)):
        assert (t[:offset] == 7.0).all() and (t[offset + n:] == 7.0).all()


@pytest.mark.parametrize("M,N,K,ldc,offset", [(300, 200, 72, 200, 0), (257, 1000, 136, 1000, 1), (130, 66, 64, 67, 0), (2049, 3584, 64, 3584, 4)])
def test_residual_in_the_output_buffer(cuda_device, M, N, K, ldc, offset):
    """C = A B^T + C in bf16, aligned and not: every element is read before it is written, by the thread that writes it."""
    from pipelinerl_b200 import _lib
    lib, g = _lib.load(), torch.Generator().manual_seed(M + N)
    A = torch.randn(M, K, generator=g).to(torch.bfloat16).to(cuda_device)
    B = torch.randn(N, K, generator=g).to(torch.bfloat16).to(cuda_device)
    C = _at(torch.randn(M, ldc, generator=g).to(torch.bfloat16).to(cuda_device), offset)
    res, want = C.clone(), torch.empty(M, ldc, dtype=torch.bfloat16, device=cuda_device)
    for out, r in ((want, res), (C, C)):
        _lib.check(lib.prl_gemm_ex(A.data_ptr(), K, 0, B.data_ptr(), K, 0, M, N, K, out.data_ptr(), ldc, 0, 0, None, r.data_ptr(), ldc, 1.0,
                                   _lib.stream_ptr()))
    assert torch.equal(C[:, :N], want[:, :N]) and torch.equal(C[:, N:], res[:, N:])
    exact = A.double() @ B.double().T + res[:, :N].double()
    slack = K * 2.0 ** -24 * (A.double().abs() @ B.double().abs().T)
    assert ((C[:, :N].double() - exact).abs() <= 2 * slack + 2.0 ** -8 * exact.abs() + 1e-6).all()


@pytest.mark.parametrize("K1,K2,N", [(72, 64, 1002), (128, 1000, 301)])
def test_dual_product_into_unaligned_rows(cuda_device, K1, K2, N):
    """Slices of a split whose rows are not a multiple of 16 bytes."""
    from pipelinerl_b200 import _lib
    lib, g, M = _lib.load(), torch.Generator().manual_seed(N), 300
    A1, B1, A2, B2 = ((torch.randn(r, k, generator=g) / k ** 0.5).to(torch.bfloat16).to(cuda_device) for r, k in ((M, K1), (N, K1), (M, K2), (N, K2)))
    want = A1.double() @ B1.double().T + A2.double() @ B2.double().T
    size = A1.double().abs() @ B1.double().abs().T + A2.double().abs() @ B2.double().abs().T
    for k in (1, 2):
        flat = torch.full((k * M * N + 8,), 7.0, device=cuda_device)
        out = flat[1:1 + k * M * N].view(k, M, N)
        _lib.check(lib.prl_gemm_tn_dual(A1.data_ptr(), B1.data_ptr(), K1, A2.data_ptr(), B2.data_ptr(), K2, M, N, k, out.data_ptr(),
                                        _lib.stream_ptr()))
        assert ((out.double().sum(0) - want).abs() <= (K1 + K2 + k) * 2.0 ** -24 * size + 1e-12).all()
        assert flat[0] == 7.0 and (flat[1 + k * M * N:] == 7.0).all()


@pytest.mark.parametrize("N,ldc", [(72, 75), (136, 136), (300, 303)])
def test_grouped_products_into_unaligned_rows(cuda_device, N, ldc):
    """The gated (bf16, weighted) and the plain (fp32) output of the grouped GEMM with rows off 16 bytes: the bits of aligned rows."""
    from pipelinerl_b200 import _lib
    lib, g = _lib.load(), torch.Generator().manual_seed(N)
    n, W, experts, top = 300, 64, 3, 2
    x = torch.randn(n, W, generator=g).to(torch.bfloat16).to(cuda_device)
    w = (torch.randn(experts * N, W, generator=g) / 8).to(torch.bfloat16).to(cuda_device)
    z = torch.randn(n, experts, generator=g).to(cuda_device)
    i32 = dict(dtype=torch.int32, device=cuda_device)
    sel, perm, meta = torch.zeros(top, n, **i32), torch.zeros(top * n, **i32), torch.zeros(4, **i32)
    wsel, tiles = torch.zeros(top, n, device=cuda_device), torch.zeros(3 * int(lib.prl_moe_max_tiles(top * n, experts)), **i32)
    st, table = _lib.stream_ptr(), (perm.data_ptr(), meta.data_ptr(), tiles.data_ptr())
    _lib.check(lib.prl_moe_choose(z.data_ptr(), experts, None, n, experts, experts, top, 1, 1, 1, 0, 0, 1.0, 256, sel.data_ptr(), wsel.data_ptr(),
                                  *table, st))
    xs = torch.zeros(top * n, W, dtype=torch.bfloat16, device=cuda_device)
    _lib.check(lib.prl_moe_gather(x.data_ptr(), *table[:2], n, top * n, W, xs.data_ptr(), st))
    for dtype, weights in ((torch.bfloat16, wsel.data_ptr()), (torch.float32, None)):
        got = []
        for ld, off in ((N + -N % 8, 0), (ldc, 1)):
            flat = torch.full((top * n * ld + 8,), 7.0, dtype=dtype, device=cuda_device)
            out = flat[off:off + top * n * ld].view(top * n, ld)
            _lib.check(lib.prl_moe_gemm_tc(xs.data_ptr(), top * n, w.data_ptr(), experts, N, W, *table, weights, 1 if weights else 0,
                                           out.data_ptr(), ld, st))
            assert (out[:, N:] == 7.0).all() and (flat[:off] == 7.0).all() and (flat[off + top * n * ld:] == 7.0).all()
            got.append(out[:, :N].clone())
        assert torch.equal(got[0], got[1]) and got[0].float().abs().max() < 100 and (got[0] != 7.0).any()


@pytest.mark.parametrize("M,V,K,chunk,with_lo,live", [(257, 520, 64, 2048, True, "some"), (700, 1032, 256, 200, True, "some"),
                                                       (640, 264, 72, 256, False, "all"), (300, 776, 128, 2048, True, "none"),
                                                       (513, 2056, 128, 128, True, "one"), (130, 520, 64, 2048, False, "some")])
def test_head_backward_of_kept_logits_and_live_rows(cuda_device, monkeypatch, M, V, K, chunk, with_lo, live):
    """The learner's head with all, some and none of its logits kept, and gradients on all, some, one and no rows: d hidden of
    the three ways agrees in its bits (one product, one formula; dW differs in the order of its terms), and both gradients with autograd in fp64 up to the bf16
    rounding of d logits (2^-9 of each term) and of d hidden."""
    import types
    from pipelinerl_b200.learner_body import Ops
    from pipelinerl_b200.learner_model import _NativeHead
    dev, T = cuda_device, 0.7
    g = torch.Generator(device=dev).manual_seed(M + V + K)
    x = (torch.randn(M, K, generator=g, device=dev) * 0.7).to(torch.bfloat16)
    Wf = torch.randn(V, K, generator=g, device=dev) * K ** -0.5
    W = Wf.to(torch.bfloat16)
    lo = (Wf - W.float()).to(torch.bfloat16) if with_lo else None
    tg = torch.randint(0, V, (M,), generator=g, device=dev)
    g_lp, g_ent = torch.randn(M, generator=g, device=dev), torch.randn(M, generator=g, device=dev) * 0.3
    on = {"all": torch.ones(M, device=dev), "none": torch.zeros(M, device=dev),
          "some": (torch.rand(M, generator=g, device=dev) < 0.6).float(), "one": (torch.arange(M, device=dev) == M // 2).float()}[live]
    g_lp, g_ent = g_lp * on, g_ent * on

    def run(kept):
        monkeypatch.setattr(_NativeHead, "_rows_to_keep", staticmethod(lambda *a: kept if M > 256 else 0))
        gW = torch.full((V, K), 0.25, device=dev)
        model = types.SimpleNamespace(p=lambda n: W, head_lo=lo, body=types.SimpleNamespace(ops=Ops(), g={"lm_head.weight": gW}))
        h = x.clone().requires_grad_()
        lp, ent = _NativeHead.apply(h, model, tg, T, chunk)
        obj = (lp * g_lp).sum() + (ent * g_ent).sum()
        obj.backward(retain_graph=True)
        first, dW = h.grad.clone(), gW.clone()
        h.grad = None
        obj.backward()                                     # a retained graph: nothing is kept any more
        assert torch.equal(h.grad, first)
        return first, dW, (gW - dW, lp, ent)

    whole, part, none = run(M), run(256 if M > 256 else 0), run(0)
    assert torch.equal(whole[0], none[0]) and torch.equal(part[0], none[0])
    assert torch.equal(whole[2][1], none[2][1]) and torch.equal(whole[2][2], none[2][2])
    z = x.double() @ (W.double() + (lo.double() if with_lo else 0.0)).T / T
    ls = torch.log_softmax(z, -1)
    p, H = ls.exp(), -(ls.exp() * ls).sum(-1, keepdim=True)
    gl, ge = g_lp.double()[:, None], g_ent.double()[:, None]
    dz = (gl * (torch.nn.functional.one_hot(tg, V) - p) - ge * p * (ls + H)) / T
    Ws = W.double()
    size = dz.abs() + (gl.abs() + ge.abs()) * p * 2.0 ** -13 / T          # fp32 exponent of a logit of up to 2^7
    for got in (whole, part, none):
        want = dz @ Ws
        assert ((got[0].double() - want).abs() <= 2.0 ** -8 * (size @ Ws.abs()) + 2.0 ** -8 * want.abs() + 1e-9).all()
        for d in (got[1].double() - 0.25, got[2][0].double()):
            assert ((d - dz.T @ x.double()).abs() <= 2.0 ** -8 * (size.T @ x.double().abs()) + 2.0 ** -21).all()


@pytest.mark.parametrize("M,V,K,chunk", [(700, 1032, 256, 200), (640, 264, 72, 256), (513, 2056, 128, 128), (257, 520, 64, 2048)])
def test_head_gradients_do_not_depend_on_what_is_kept(cuda_device, monkeypatch, M, V, K, chunk):
    """d hidden and dW have the same bits whether the memory held the logits of all rows, of the first chunks, of none, or the buffer was refused: dW is summed chunk
    by chunk in any case."""
    import types
    from pipelinerl_b200.learner_body import Ops
    from pipelinerl_b200.learner_model import _NativeHead
    dev, g = cuda_device, torch.Generator(device=cuda_device).manual_seed(M + V)
    x, W, lo = (torch.randn(n, K, generator=g, device=dev).to(torch.bfloat16) * s for n, s in ((M, 1.0), (V, 0.1), (V, 0.0005)))
    tg, on = torch.randint(0, V, (M,), generator=g, device=dev), (torch.rand(M, generator=g, device=dev) < 0.7).float()
    got = []
    for kept in (0, chunk, 2 * chunk, M, 1 << 36):           # the last is more than any memory: the forward goes on without a buffer
        if kept <= M or kept == 1 << 36:
            monkeypatch.setattr(_NativeHead, "_rows_to_keep", staticmethod(lambda *a: kept))
            gW = torch.full((V, K), 0.25, device=dev)
            model = types.SimpleNamespace(p=lambda n: W, head_lo=lo, body=types.SimpleNamespace(ops=Ops(), g={"lm_head.weight": gW}))
            h = x.clone().requires_grad_()
            lp, ent = _NativeHead.apply(h, model, tg, 0.8, chunk)
            torch.autograd.backward([lp, ent], [on * 0.5, on * 0.1])
            got.append((h.grad, gW, lp.detach(), ent.detach()))
    assert len(got) >= 3 and all(torch.equal(a, b) for other in got[1:] for a, b in zip(got[0], other)) and got[0][1].std() > 0


def test_former_head_backward_keeps_no_logits(cuda_device, monkeypatch):
    """PRL_HEAD_BWD_FUSED=0 recomputes: nothing is stored for it, and what a forward before the switch stored is let go."""
    import types
    from pipelinerl_b200 import learner_model
    from pipelinerl_b200.learner_body import Ops
    dev, M, V, K = cuda_device, 300, 520, 64
    g = torch.Generator(device=dev).manual_seed(3)
    x, W = (torch.randn(n, K, generator=g, device=dev).to(torch.bfloat16) for n in (M, V))
    tg, got = torch.randint(0, V, (M,), generator=g, device=dev), []
    for before, after in (("1", "1"), ("0", "0"), ("1", "0")):
        monkeypatch.setenv("PRL_HEAD_BWD_FUSED", before)
        model = types.SimpleNamespace(p=lambda n: W, head_lo=None, body=types.SimpleNamespace(ops=Ops(), g={"lm_head.weight": torch.zeros(V, K, device=dev)}))
        h = x.clone().requires_grad_()
        lp, ent = learner_model._NativeHead.apply(h, model, tg, 1.0, 320)
        assert len(learner_model._KEPT) == int(before)
        monkeypatch.setenv("PRL_HEAD_BWD_FUSED", after)
        torch.autograd.backward([lp, ent], [torch.ones_like(lp), torch.ones_like(ent)], retain_graph=True)
        assert not len(learner_model._KEPT)
        got.append(h.grad)
    assert torch.equal(got[1], got[2]) and (got[0] - got[1]).abs().max() <= 2.0 ** -6 * got[1].abs().max()


def test_head_backward_with_little_memory(cuda_device, monkeypatch):
    """Logits that wait for a backward count as held until it took them; where a chunk's d logits find no room the chunk is halved."""
    import types
    from pipelinerl_b200 import learner_model
    from pipelinerl_b200.learner_body import Ops
    dev, M, V, K = cuda_device, 1100, 520, 64
    g = torch.Generator(device=dev).manual_seed(3)
    x, W = (torch.randn(n, K, generator=g, device=dev).to(torch.bfloat16) for n in (M, V))
    tg = torch.randint(0, V, (M,), generator=g, device=dev)
    empty, seen, asked = torch.empty, [], []

    def keep(M_, V_, d, chunk, held):
        seen.append(held)
        return M if len(seen) < 3 else 0

    def small(*a, **k):
        if k.get("dtype") == torch.bfloat16 and a[1:] == (V,):
            asked.append(a[0])
            if a[0] > 320:
                raise torch.cuda.OutOfMemoryError("no room")
        return empty(*a, **k)

    monkeypatch.setattr(learner_model._NativeHead, "_rows_to_keep", staticmethod(keep))
    gW = [torch.zeros(V, K, device=dev) for _ in range(3)]
    hs = [x.clone().requires_grad_() for _ in range(3)]
    outs = [learner_model._NativeHead.apply(h, types.SimpleNamespace(p=lambda n: W, head_lo=None, body=types.SimpleNamespace(ops=Ops(), g={"lm_head.weight": w})),
                                            tg, 1.0, 1152) for h, w in zip(hs, gW)]
    one = 4 * 1152 * V
    assert seen == [0, one, 2 * one]
    for lp, ent in outs[:2]:
        torch.autograd.backward([lp, ent], [torch.ones_like(lp), torch.ones_like(ent)])
    assert not list(learner_model._KEPT.values())
    monkeypatch.setattr(torch, "empty", small)
    torch.autograd.backward(outs[2], [torch.ones_like(outs[2][0]), torch.ones_like(outs[2][1])])
    assert asked == [1152, 512, 256] and torch.equal(hs[2].grad, hs[0].grad) and torch.equal(gW[0], gW[1])
    assert (gW[2] - gW[0]).norm() <= M * 2.0 ** -24 * gW[0].norm()          # the same M fp32 terms in more sums


@pytest.mark.parametrize("M,kept", [(300, 0), (300, 300), (200, 0)])
def test_head_backward_of_a_masked_row_that_is_no_number(cuda_device, monkeypatch, M, kept):
    """A token without a gradient whose hidden state is not a number: its d hidden and dW are none either (0 x NaN), the other rows' stay what they are."""
    import types
    from pipelinerl_b200.learner_body import Ops
    from pipelinerl_b200.learner_model import _NativeHead
    dev, V, K = cuda_device, 520, 64
    g = torch.Generator(device=dev).manual_seed(M)
    x, W = (torch.randn(n, K, generator=g, device=dev).to(torch.bfloat16) for n in (M, V))
    tg, on = torch.randint(0, V, (M,), generator=g, device=dev), (torch.arange(M, device=dev) % 3 > 0).float()
    monkeypatch.setattr(_NativeHead, "_rows_to_keep", staticmethod(lambda *a: kept))
    got = []
    for bad in (False, True):
        if bad:
            x[6, 5], x[9, 0] = math.nan, math.inf
        gW = torch.zeros(V, K, device=dev)
        model = types.SimpleNamespace(p=lambda n: W, head_lo=None, body=types.SimpleNamespace(ops=Ops(), g={"lm_head.weight": gW}))
        h = x.clone().requires_grad_()
        lp, ent = _NativeHead.apply(h, model, tg, 1.0, 2048)
        torch.autograd.backward([lp, ent], [on, 0.1 * on])
        got.append((h.grad, gW))
    rows = torch.arange(M, device=dev)
    rest = (rows != 6) & (rows != 9)
    assert torch.equal(got[0][0][rest], got[1][0][rest]) and torch.count_nonzero(got[0][0][[6, 9]]) == 0
    assert got[1][0][[6, 9]].isnan().all() and got[1][1].isnan().all() and not got[0][1].isnan().any()
