"""Workloads of the framework's three users: the learner (norms, attention, a decoder layer, a whole RL step, the loss on
full logits, the optimizer), the sampler engine (token steps of few and of many sequences, prompts) and the hybrid
decoders on the same engine (prompts, token steps).

A case is a dict of plain values.  `prepare` builds what a program holds before the call (inputs from the seed, weights,
engines), `run` makes one pass through the public entry points, `work` counts what a pass cannot do without, `exact`
computes the same outputs in 64 bits with plain torch.
"""
from __future__ import annotations

import math
import random
import types

import torch

DEV = "cuda:0"
F64 = torch.float64
BF16 = torch.bfloat16
PAGE = 64                     # tokens per page of the engine's KV cache


# ---- the cases -------------------------------------------------------------------------------------------------------------
def listed():
    q7 = dict(width=3584, ff=18944, heads=28, kv_heads=4)          # one layer of Qwen2.5-7B
    return [
        # every sublayer of the learner opens with this norm, and its backward closes it: one packed row of 16384 tokens
        dict(name="norm_row", kind="norm", rows=16384, width=3584),
        # attention of a learner over a packed row of samples of odd lengths (short rollouts packed together)
        dict(name="attention_packed", kind="attention", segments="1531,977,64,2300,1,411", heads=14, kv_heads=2),
        # ... and over one long rollout that fills the row
        dict(name="attention_long", kind="attention", segments="16384", heads=28, kv_heads=4),
        # one decoder layer of the learner, forward and backward (the unit that a 28-layer step repeats)
        dict(name="layer", kind="layer", segments="2049,1500,547", vocab=32768, **q7),
        # one RL micro-batch end to end: forward, fp32-equivalent head, PPO loss, backward into the gradient arena
        dict(name="train_step", kind="train", segments="1024,1001,1047", layers=2, vocab=152064, **q7),
        # the RL step of any model that hands over full fp32 logits: log-probs, entropy, loss, and d logits
        dict(name="loss_logits", kind="loss", segments="700,400,901", vocab=151936, policy="ppo", temperature=1.0),
        # an optimizer step over the parameters of a few layers
        dict(name="adamw", kind="adamw", params=466_120_000, tensors=14, grad="float32", clip=0.3),
        # token step of a small model with a few sequences left: launches and latency
        dict(name="decode_small", kind="decode", batch=4, context=333, layers=8, width=1024, ff=4096, heads=8, kv_heads=2,
             vocab=32768, fp32_head=False),
        # token step of a full batch with long contexts, fp32-equivalent head (the benchmark's shape, fewer layers)
        dict(name="decode_full", kind="decode", batch=64, context=8192, layers=4, vocab=152064, fp32_head=True, **q7),
        # a prompt of odd length through the engine in chunks
        dict(name="prompt", kind="prompt", tokens=2999, layers=4, vocab=32768, **q7),
        # hybrid decoder: windowed attention beside the gated delta rule, routed experts; a prompt
        dict(name="hybrid_prompt", kind="hybrid_prompt", tokens=2500, layers=2, width=2048, ff=8192, vocab=32768),
        # ... and token steps of a batch that has its prompts behind it
        dict(name="hybrid_decode", kind="hybrid_decode", batch=32, context=1100, layers=4, width=2048, ff=8192, vocab=32768),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _split(rng, total, most):
    """`total` tokens cut into up to `most` samples of uneven lengths."""
    n = rng.randint(1, max(1, min(most, total // 8)))
    cuts = sorted(rng.sample(range(1, total), n - 1)) if n > 1 else []
    return ",".join(str(b - a) for a, b in zip([0] + cuts, cuts + [total]))


def draw(rng: random.Random):
    kind = rng.choice(["norm", "norm", "attention", "attention", "layer", "train", "loss", "adamw", "decode", "decode", "prompt",
                       "hybrid_prompt", "hybrid_decode"])
    width, ff, heads, kv = rng.choice([(1024, 4096, 8, 2), (2048, 8192, 16, 4), (3584, 18944, 28, 4)])
    size = dict(width=width, ff=ff, heads=heads, kv_heads=kv)
    if kind == "norm":
        return dict(kind=kind, rows=_log(rng, 1, 16384), width=rng.choice([896, 1024, 2048, 3584, 8 * rng.randint(16, 512)]))
    if kind == "attention":
        heads, kv = rng.choice([(28, 4), (14, 2), (8, 2), (16, 4), (4, 4), (5, 1), (16, 1)])
        return dict(kind=kind, segments=_split(rng, _log(rng, 40, 9000), 12), heads=heads, kv_heads=kv)
    if kind == "layer":
        return dict(kind=kind, segments=_split(rng, _log(rng, 100, 4096), 6), vocab=32768, **size)
    if kind == "train":
        return dict(kind=kind, segments=_split(rng, _log(rng, 200, 3000), 5), layers=rng.randint(1, 2), vocab=32768, **size)
    if kind == "loss":
        return dict(kind=kind, segments=_split(rng, _log(rng, 30, 2000), 6), vocab=rng.choice([151936, 32768, 4 * rng.randint(300, 37000)]),
                    policy=rng.choice(["ppo", "reinforce", "gspo"]), temperature=rng.choice([1.0, 0.7]))
    if kind == "adamw":
        return dict(kind=kind, params=_log(rng, 100_000, 400_000_000), tensors=rng.randint(1, 40), grad=rng.choice(["float32", "bfloat16"]),
                    clip=rng.choice([0.0, 0.3]))
    if kind == "decode":
        return dict(kind=kind, batch=_log(rng, 1, 64), context=_log(rng, 20, 8000), layers=rng.randint(1, 4), vocab=32768,
                    fp32_head=rng.random() < 0.5, **size)
    if kind == "prompt":
        return dict(kind=kind, tokens=_log(rng, 150, 3000), layers=rng.randint(1, 4), vocab=32768, **size)
    width, ff = rng.choice([(1024, 4096), (2048, 8192)])
    if kind == "hybrid_prompt":
        return dict(kind=kind, tokens=_log(rng, 150, 2500), layers=rng.randint(1, 2), width=width, ff=ff, vocab=32768)
    return dict(kind=kind, batch=_log(rng, 1, 32), context=_log(rng, 30, 1100), layers=rng.randint(1, 4), width=width, ff=ff, vocab=32768)


# ---- inputs ------------------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _normal(g, shape, std=1.0, dtype=BF16, mean=0.0):
    """Normal values, made in slices so that a large tensor needs no fp32 copy of itself."""
    out = torch.empty(shape, dtype=dtype, device=DEV)
    flat, step = out.view(-1), 1 << 27
    for s in range(0, flat.numel(), step):
        n = min(step, flat.numel() - s)
        flat[s:s + n] = torch.randn(n, generator=g, device=DEV).mul_(std).add_(mean).to(dtype)
    return out


def _segments(case):
    return [int(s) for s in case["segments"].split(",")]


def _positions(lengths):
    return torch.cat([torch.arange(n) for n in lengths]).to(DEV)


def _qwen_shapes(case, layers):
    """Tensor names and shapes of the Qwen2 family's fused layout."""
    H, I, nq, nk = case["width"], case["ff"], case["heads"] * 128, case["kv_heads"] * 128
    out = []
    for l in range(layers):
        p = f"layers.{l}."
        out += [(p + "input_layernorm.weight", (H,)), (p + "qkv_proj.weight", (nq + 2 * nk, H)), (p + "qkv_proj.bias", (nq + 2 * nk,)),
                (p + "o_proj.weight", (H, nq)), (p + "post_attention_layernorm.weight", (H,)), (p + "gate_up_proj.weight", (2 * I, H)),
                (p + "down_proj.weight", (H, I))]
    return out + [("embed_tokens.weight", (case["vocab"], H)), ("norm.weight", (H,)), ("lm_head.weight", (case["vocab"], H))]


def _qwen_weights(case, seed, layers, head_lo=False):
    g, w = _gen(seed), {}
    for name, shape in _qwen_shapes(case, layers):
        if name.endswith("norm.weight"):
            w[name] = _normal(g, shape, 0.1, mean=1.0)
        elif name.endswith(".bias"):
            w[name] = _normal(g, shape, 0.2)
        elif name == "embed_tokens.weight":
            w[name] = _normal(g, shape, 1.0)                        # trained embeddings give the residual stream its scale
        else:
            w[name] = _normal(g, shape, 0.02)
    if head_lo:                                                     # the bf16 residual of an fp32 head
        w["lm_head.weight_lo"] = _normal(g, w["lm_head.weight"].shape, 0.02 / 512)
    return w


def _qwen_config(case, layers, **kw):
    from pipelinerl_b200.model import ModelConfig
    return ModelConfig(vocab_size=case["vocab"], hidden_size=case["width"], intermediate_size=case["ff"], num_layers=layers,
                       num_q_heads=case["heads"], num_kv_heads=case["kv_heads"], **kw)


def _tokens(case, seed, n):
    return torch.randint(8, case["vocab"] - 8, (n,), generator=torch.Generator().manual_seed(seed + 7919))


# ---- learner: norm -----------------------------------------------------------------------------------------------------------
def _norm_inputs(case, seed):
    g = _gen(seed)
    T, H = case["rows"], case["width"]
    return dict(x=_normal(g, (T, H), 1.5), gamma=_normal(g, (H,), 0.1, mean=1.0), dy=_normal(g, (T, H), 0.02), dres=_normal(g, (T, H), 0.02))


def _prepare_norm(case, seed):
    from pipelinerl_b200.learner_body import Ops
    return dict(_norm_inputs(case, seed), ops=Ops(), dgamma=torch.zeros(case["width"], device=DEV))


def _run_norm(s):
    s["dgamma"].zero_()
    y, rstd = s["ops"].rmsnorm(s["x"], s["gamma"], 1e-6)
    dx = s["ops"].rmsnorm_bwd(s["x"], s["gamma"], rstd, s["dy"], s["dres"], s["dgamma"])
    return [y, rstd, dx, s["dgamma"]]


def _exact_norm(case, seed):
    i = {k: v.double() for k, v in _norm_inputs(case, seed).items()}
    x, g, dy = i["x"], i["gamma"], i["dy"]
    rstd = torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6)
    xh, dn = x * rstd, dy * g
    return [xh * g, rstd[:, 0], i["dres"] + rstd * (dn - xh * (dn * xh).mean(-1, keepdim=True)), (dy * xh).sum(0)]


# ---- learner: attention ------------------------------------------------------------------------------------------------------
def _attention_inputs(case, seed):
    g = _gen(seed)
    T, nq, nk = sum(_segments(case)), case["heads"], case["kv_heads"]
    return dict(qkv=_normal(g, (T, (nq + 2 * nk) * 128)), d_out=_normal(g, (T, nq * 128), 0.05))


def _prepare_attention(case, seed):
    from pipelinerl_b200.learner_body import Ops
    n = _segments(case)
    start = [sum(n[:i]) for i in range(len(n))]
    i32 = dict(dtype=torch.int32, device=DEV)
    return dict(_attention_inputs(case, seed), ops=Ops(), start=torch.tensor(start, **i32), length=torch.tensor(n, **i32),
                most=max(n), nq=case["heads"], nk=case["kv_heads"])


def _run_attention(s):
    shape = (s["start"], s["length"], s["most"], s["nq"], s["nk"], 128)
    out, lse = s["ops"].attn_fwd(s["qkv"], *shape)
    return [out, s["ops"].attn_bwd(s["qkv"], out, s["d_out"], lse, *shape)]


def _exact_attention(case, seed):
    i, nq, nk = _attention_inputs(case, seed), case["heads"], case["kv_heads"]
    qkv, d_out = i["qkv"], i["d_out"]
    out = torch.zeros(d_out.shape, dtype=F64, device=DEV)
    grad = torch.zeros(qkv.shape, dtype=F64, device=DEV)
    at = 0
    for n in _segments(case):
        rows = slice(at, at + n)
        at += n
        for h in range(nq):
            col = lambda j: slice(j * 128, (j + 1) * 128)  # noqa: E731
            kh = nq + h // (nq // nk)
            q, k, v = (qkv[rows, col(c)].double() for c in (h, kh, kh + nk))
            p = (q @ k.T).mul_(128 ** -0.5)
            p = torch.softmax(p.masked_fill_(torch.ones(n, n, dtype=torch.bool, device=DEV).triu_(1), -math.inf), -1)
            d = d_out[rows, col(h)].double()
            o = p @ v
            ds = (d @ v.T).sub_((d * o).sum(-1, keepdim=True)).mul_(p).mul_(128 ** -0.5)
            out[rows, col(h)] = o
            grad[rows, col(h)] = ds @ k
            grad[rows, col(kh)] += ds.T @ q
            grad[rows, col(kh + nk)] += p.T @ d
    return [out, grad]


# ---- the Qwen2 family in 64 bits -----------------------------------------------------------------------------------------------
def _ref_norm(x, g):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6) * g


def _ref_rope(x, pos):
    """x [T, heads, 128]"""
    inv = 1.0 / (1_000_000.0 ** (torch.arange(0, 128, 2, device=DEV, dtype=F64) / 128))
    a = pos.double()[:, None] * inv
    c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]
    u, v = x[..., :64], x[..., 64:]
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _ref_layer(case, w, l, h, lengths):
    p, T, nq, nk, I = f"layers.{l}.", h.shape[0], case["heads"], case["kv_heads"], case["ff"]
    qkv = (_ref_norm(h, w[p + "input_layernorm.weight"]) @ w[p + "qkv_proj.weight"].T + w[p + "qkv_proj.bias"]).view(T, nq + 2 * nk, 128)
    pos = _positions(lengths)
    q, k, v = _ref_rope(qkv[:, :nq], pos), _ref_rope(qkv[:, nq:nq + nk], pos), qkv[:, nq + nk:]
    parts, at = [], 0
    for n in lengths:
        qs, ks, vs = (t[at:at + n].transpose(0, 1).reshape(nk, -1, n, 128) for t in (q, k, v))
        at += n
        sc = (qs @ ks.transpose(-1, -2)) * 128 ** -0.5
        sc = sc.masked_fill(torch.ones(n, n, dtype=torch.bool, device=DEV).triu_(1), -math.inf)
        parts.append((torch.softmax(sc, -1) @ vs).reshape(nq, n, 128).transpose(0, 1).reshape(n, nq * 128))
    h = h + torch.cat(parts) @ w[p + "o_proj.weight"].T
    gu = _ref_norm(h, w[p + "post_attention_layernorm.weight"]) @ w[p + "gate_up_proj.weight"].T
    return h + (torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]) @ w[p + "down_proj.weight"].T


# ---- learner: one layer --------------------------------------------------------------------------------------------------------
def _prepare_layer(case, seed):
    from pipelinerl_b200.learner_body import NativeBody
    w = _qwen_weights(case, seed, 1)
    w.pop("lm_head.weight")
    n = _segments(case)
    body = NativeBody(_qwen_config(case, 1), w, {k: torch.zeros(v.shape, device=DEV) for k, v in w.items()})
    body.keep_gate_up_layers = 1
    return dict(body=body, ids=_tokens(case, seed, sum(n)).to(DEV), pos=_positions(n), d=_normal(_gen(seed + 1), (sum(n), case["width"]), 0.02))


def _run_layer(s):
    grads = s["body"].g
    for g in grads.values():
        g.zero_()
    y = s["body"].forward(s["ids"], s["pos"])
    s["body"].backward(s["d"])
    return [y, dict(grads)]


def _exact_layer(case, seed):
    w = {k: v.double().requires_grad_() for k, v in _qwen_weights(case, seed, 1).items() if k != "lm_head.weight"}
    n = _segments(case)
    d = _normal(_gen(seed + 1), (sum(n), case["width"]), 0.02).double()
    h = w["embed_tokens.weight"][_tokens(case, seed, sum(n)).to(DEV)]
    y = _ref_norm(_ref_layer(case, w, 0, h, n), w["norm.weight"])
    y.backward(d)
    return [y.detach(), {k: v.grad for k, v in w.items()}]


# ---- learner: RL batches -------------------------------------------------------------------------------------------------------
def _rl_columns(case, seed, level):
    """Columns of a packed row: the first third of every sample is its prompt; the sampler's log-probs lie around
    `level` (a number, or one value per token), a little off what the learner computes."""
    n = _segments(case)
    T, g = sum(n), torch.Generator().manual_seed(seed + 17)
    sample = torch.arange(len(n)).repeat_interleave(torch.tensor(n))
    ids = _tokens(case, seed, T)
    labels, at = ids.clone(), 0
    for k in n:
        labels[at:at + max(1, k // 3)] = -100
        at += k
    count = torch.zeros(len(n)).index_add_(0, sample, (labels >= 0).float()).clamp_min(1.0)
    adv = (torch.rand(len(n), generator=g) + 0.25) * (torch.randint(0, 2, (len(n),), generator=g).float() * 2 - 0.8)
    old = level + 0.03 * torch.randn(T, generator=g)
    return dict(ids=ids, labels=labels, sample=sample, lengths=n, num_labels=count[sample], advantages=adv[sample],
                rewards=(adv[sample] > 0).float(), old=old, ref=old + 0.1 * torch.randn(T, generator=g))


def _rl_batch(c):
    from pipelinerl_b200.finetune.types import PipelineBatchEncoding
    T, row = len(c["ids"]), lambda t: t[None]  # noqa: E731
    edges = [0]
    for k in c["lengths"]:
        edges.append(edges[-1] + k)
    return PipelineBatchEncoding(
        input_ids=row(c["ids"]), attention_mask=torch.ones(1, T, dtype=torch.long), labels=row(c["labels"]),
        position_ids=row(_positions(c["lengths"]).cpu()), segment_ids=row(c["sample"]), rewards=row(c["rewards"]),
        advantages=row(c["advantages"]), ref_logprobs=row(c["ref"]), old_logprobs=row(c["old"]),
        group_tokens=torch.full((1, T), float(T) / len(c["lengths"])), num_labels=row(c["num_labels"]), overflow=torch.zeros(1, T),
        seq_boundaries=torch.tensor(edges, dtype=torch.int32), model_version=0, is_packed=True).to_device(DEV)


def _rl_config(case):
    from pipelinerl_b200.finetune.rl import RLConfig
    return RLConfig(policy_loss=case.get("policy", "ppo"), temperature=case.get("temperature", 1.0), batch_size=len(_segments(case)))


def _ref_loss(case, c, logits):
    """PPO or REINFORCE loss with the KL term of the default configuration, from logits [T, V]."""
    temperature = case.get("temperature", 1.0)
    lp = torch.log_softmax(logits[:-1] / temperature, -1).gather(1, c["ids"][1:, None].to(DEV))[:, 0]
    col = lambda k: c[k][1:].float().to(DEV).double()  # noqa: E731
    ratio = torch.exp(lp - col("old"))
    d = (col("ref") - lp).clamp(-10.0, 10.0)
    kl = torch.exp(d) - d - 1.0
    if case.get("policy", "ppo") == "ppo":
        gain = torch.minimum(ratio * col("advantages"), ratio.clamp(0.8, 1.2) * col("advantages"))
    else:
        gain = lp * col("advantages") * ratio.clamp(0.0, 1.2).detach()
    mask = (c["labels"][1:] >= 0).to(DEV)
    return -((gain - 0.1 * kl) * mask).sum() / len(c["lengths"])


# ---- learner: whole micro-batch ------------------------------------------------------------------------------------------------
def _prepare_train(case, seed):
    from pipelinerl_b200.finetune.optim import FusedAdamW
    from pipelinerl_b200.learner_model import NativeQwen2
    model = NativeQwen2(_qwen_config(case, case["layers"], fp32_head=True), torch.device(DEV), init=_train_weights(case, seed))
    opt = FusedAdamW(model.named_parameters(), lr=1e-6, weight_decay=0.01, max_grad_norm=0.3, grad_dtype=torch.float32,
                     **model.optimizer_kwargs())
    model.bind(opt)
    model.body.keep_gate_up_layers = case["layers"]
    return dict(model=model, opt=opt, batch=_rl_batch(_rl_columns(case, seed, _level(case))), config=_rl_config(case))


def _level(case):
    return -math.log(case["vocab"])


def _train_weights(case, seed):
    """A narrow head: the policy is close to uniform, so its log-probs are known without running it."""
    w = _qwen_weights(case, seed, case["layers"])
    w["lm_head.weight"] = _normal(_gen(seed + 3), w["lm_head.weight"].shape, 0.06 * case["width"] ** -0.5)
    return w


def _run_train(s):
    from pipelinerl_b200.finetune.rl import rl_step
    s["opt"].zero_grad()
    loss, _ = rl_step(s["model"], s["batch"], 0, 1000, s["config"])
    loss.backward()
    return [loss.detach(), s["opt"].grad_views()]


def _exact_train(case, seed):
    w = {k: v.double().requires_grad_() for k, v in _train_weights(case, seed).items()}
    c = _rl_columns(case, seed, _level(case))
    h = w["embed_tokens.weight"][c["ids"].to(DEV)]
    for l in range(case["layers"]):
        h = _ref_layer(case, w, l, h, c["lengths"])
    loss = _ref_loss(case, c, _ref_norm(h, w["norm.weight"]) @ w["lm_head.weight"].T)
    loss.backward()
    return [loss.detach(), {k: v.grad for k, v in w.items()}]


# ---- learner: loss on full logits ----------------------------------------------------------------------------------------------
class _LogitsModel(torch.nn.Module):
    """Any model of the contract `model(...).logits`, without the model."""

    def __init__(self, logits):
        super().__init__()
        self.logits = torch.nn.Parameter(logits)

    def forward(self, **_):
        return types.SimpleNamespace(logits=self.logits)


def _loss_logits(case, seed):
    return _normal(_gen(seed), (1, sum(_segments(case)), case["vocab"]), 2.0, torch.float32)


def _loss_columns(case, seed, logits):
    """The sampler's log-probs are near the learner's, as they are a few updates apart."""
    x, t = logits[0], case["temperature"]
    ids = _tokens(case, seed, x.shape[0]).to(DEV)
    lp = torch.cat([(r[:-1] / t).gather(1, i[1:, None])[:, 0] - torch.logsumexp(r[:-1] / t, -1)
                    for r, i in ((x[a:a + 257], ids[a:a + 257]) for a in range(0, x.shape[0] - 1, 256))])
    return _rl_columns(case, seed, torch.cat([lp.new_zeros(1), lp]).cpu())


def _prepare_loss(case, seed):
    logits = _loss_logits(case, seed)
    return dict(model=_LogitsModel(logits), batch=_rl_batch(_loss_columns(case, seed, logits)), config=_rl_config(case))


def _run_loss(s):
    from pipelinerl_b200.finetune.rl import rl_step
    s["model"].logits.grad = None
    loss, stats = rl_step(s["model"], s["batch"], 0, 1000, s["config"])
    loss.backward()
    return [loss.detach(), s["model"].logits.grad, torch.tensor(list(stats.values()), dtype=F64)]


def _exact_loss(case, seed):
    if case["policy"] == "gspo":
        return None
    logits = _loss_logits(case, seed)
    x = logits[0].double().requires_grad_()
    loss = _ref_loss(case, _loss_columns(case, seed, logits), x)
    loss.backward()
    return [loss.detach(), x.grad[None], None]


# ---- learner: optimizer --------------------------------------------------------------------------------------------------------
def _adamw_sizes(case):
    """Sizes of the tensors: uneven shares of the parameters, one of them a bias."""
    r = random.Random(case["tensors"])
    share = [r.random() + 0.01 for _ in range(case["tensors"])]
    return [max(3, int(case["params"] * x / sum(share))) for x in share]


def _adamw_inputs(case, seed):
    g, f32 = _gen(seed), torch.float32
    return [dict(p=_normal(g, (n,), 0.02), g=_normal(g, (n,), 1e-3, getattr(torch, case["grad"])), m=_normal(g, (n,), 1e-3, f32),
                 v=_normal(g, (n,), 1e-3, f32).square_()) for n in _adamw_sizes(case)]


def _prepare_adamw(case, seed):
    from pipelinerl_b200.finetune.optim import FusedAdamW
    inputs = _adamw_inputs(case, seed)
    named = [("bias" if i == 0 else f"w{i}", torch.nn.Parameter(t["p"])) for i, t in enumerate(inputs)]
    opt = FusedAdamW(named, lr=1e-4, weight_decay=0.01, max_grad_norm=case["clip"] or None, grad_dtype=getattr(torch, case["grad"]))
    opt.step_count = 9
    for t, o in zip(inputs, opt.offsets):
        n = t["p"].numel()
        opt.grad[o:o + n], opt.exp_avg[o:o + n], opt.exp_avg_sq[o:o + n] = t["g"], t["m"], t["v"]
    return dict(opt=opt)


def _run_adamw(s):
    o = s["opt"]
    return [o.step(), o.master, o.exp_avg, o.exp_avg_sq, o.shadow_bf16]


def _exact_adamw(case, seed):
    inputs = _adamw_inputs(case, seed)
    norm = math.sqrt(sum(float(t["g"].double().square().sum()) for t in inputs))
    clip = min(1.0, case["clip"] / (norm + 1e-6)) if case["clip"] else 1.0
    total = sum((t["p"].numel() + 63) // 64 * 64 for t in inputs)      # tensors start on 64-element boundaries
    P, M, V = (torch.zeros(total, dtype=F64, device=DEV) for _ in range(3))
    at = 0
    for i, t in enumerate(inputs):
        n = t["p"].numel()
        g = t["g"].double() * clip
        m, v = 0.9 * t["m"].double() + 0.1 * g, 0.999 * t["v"].double() + 0.001 * g * g
        p = t["p"].double() * (1 - 1e-4 * (0.0 if i == 0 else 0.01))
        P[at:at + n] = p - 1e-4 * (m / (1 - 0.9 ** 10)) / ((v / (1 - 0.999 ** 10)).sqrt() + 1e-8)
        M[at:at + n], V[at:at + n] = m, v
        at += (n + 63) // 64 * 64
    return [torch.tensor([norm], dtype=F64), P, M, V, P]


# ---- sampler: token steps ------------------------------------------------------------------------------------------------------
def _contexts(case):
    """Tokens that each sequence holds: the longest first, the others a little shorter."""
    c = case["context"]
    return [max(1, c - (i * c) // (4 * case["batch"])) for i in range(case["batch"])]


def _qwen_engine(case, seed, max_batch, max_len, **kw):
    from pipelinerl_b200.engine import DecodeEngine
    from pipelinerl_b200.model import ParamArena
    cfg = _qwen_config(case, case["layers"], fp32_head=case.get("fp32_head", False))
    arena = ParamArena(cfg, torch.device(DEV))
    for name, t in _qwen_weights(case, seed, case["layers"], cfg.fp32_head).items():
        arena.view(name).copy_(t)
    return DecodeEngine(cfg, arena, max_batch=max_batch, max_seq_len=max_len, device=DEV, eos_id=-1, **kw)


def _cache(case, seed, numel):
    return _normal(_gen(seed + 31), (numel,), 0.5)


def _hold(eng, case, seed, contexts):
    """What the scheduler has on the device for sequences that hold `contexts` tokens and feed one more."""
    i32 = dict(dtype=torch.int32, device=DEV)
    return dict(eng=eng, tokens=_tokens(case, seed + 1, len(contexts)).to(torch.int32).to(DEV), pos=torch.tensor(contexts, **i32),
                count=torch.ones(len(contexts), **i32), vocab=case["vocab"])


def _prepare_decode(case, seed):
    contexts = _contexts(case)
    eng = _qwen_engine(case, seed, case["batch"], case["context"] + 64, max_new_tokens=64)
    eng.kv_cache.copy_(_cache(case, seed, eng.kv_cache.numel()))
    eng.block_table.copy_(torch.arange(1, 1 + eng.block_table.numel(), device=DEV, dtype=torch.int32).view(eng.block_table.shape))
    eng.free_pages.clear()
    s = _hold(eng, case, seed, contexts)
    eng.prompt_len.copy_(s["pos"])
    eng.max_new_t.fill_(64)
    eng.active.fill_(1)
    eng.ignore_eos = True
    _run_decode(s)                                  # the engine of a running program has its step captured
    return s


def _run_decode(s):
    """One token for every sequence, the tokens given by the host; sampled ids and log-probs stay on the device."""
    eng = s["eng"]
    eng.tokens.copy_(s["tokens"])
    eng.positions.copy_(s["pos"])
    torch.add(s["pos"], 1, out=eng.seq_lens)
    eng.gen_count.copy_(s["count"])
    eng.step()
    return eng.logits[:, :s["vocab"]]


def _exact_decode(case, seed):
    B, L, nq, nk, I = case["batch"], case["layers"], case["heads"], case["kv_heads"], case["ff"]
    contexts, w = _contexts(case), _qwen_weights(case, seed, L, case["fp32_head"])
    blocks = (case["context"] + 64 + PAGE - 1) // PAGE
    pages = 1 + B * blocks
    cache = _cache(case, seed, L * 2 * pages * nk * PAGE * 128).view(L, 2, pages, nk, PAGE, 128)
    pos = torch.tensor(contexts, device=DEV)
    h = w["embed_tokens.weight"].double()[_tokens(case, seed + 1, B).to(DEV)]
    for l in range(L):
        p, m = f"layers.{l}.", lambda n: w[p + n].double()  # noqa: B023, E731
        qkv = (_ref_norm(h, m("input_layernorm.weight")) @ m("qkv_proj.weight").T + m("qkv_proj.bias")).view(B, nq + 2 * nk, 128)
        q, k, v = _ref_rope(qkv[:, :nq], pos), _ref_rope(qkv[:, nq:nq + nk], pos), qkv[:, nq + nk:]
        outs = []
        for b in range(B):
            kv = cache[l, :, 1 + b * blocks:1 + (b + 1) * blocks].transpose(1, 2).reshape(2, nk, -1, 128)[:, :, :contexts[b]].double()
            K, V = torch.cat([kv[0], k[b][:, None]], 1), torch.cat([kv[1], v[b][:, None]], 1)
            sc = (q[b].view(nk, -1, 128) @ K.transpose(1, 2)) * 128 ** -0.5
            outs.append((torch.softmax(sc, -1) @ V).reshape(nq * 128))
        h = h + torch.stack(outs) @ m("o_proj.weight").T
        gu = _ref_norm(h, m("post_attention_layernorm.weight")) @ m("gate_up_proj.weight").T
        h = h + (torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]) @ m("down_proj.weight").T
    head = w["lm_head.weight"].double() + (w["lm_head.weight_lo"].double() if case["fp32_head"] else 0.0)
    return _ref_norm(h, w["norm.weight"].double()) @ head.T


# ---- sampler: prompts ------------------------------------------------------------------------------------------------------------
def _wanted(case):
    """Rows of a prompt whose logits are asked for: a spread of them, and the last."""
    n = case["tokens"]
    return sorted({(i * n) // 48 for i in range(48)} | {n - 1})


def _prepare_prompt(case, seed):
    eng = _qwen_engine(case, seed, 2, case["tokens"] + 64, max_new_tokens=16)
    return dict(eng=eng, tokens=_tokens(case, seed, case["tokens"]).tolist(), want=_wanted(case))


def _run_prompt(s):
    eng = s["eng"]
    stream = eng.open_stream()
    logits = eng.feed([(stream, s["tokens"], s["want"])])
    eng.close_stream(stream)
    return logits


def _exact_prompt(case, seed):
    w = _qwen_weights(case, seed, case["layers"])
    h = w["embed_tokens.weight"].double()[_tokens(case, seed, case["tokens"]).to(DEV)]
    for l in range(case["layers"]):
        h = _ref_layer(case, {k: v.double() for k, v in w.items() if k.startswith(f"layers.{l}.")}, l, h, [case["tokens"]])
    return _ref_norm(h[_wanted(case)], w["norm.weight"].double()) @ w["lm_head.weight"].double().T


# ---- hybrid decoder: windowed attention beside the gated delta rule, routed experts ---------------------------------------------
WINDOW, TAPS, EXPERTS, TOP, GROUPS, KEEP, ROT = 1024, 4, 16, 4, 8, 6, 64


def _hybrid_sizes(case):
    """heads, kv heads (attention), heads, kv heads (delta rule), expert width"""
    W = case["width"]
    return W // 128, W // 512, W // 128, W // 256, case["ff"] // 4


def _hybrid_dict(case):
    H, G, RH, RK, ff = _hybrid_sizes(case)
    layer = dict(type="parallel",
                 mixer=dict(left=dict(heads=H, kv_heads=G, dim=128, vdim=128, scale=128 ** -0.5, mask=dict(size=WINDOW),
                                      rot=dict(base=1e6, dims=ROT)),
                            right=dict(heads=RH, kv_heads=RK, dim=128, vdim=128, conv=TAPS)),
                 mlp=dict(kind="moe", router=dict(experts=EXPERTS, top=TOP, scale=1.25, groups=dict(count=GROUPS, keep=KEEP)),
                          expert=dict(ff=ff)))
    return dict(architecture="Modadra", vocab=case["vocab"], width=case["width"], norm=dict(eps=1e-5), residual_mult=0.5,
                logit_softcap=40.0, layers=[layer] * case["layers"])


def _hybrid_weights(case, seed):
    """Tensors of the fused layout: `mix.in` holds the rows [q k v | conv channels q k v | gate | head gates | b a]."""
    W, V = case["width"], case["vocab"]
    H, G, RH, RK, ff = _hybrid_sizes(case)
    g, w = _gen(seed), {}
    gain = lambda n: _normal(g, (n,), 0.2, mean=1.0)  # noqa: E731
    mat = lambda n, k, s=1.0: _normal(g, (n, k), s * k ** -0.5)  # noqa: E731
    for i in range(case["layers"]):
        p, conv = f"l{i}.", (2 * RK + RH) * 128
        rows = (H + 2 * G) * 128 + conv + RH * 128 + H + 2 * RH
        w[p + "mix.in"] = mat((rows + 7) // 8 * 8, W)
        w[p + "mix.left.o"], w[p + "mix.right.o"] = mat(W, H * 128), mat(W, RH * 128)
        w[p + "mix.right.conv"] = _normal(g, (conv, TAPS), 0.6)
        w[p + "mix.right.A_log"] = torch.log(0.05 + 0.5 * torch.rand(RH, generator=g, device=DEV)).to(BF16)
        w[p + "mix.right.dt_bias"] = _normal(g, (RH,))
        w[p + "mix.right.norm"] = gain(128)
        for name in ("mix.left.out", "mix.right.out", "norm1", "norm2"):
            w[p + name] = gain(W)
        w[p + "mlp.router"] = mat(EXPERTS, W, 2.0)
        w[p + "mlp.correction"] = _normal(g, (EXPERTS,), 0.3)
        w[p + "mlp.experts.up"], w[p + "mlp.experts.down"] = mat(EXPERTS * ff, W), mat(EXPERTS * W, ff)
    w["embed"], w["final.norm"], w["head"] = _normal(g, (V, W)), gain(W), mat(V, W, 4.0)
    return w


def _hybrid_engine(case, seed, **kw):
    from pipelinerl_b200.hybrid import HybridConfig, HybridEngine
    from pipelinerl_b200.model import ParamArena
    cfg = HybridConfig.from_modadra(_hybrid_dict(case))
    arena = ParamArena(cfg, torch.device(DEV))
    for name, t in _hybrid_weights(case, seed).items():
        arena.view(name).copy_(t)
    return HybridEngine(cfg, arena, device=DEV, eos_id=-1, **kw)


def _prepare_hybrid_prompt(case, seed):
    eng = _hybrid_engine(case, seed, max_batch=2, max_seq_len=case["tokens"] + 64, max_new_tokens=16)
    return dict(eng=eng, tokens=_tokens(case, seed, case["tokens"]).tolist(), want=_wanted(case))


def _hybrid_rows(case, seed):
    """Prompts of a batch; the last token of each is fed by the first step, one more by the measured one."""
    return [_tokens(case, seed + 100 * (i + 1), n).tolist() for i, n in enumerate(_contexts(case))]


def _prepare_hybrid_decode(case, seed):
    from pipelinerl_b200.engine import SamplingParams
    eng = _hybrid_engine(case, seed, max_batch=case["batch"], max_seq_len=case["context"] + 64, max_new_tokens=64)
    params = SamplingParams(max_tokens=60, ignore_eos=True)
    slots = [eng.add_request(t, params).slot for t in _hybrid_rows(case, seed)]
    eng.step()                                      # the prompts and their last tokens; captures the step
    contexts = [0] * case["batch"]
    for slot, n in zip(slots, _contexts(case)):
        contexts[slot] = n
    s = _hold(eng, case, seed, contexts)
    return s


def _ref_hybrid(case, seed, tokens, want):
    """tokens [B, T] (rows padded at the end), want [(row, position)] -> logits"""
    W, (B, T) = case["width"], tokens.shape
    H, G, RH, RK, ff = _hybrid_sizes(case)
    raw = _hybrid_weights(case, seed)
    rms = lambda x: x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-5)  # noqa: E731
    unit = lambda x: x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    silu = torch.nn.functional.silu
    x = raw["embed"].double()[tokens.to(DEV)]
    back = torch.arange(T, device=DEV)[:, None] - torch.arange(T, device=DEV)
    hidden = (back < 0) | (back >= WINDOW)
    ang = torch.arange(T, device=DEV, dtype=F64)[:, None] * 1e6 ** (-torch.arange(0, ROT, 2, device=DEV, dtype=F64) / ROT)
    cos, sin = torch.cos(ang)[:, None], torch.sin(ang)[:, None]

    def rot(t):                                     # rotate-half on the leading channels
        u, v = t[..., :ROT // 2], t[..., ROT // 2:ROT]
        return torch.cat([u * cos - v * sin, v * cos + u * sin, t[..., ROT:]], -1)
    for i in range(case["layers"]):
        w = {k.split(".", 1)[1]: v.double() for k, v in raw.items() if k.startswith(f"l{i}.")}
        h = rms(x) * w["norm1"]
        sizes = [H * 128, G * 128, G * 128, RK * 128, RK * 128, RH * 128, RH * 128, H, RH, RH]
        q, k, v, rq, rk, rv, rg, hg, b, a = torch.split(h @ w["mix.in"][:sum(sizes)].T, sizes, -1)
        q, k, v = rot(q.reshape(B, T, H, 128)), rot(k.reshape(B, T, G, 128)), v.reshape(B, T, G, 128)
        o = torch.empty(B, T, H, 128, dtype=F64, device=DEV)
        for r in range(B):
            for j in range(H):
                s = (q[r, :, j] @ k[r, :, j // (H // G)].T * 128 ** -0.5).masked_fill_(hidden, -math.inf)
                m = s.amax(-1, keepdim=True).clamp_min(0.0)
                e = torch.exp(s - m)
                o[r, :, j] = e @ v[r, :, j // (H // G)] / (torch.exp(-m) + e.sum(-1, keepdim=True))
        left = (o * torch.sigmoid(hg)[..., None]).reshape(B, T, -1) @ w["mix.left.o"].T
        c = torch.nn.functional.pad(torch.cat([rq, rk, rv], -1), (0, 0, TAPS - 1, 0))
        c = silu(sum(c[:, t:t + T] * w["mix.right.conv"][:, t] for t in range(TAPS)))
        rq, rk, rv = torch.split(c, [RK * 128, RK * 128, RH * 128], -1)
        per = RH // RK
        rq = (unit(rq.reshape(B, T, RK, 128)) * 128 ** -0.5).repeat_interleave(per, 2)
        rk = unit(rk.reshape(B, T, RK, 128)).repeat_interleave(per, 2)
        rv, beta = rv.reshape(B, T, RH, 128), torch.sigmoid(b)
        keep = torch.exp(-torch.exp(w["mix.right.A_log"]) * torch.nn.functional.softplus(a + w["mix.right.dt_bias"]))
        S, o = torch.zeros(B, RH, 128, 128, dtype=F64, device=DEV), torch.empty(B, T, RH, 128, dtype=F64, device=DEV)
        for t in range(T):
            S = S * keep[:, t, :, None, None]
            u = beta[:, t, :, None] * (rv[:, t] - (rk[:, t, :, None] @ S)[:, :, 0])
            S = S + rk[:, t, :, :, None] * u[:, :, None]
            o[:, t] = (rq[:, t, :, None] @ S)[:, :, 0]
        o = rms(o) * w["mix.right.norm"] * silu(rg.reshape(B, T, RH, 128))
        right = o.reshape(B, T, -1) @ w["mix.right.o"].T
        x = x + 0.5 * 0.5 * (rms(left) * w["mix.left.out"] + rms(right) * w["mix.right.out"])
        h = (rms(x) * w["norm2"]).reshape(B * T, W)
        score = torch.sigmoid(h @ w["mlp.router"].T)
        pick = score + w["mlp.correction"]
        rank = pick.view(-1, GROUPS, EXPERTS // GROUPS).topk(2, -1).values.sum(-1)
        closed = torch.ones_like(rank, dtype=torch.bool).scatter_(1, rank.topk(KEEP, -1).indices, False)
        pick = pick.masked_fill(closed.repeat_interleave(EXPERTS // GROUPS, 1), -math.inf)
        chosen = torch.zeros_like(score).scatter_(1, pick.topk(TOP, -1).indices, 1.0) * score
        chosen = chosen / chosen.sum(-1, keepdim=True) * 1.25
        y = torch.zeros_like(h)
        for e in range(EXPERTS):
            at = torch.nonzero(chosen[:, e]).flatten()
            act = torch.nn.functional.gelu(h[at] @ w["mlp.experts.up"][e * ff:(e + 1) * ff].T)
            y.index_add_(0, at, chosen[at, e, None] * (act @ w["mlp.experts.down"][e * W:(e + 1) * W].T))
        x = x + 0.5 * y.view(B, T, W)
    x = torch.stack([x[r, t] for r, t in want])
    z = (rms(x) * raw["final.norm"].double()) @ raw["head"].double().T
    return 40.0 * torch.tanh(z / 40.0)


def _exact_hybrid_prompt(case, seed):
    return _ref_hybrid(case, seed, _tokens(case, seed, case["tokens"])[None], [(0, t) for t in _wanted(case)])


def _exact_hybrid_decode(case, seed):
    """Slots are handed out from zero, so the rows of the logits are the prompts in their order."""
    rows, last = _hybrid_rows(case, seed), _tokens(case, seed + 1, case["batch"]).tolist()
    rows = [r + [t] for r, t in zip(rows, last)]
    T = max(len(r) for r in rows)
    tokens = torch.tensor([r + [8] * (T - len(r)) for r in rows])
    return _ref_hybrid(case, seed, tokens, [(i, len(r) - 1) for i, r in enumerate(rows)])


# ---- the interface ---------------------------------------------------------------------------------------------------------------
_PREPARE = dict(norm=_prepare_norm, attention=_prepare_attention, layer=_prepare_layer, train=_prepare_train, loss=_prepare_loss,
                adamw=_prepare_adamw, decode=_prepare_decode, prompt=_prepare_prompt, hybrid_prompt=_prepare_hybrid_prompt,
                hybrid_decode=_prepare_hybrid_decode)
_RUN = dict(norm=_run_norm, attention=_run_attention, layer=_run_layer, train=_run_train, loss=_run_loss, adamw=_run_adamw,
            decode=_run_decode, prompt=_run_prompt, hybrid_prompt=_run_prompt, hybrid_decode=_run_decode)
_EXACT = dict(norm=_exact_norm, attention=_exact_attention, layer=_exact_layer, train=_exact_train, loss=_exact_loss,
              adamw=_exact_adamw, decode=_exact_decode, prompt=_exact_prompt, hybrid_prompt=_exact_hybrid_prompt,
              hybrid_decode=_exact_hybrid_decode)


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, seed)
    state["kind"] = case["kind"]
    return state


def run(state):
    return _RUN[state["kind"]](state)


def exact(case, seed):
    if case["kind"] == "hybrid_decode" and case["batch"] * case["context"] > 40_000:
        return None
    return _EXACT[case["kind"]](case, seed)


def _pairs(lengths, window=0):
    """(query, key) pairs under the causal mask."""
    return sum(n * (n + 1) // 2 - (max(0, n - window) * (max(0, n - window) + 1) // 2 if window else 0) for n in lengths)


def _layer_params(case):
    H, nq, nk = case["width"], case["heads"] * 128, case["kv_heads"] * 128
    return (nq + 2 * nk) * H + nq * H + 3 * case["ff"] * H


def _hybrid_layer(case):
    """Matrix parameters of a layer: those of every token, and those of one expert."""
    W = case["width"]
    H, G, RH, RK, ff = _hybrid_sizes(case)
    return W * ((2 * H + 2 * G + 2 * RK + 3 * RH) * 128 + H + 2 * RH + EXPERTS), 2 * ff * W


def work(case):
    """Bytes: each input read once, each output written once; FLOPs: products that the results need, none recomputed."""
    k = case["kind"]
    if k == "norm":
        n = case["rows"] * case["width"]
        return dict(bytes=2 * 5 * n, flops=16 * n)                  # x, dy, dres in; y, dx out
    if k == "attention":
        T, nq, nk = sum(_segments(case)), case["heads"], case["kv_heads"]
        return dict(bytes=2 * 128 * T * (2 * (nq + 2 * nk) + 2 * nq), flops=(4 + 10) * 128 * nq * _pairs(_segments(case)))
    if k in ("layer", "train"):
        T, L, H, V = sum(_segments(case)), case.get("layers", 1), case["width"], case["vocab"]
        n = L * _layer_params(case) + (V * H if k == "train" else 0)
        att = (4 + 10) * 128 * case["heads"] * _pairs(_segments(case)) * L
        head = 2 * V * H * T if k == "train" else 0                 # the head's second operand stream
        return dict(bytes=n * (2 + 4) + V * H * 4 + 4 * T * H * L, flops=6 * n * T + att + head)
    if k == "loss":
        n = sum(_segments(case)) * case["vocab"]
        return dict(bytes=8 * n, flops=8 * n)
    if k == "adamw":
        g = 4 if case["grad"] == "float32" else 2
        return dict(bytes=case["params"] * (6 * 4 + g + 2), flops=15 * case["params"])
    if k == "decode":
        B, L, H, V = case["batch"], case["layers"], case["width"], case["vocab"]
        n = L * _layer_params(case) + V * H * (2 if case["fp32_head"] else 1)
        held = sum(_contexts(case)) + B
        return dict(bytes=2 * n + held * L * 2 * case["kv_heads"] * 128 * 2 + 4 * B * V,
                    flops=2 * n * B + 4 * 128 * case["heads"] * held * L)
    if k == "prompt":
        T, L, n = case["tokens"], case["layers"], case["layers"] * _layer_params(case)
        head = case["vocab"] * case["width"]
        return dict(bytes=2 * (n + head) + T * L * 2 * case["kv_heads"] * 128 * 2,
                    flops=2 * n * T + 4 * 128 * case["heads"] * _pairs([T]) * L + 2 * head * len(_wanted(case)))
    common, expert = _hybrid_layer(case)
    H, G, RH, RK, ff = _hybrid_sizes(case)
    L, head = case["layers"], case["vocab"] * case["width"]
    if k == "hybrid_prompt":
        T = case["tokens"]
        return dict(bytes=2 * (L * (common + EXPERTS * expert) + head) + T * L * 2 * G * 128 * 2,
                    flops=L * (2 * T * (common + TOP * expert) + 4 * 128 * H * _pairs([T], WINDOW) + 6 * T * RH * 128 * 128)
                    + 2 * head * len(_wanted(case)))
    B, held = case["batch"], sum(min(n + 1, WINDOW) for n in _contexts(case))
    used = EXPERTS * (1 - (1 - TOP / EXPERTS) ** B)                 # experts that a batch of this size touches
    state = B * RH * 128 * 128 * 4
    return dict(bytes=int(2 * (L * (common + used * expert) + head) + L * (2 * state + held * 2 * G * 128 * 2) + 4 * B * case["vocab"]),
                flops=int(2 * B * (L * (common + TOP * expert) + head) + L * (4 * 128 * H * held + 6 * B * RH * 128 * 128)))


def tolerance(case):
    """Relative errors (2-norm) that rounding alone explains, about four times the distance of the outputs to their 64-bit
    values: one bf16 rounding of an output is 2.3e-3 off, attention 2.4e-3, gradients that come through a layer in bf16
    1.0e-2 and through two 1.6e-2, logits behind four layers 6e-3; sums in fp32 5e-7, of 150 000 terms.  A different
    rounding may also change which expert a token goes to: single logits of the hybrid decoders were 0.12 off."""
    return {"norm": {"rel": 9e-3}, "attention": {"rel": 1e-2}, "layer": {"rel": 3e-2}, "train": {"rel": 3e-2, "max": 0.9},
            "loss": {"rel": 1e-5}, "adamw": {"rel": 4e-3}, "decode": {"rel": 2.4e-2}, "prompt": {"rel": 2.4e-2},
            "hybrid_prompt": {"rel": 3e-2, "max": 0.9}, "hybrid_decode": {"rel": 3e-2, "max": 0.9}}[case["kind"]]
