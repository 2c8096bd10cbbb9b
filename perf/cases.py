"""What users of this framework have it do, as cases that can be timed and compared.

``listed()`` names the cases, ``draw(rng)`` gives one more of the same ranges, ``prepare(case, seed)`` builds what a
program holds before the call (sharded model, optimizer, token batch, weights), ``run(state)`` is one pass through the
public entry points and returns what it computed, ``work(case)`` the bytes and operations that the pass cannot do
without, ``tolerance(case)`` how far another correct implementation of the same precision may be off, ``exact(case, seed)`` what
the pass gives in 64 bits with plain torch.

Kinds:

``train``      one optimisation step of a sharded Llama model (``shard_llama`` + ``configure_optimizer``): AdamW inside
               the reduction, or mixed Muon / AdamW; with activation checkpointing; with two accumulated
               micro-batches, masked targets and gradient clipping
``eval``       logits of a batch of prompts under ``no_grad`` (prefill / validation)
``moe``        one optimisation step of the mixture-of-experts model
``attention``  the causal attention op forward and backward, as a model with its own block calls it
``muon``       ``MatrixMuon.step`` on the matrices that one rank owns of a model
``ops``        the differentiable ops one by one (norm, projections, SwiGLU, loss) in a user's own layer
``module``     ``fully_shard`` on blocks of ordinary ``torch.nn`` layers, AdamW
"""
import math

import torch
import torch.utils.checkpoint
from torch import nn
from torch.distributed.fsdp import MixedPrecisionPolicy

from matrix_fsdp_b200 import configure_optimizer, fully_shard
from matrix_fsdp_b200.models.llama import LlamaConfig, LlamaModel, shard_llama
from matrix_fsdp_b200.models.moe import MoEConfig, MoEModel, configure_moe_optimizer, shard_moe
from matrix_fsdp_b200.ops import attention as attention_ops
from matrix_fsdp_b200.ops import functional as ops
from matrix_fsdp_b200.optim.muon import MatrixMuon
from matrix_fsdp_b200.parallel.unit_collection import collect_param_groups
from matrix_fsdp_b200.utils.training import clip_grad_norm_, device_train_step

DEVICE = "cuda"
BF16 = torch.bfloat16
IGNORED = -100


def listed():
    return [
        # the smallest training step: a two-layer toy model (``bench.py --config tiny``), bound by launches
        dict(name="train_tiny", kind="train", layers=2, heads=2, ffn=688, vocab=1024, batch=2, seq=128, optimizer="adamw",
             checkpointing=False, accumulate=1, masked=False, clip=False),
        # the default benchmark workload
        dict(name="train_8l_h2048", kind="train", layers=8, heads=16, ffn=5504, vocab=32000, batch=4, seq=1024,
             optimizer="adamw", checkpointing=False, accumulate=1, masked=False, clip=False),
        # fine-tuning as people do it: ragged length, padded targets, two micro-batches, clipping
        dict(name="train_ragged_accumulated", kind="train", layers=4, heads=8, ffn=2752, vocab=32000, batch=3, seq=1000,
             optimizer="adamw", checkpointing=False, accumulate=2, masked=True, clip=True),
        # one layer's worth of the 32-layer h4096 configuration: Muon on whole matrices, checkpointing, long rows
        dict(name="train_h4096_muon", kind="train", layers=2, heads=32, ffn=11008, vocab=32000, batch=1, seq=4096,
             optimizer="mixed_muon_adamw", checkpointing=True, accumulate=1, masked=False, clip=False),
        # long context: the published 16384-token rows of the h4096 model, one layer
        dict(name="train_h4096_16k", kind="train", layers=1, heads=32, ffn=11008, vocab=32000, batch=1, seq=16384,
             optimizer="adamw", checkpointing=True, accumulate=1, masked=False, clip=False),
        # scoring a batch of prompts of one odd length
        dict(name="eval_8l_h2048", kind="eval", layers=8, heads=16, ffn=5504, vocab=32000, batch=3, seq=777),
        # the small mixture of experts of ``bench.py --config 5s``
        dict(name="moe_4l_h1024", kind="moe", layers=4, heads=8, experts=16, ffn=512, top_k=2, vocab=8192, batch=2, seq=1024),
        # two layers of the 64-expert top-6 configuration at its own batch
        dict(name="moe_2l_h2048", kind="moe", layers=2, heads=16, experts=64, ffn=1408, top_k=6, vocab=32000, batch=2, seq=4096),
        # attention of a user's own block, odd length that leaves ragged tiles
        dict(name="attention_ragged", kind="attention", batch=3, seq=1333, heads=16),
        # the optimizer step of a rank that owns two blocks of the h2048 model
        dict(name="muon_2_blocks_h2048", kind="muon", blocks=2, hidden=2048, ffn=5504, steps=5, nesterov=True),
        # a layer written with the single ops, short odd batch, part of the targets masked
        dict(name="ops_h1024", kind="ops", tokens=515, hidden=1024, ffn=2752, vocab=8192),
        # ordinary torch.nn blocks under fully_shard
        dict(name="module_4l_h1024", kind="module", layers=4, hidden=1024, ffn=4096, tokens=2048),
    ]


# --------------------------------------------------------------------------------------------- drawing
def _log_int(rng, lo, hi, multiple=1):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / multiple)) * multiple
    return max(lo, min(hi, v))


def _draw_once(rng):
    kind = rng.choice(["train", "train", "train", "eval", "moe", "attention", "muon", "ops", "module"])
    if kind in ("train", "eval"):
        heads = _log_int(rng, 2, 32)
        c = dict(kind=kind, layers=_log_int(rng, 1, 8), heads=heads, ffn=int(heads * 128 * rng.uniform(2.0, 4.0)) // 8 * 8,
                 vocab=_log_int(rng, 1000, 48000, 8), batch=rng.randint(1, 4), seq=_log_int(rng, 64, 4096))
        if kind == "train":
            muon = rng.random() < 0.4
            extras = not muon and rng.random() < 0.4
            c.update(optimizer="mixed_muon_adamw" if muon else "adamw", checkpointing=rng.random() < 0.4,
                     accumulate=2 if extras else 1, masked=extras or rng.random() < 0.3, clip=extras)
        return c
    if kind == "moe":
        heads = _log_int(rng, 2, 16)
        experts = rng.choice([8, 16, 32, 64])
        return dict(kind=kind, layers=_log_int(rng, 1, 4), heads=heads, experts=experts, ffn=_log_int(rng, 128, 1408, 64),
                    top_k=rng.choice([k for k in (1, 2, 4, 6) if k <= experts // 2]), vocab=_log_int(rng, 1000, 32000, 8),
                    batch=rng.randint(1, 2), seq=_log_int(rng, 64, 4096))
    if kind == "attention":
        return dict(kind=kind, batch=rng.randint(1, 4), seq=_log_int(rng, 64, 8192), heads=_log_int(rng, 2, 32))
    if kind == "muon":
        hidden = _log_int(rng, 256, 4096, 64)
        return dict(kind=kind, blocks=rng.randint(1, 3), hidden=hidden, ffn=int(hidden * rng.uniform(2.0, 4.0)) // 8 * 8,
                    steps=5, nesterov=rng.random() < 0.8)
    if kind == "ops":
        hidden = _log_int(rng, 256, 4096, 8)
        return dict(kind=kind, tokens=_log_int(rng, 64, 8192), hidden=hidden, ffn=int(hidden * rng.uniform(2.0, 4.0)) // 8 * 8,
                    vocab=_log_int(rng, 1000, 48000, 8))
    return dict(kind=kind, layers=_log_int(rng, 2, 8), hidden=_log_int(rng, 256, 2048, 8), ffn=_log_int(rng, 512, 8192, 8),
                tokens=_log_int(rng, 64, 8192))


def draw(rng):
    most = max((work(c) for c in listed()), key=lambda w: w["flops"])
    bytes_most = max(work(c)["bytes"] for c in listed())
    while True:
        c = _draw_once(rng)
        w = work(c)
        if w["flops"] <= 0.8 * most["flops"] and w["bytes"] <= 0.8 * bytes_most:
            return c


# --------------------------------------------------------------------------------------------- preparing
def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _tokens(case, gen, masked=False):
    shape = (case["batch"], case["seq"])
    tokens = torch.randint(0, case["vocab"], shape, device=DEVICE, generator=gen)
    targets = torch.randint(0, case["vocab"], shape, device=DEVICE, generator=gen)
    if masked:                       # padded rows of a batch: about a fifth of the targets does not count
        targets = torch.where(torch.rand(shape, device=DEVICE, generator=gen) < 0.2, IGNORED, targets)
    return tokens, targets


def _quiet(model):
    """Training runs keep the per-unit event log off, as the benchmark does."""
    units = collect_param_groups(model)
    for u in units:
        u.runtime_trace_enabled = False
    return units


def _llama(case, seed, **kw):
    torch.manual_seed(seed)
    cfg = LlamaConfig(vocab_size=case["vocab"], hidden=128 * case["heads"], n_layers=case["layers"], n_heads=case["heads"],
                      head_dim=128, ffn=case["ffn"], max_seq_len=case["seq"], **kw)
    with torch.device(DEVICE):
        return LlamaModel(cfg)


def _prepare_train(case, seed):
    model = _llama(case, seed, activation_checkpointing=case["checkpointing"],
                   loss_ignore_index=IGNORED if case["masked"] else None)
    model.loss_is_final = case["accumulate"] == 1
    muon = case["optimizer"] == "mixed_muon_adamw"
    shard_llama(model, mp_policy=MixedPrecisionPolicy(param_dtype=BF16), optimizer_policy="mixed_muon_adamw" if muon else None)
    if muon:
        opt = configure_optimizer(model, "mixed_muon_adamw", muon_lr=0.02, adamw_lr=3e-4, adamw_betas=(0.9, 0.95),
                                  weight_decay=0.1, muon_momentum=0.95, muon_ns_steps=5, muon_adjust_lr_fn="original")
    else:
        # clipping needs the reduced gradients before the update, so the update is fused into the reduction without it
        opt = configure_optimizer(model, "adamw", lr=3e-4, betas=(0.9, 0.95), weight_decay=0.1,
                                  fused_reduce_update=not case["clip"])
    gen = _generator(seed)
    batches = [_tokens(case, gen, case["masked"]) for _ in range(case["accumulate"])]
    return dict(model=model, opt=opt, units=_quiet(model), batches=batches, muon=muon)


def _prepare_eval(case, seed):
    model = _llama(case, seed)
    shard_llama(model, mp_policy=MixedPrecisionPolicy(param_dtype=BF16))
    model.eval()
    return dict(model=model, units=_quiet(model), tokens=_tokens(case, _generator(seed))[0])


def _prepare_moe(case, seed):
    torch.manual_seed(seed)
    cfg = MoEConfig(vocab_size=case["vocab"], hidden=128 * case["heads"], n_layers=case["layers"], n_heads=case["heads"],
                    head_dim=128, n_experts=case["experts"], expert_ffn=case["ffn"], top_k=case["top_k"],
                    max_seq_len=case["seq"], seed=seed)
    with torch.device(DEVICE):
        model = MoEModel(cfg, ep_group=False, device=DEVICE, dtype=BF16)
    shard_moe(model, mp_policy=MixedPrecisionPolicy(param_dtype=BF16), optimizer_policy="mixed_muon_adamw")
    opt = configure_moe_optimizer(model, "mixed_muon_adamw", muon_lr=0.02, adamw_lr=3e-4, adamw_betas=(0.9, 0.95),
                                  weight_decay=0.1, muon_momentum=0.95, muon_ns_steps=5, muon_adjust_lr_fn="original")
    return dict(model=model, opt=opt, units=_quiet(model), batch=_tokens(case, _generator(seed)))


def _prepare_attention(case, seed):
    gen = _generator(seed)
    rows, hidden = case["batch"] * case["seq"], 128 * case["heads"]
    qkv = torch.randn(rows, 3 * hidden, device=DEVICE, generator=gen).to(BF16)
    dout = torch.randn(rows, hidden, device=DEVICE, generator=gen).to(BF16)
    return dict(qkv=qkv, dout=dout, shape=(case["batch"], case["seq"], case["heads"], 128))


def _muon_shapes(case):
    h, f = case["hidden"], case["ffn"]
    return [(h, h)] * 4 + [(f, h)] * 2 + [(h, f)]


def _prepare_muon(case, seed):
    gen = _generator(seed)
    params = []
    for _ in range(case["blocks"]):
        for shape in _muon_shapes(case):
            p = nn.Parameter(0.02 * torch.randn(shape, device=DEVICE, generator=gen))
            p.grad = 1e-3 * torch.randn(shape, device=DEVICE, generator=gen)
            params.append(p)
    opt = MatrixMuon(params, lr=0.02, weight_decay=0.1, momentum=0.95, nesterov=case["nesterov"], ns_steps=case["steps"],
                     adjust_lr_fn="match_rms_adamw")
    return dict(opt=opt, params=params)


def _prepare_ops(case, seed):
    gen = _generator(seed)
    t, h, f, v = case["tokens"], case["hidden"], case["ffn"], case["vocab"]

    def weight(rows, cols):
        return nn.Parameter((0.02 * torch.randn(rows, cols, device=DEVICE, generator=gen)).to(BF16))

    w = dict(norm1=nn.Parameter(torch.ones(h, device=DEVICE, dtype=BF16)), gate_up=weight(2 * f, h), down=weight(h, f),
             norm2=nn.Parameter(torch.ones(h, device=DEVICE, dtype=BF16)), head=weight(v, h))
    x = torch.randn(t, h, device=DEVICE, generator=gen).to(BF16).requires_grad_(True)
    targets = torch.randint(0, v, (t,), device=DEVICE, generator=gen)
    targets = torch.where(torch.rand(t, device=DEVICE, generator=gen) < 0.2, IGNORED, targets)
    return dict(w=w, x=x, targets=targets)


class _MLPBlock(nn.Module):
    def __init__(self, hidden, ffn):
        super().__init__()
        self.norm, self.up, self.down = nn.LayerNorm(hidden), nn.Linear(hidden, ffn), nn.Linear(ffn, hidden)

    def forward(self, x):
        return x + self.down(nn.functional.gelu(self.up(self.norm(x))))


def _prepare_module(case, seed):
    torch.manual_seed(seed)
    with torch.device(DEVICE):
        model = nn.Sequential(*[_MLPBlock(case["hidden"], case["ffn"]) for _ in range(case["layers"])])
    for block in model:
        fully_shard(block, mp_policy=MixedPrecisionPolicy(param_dtype=BF16))
    opt = configure_optimizer(model, "adamw", lr=3e-4, betas=(0.9, 0.95), weight_decay=0.1)
    gen = _generator(seed)
    x, y = (torch.randn(case["tokens"], case["hidden"], device=DEVICE, generator=gen).to(BF16) for _ in range(2))
    return dict(model=model, opt=opt, units=_quiet(model), x=x, y=y)


class _State(dict):
    """Gives the model back when it is dropped: a hook on a parameter refers to the parameter's unit, a cycle
    through the tensor that Python's collector does not see."""

    def __del__(self):
        for unit in self.get("units", ()):
            for handle in unit._hook_handles:
                handle.remove()


_PREPARE = dict(train=_prepare_train, eval=_prepare_eval, moe=_prepare_moe, attention=_prepare_attention,
                muon=_prepare_muon, ops=_prepare_ops, module=_prepare_module)


def prepare(case, seed):
    return _State(_PREPARE[case["kind"]](case, int(seed)), kind=case["kind"])


# --------------------------------------------------------------------------------------------- running
def _weights(units):
    return [u.flat_buffer.local_shard for u in units]


def _run_train(s):
    model, opt = s["model"], s["opt"]
    if len(s["batches"]) == 1:
        loss = device_train_step(model, opt, *s["batches"][0])
    else:
        with model.no_sync():
            for tokens, targets in s["batches"][:-1]:
                (model(tokens, targets) / len(s["batches"])).backward()
        tokens, targets = s["batches"][-1]
        loss = model(tokens, targets) / len(s["batches"])
        loss.backward()
        clip_grad_norm_(model, 1.0)
        opt.step()
        opt.zero_grad(set_to_none=True)
        loss = loss.detach()
    out = dict(loss=loss, weights=_weights(s["units"]))
    if not s["muon"]:                # the first moments are the gradients of the steps so far
        out["moments"] = [opt.optimizer.flat_state(u)["exp_avg"] for u in s["units"]]
    return out


def _run_eval(s):
    with torch.no_grad():
        return s["model"](s["tokens"])


def _run_moe(s):
    loss = device_train_step(s["model"], s["opt"], *s["batch"])
    return dict(loss=loss, weights=_weights(s["units"]), experts=s["opt"].experts.masters)


def _run_attention(s):
    out, lse = attention_ops.attention_fwd(s["qkv"], *s["shape"])
    dqkv = attention_ops.attention_bwd(s["dout"], s["qkv"], out, lse, *s["shape"])
    return out, lse, dqkv


def _run_muon(s):
    s["opt"].step()
    return s["params"], [s["opt"].state[p]["momentum_buffer"] for p in s["params"]]


def _run_ops(s):
    w, x = s["w"], s["x"]
    h = ops.linear(ops.swiglu(ops.linear(ops.rms_norm(x, w["norm1"]), w["gate_up"])), w["down"]) + x
    logits = ops.linear(ops.rms_norm(h, w["norm2"]), w["head"])
    loss = ops.fused_cross_entropy(logits, s["targets"], ignore_index=IGNORED)
    grads = torch.autograd.grad(loss, [x, *w.values()])
    return loss.detach(), grads


def _run_module(s):
    loss = nn.functional.mse_loss(s["model"](s["x"]).float(), s["y"].float())
    loss.backward()
    s["opt"].step()
    s["opt"].zero_grad(set_to_none=True)
    return dict(loss=loss.detach(), weights=_weights(s["units"]),
                moments=[s["opt"].optimizer.flat_state(u)["exp_avg"] for u in s["units"]])


_RUN = dict(train=_run_train, eval=_run_eval, moe=_run_moe, attention=_run_attention, muon=_run_muon, ops=_run_ops,
            module=_run_module)


def run(state):
    return _RUN[state["kind"]](state)


# --------------------------------------------------------------------------------------------- work
def _ns_flops(rows, cols, steps):
    """Newton-Schulz iterations: the Gram matrix and its square are symmetric, so half of each is enough."""
    n, m = min(rows, cols), max(rows, cols)
    return float(steps) * (n * n * m + n ** 3 + 2 * n * n * m)


_ADAMW_BYTES = 2 * 12 + 2 + 2 + 2   # master and both moments read and written, bf16 weights and gradients
_MUON_BYTES = 2 * 8 + 2 + 2 + 2     # master and momentum


def work(case):
    kind = case["kind"]
    if kind in ("train", "eval", "moe"):
        h, f, v, n, s = 128 * case["heads"], case["ffn"], case["vocab"], case["layers"], case["seq"]
        t = case["batch"] * s
        attention = 4.0 * t * s * h / 2
        if kind == "moe":
            k, e = case["top_k"], case["experts"]
            dense, experts = 4 * h * h + e * h, 3 * h * f * e
            flops = 6.0 * t * (n * (dense + 3 * h * f * k) + v * h) + n * 3.5 * attention
            flops += n * (4 * _ns_flops(h, h, 5) + e * (_ns_flops(2 * f, h, 5) + _ns_flops(h, f, 5)))
            return dict(bytes=n * (4 * h * h + experts) * _MUON_BYTES + (n * e * h + 2 * v * h) * _ADAMW_BYTES + 16.0 * t, flops=flops)
        layer = 4 * h * h + 3 * h * f
        if kind == "eval":
            return dict(bytes=2.0 * (n * layer + v * h + t * h) + 2.0 * t * v + 8 * t,
                        flops=2.0 * t * (n * layer + v * h) + n * attention)
        a = case["accumulate"]
        passes, att_passes = (4, 4.5) if case["checkpointing"] else (3, 3.5)
        flops = a * (2.0 * t * (passes * n * layer + 3 * v * h) + n * att_passes * attention)
        if case["optimizer"] == "adamw":
            return dict(bytes=(n * layer + 2 * v * h) * _ADAMW_BYTES + 16.0 * t * a, flops=flops)
        flops += n * (4 * _ns_flops(h, h, 5) + 3 * _ns_flops(f, h, 5))
        return dict(bytes=n * layer * _MUON_BYTES + 2 * v * h * _ADAMW_BYTES + 16.0 * t, flops=flops)
    if kind == "attention":
        b, s, n = case["batch"], case["seq"], case["heads"]
        return dict(bytes=2.0 * b * s * n * 128 * (3 + 1 + 1 + 1 + 3 + 3) + 8.0 * b * s * n, flops=3.5 * 4.0 * b * n * s * s * 128 / 2)
    if kind == "muon":
        shapes = _muon_shapes(case) * case["blocks"]
        return dict(bytes=20.0 * sum(r * c for r, c in shapes), flops=sum(_ns_flops(r, c, case["steps"]) for r, c in shapes))
    if kind == "ops":
        t, h, f, v = case["tokens"], case["hidden"], case["ffn"], case["vocab"]
        weights = 3 * h * f + v * h
        return dict(bytes=2.0 * (2 * weights + 2 * t * h) + 8 * t, flops=6.0 * t * weights)
    h, f, t, n = case["hidden"], case["ffn"], case["tokens"], case["layers"]
    return dict(bytes=2.0 * n * h * f * _ADAMW_BYTES + 4.0 * t * h, flops=12.0 * t * n * h * f)


def tolerance(case):
    """About four times the relative error that the path shows against another implementation of the same precision
    (the same module on PyTorch's bf16 kernels; attention against fp32), at most 3e-2: first moments of an 8-layer
    step 2.5e-2 and logits 1.8e-2 (bf16 rounding of every layer adds up), Muon-updated weights 2e-3, expert weights
    5e-3 (a few tokens of equal rounded logits change their expert), attention 2.4e-3, Newton-Schulz 2.7e-3, the
    single ops 4.7e-3."""
    kind = case["kind"]
    if kind == "train":
        return {"rel": 1e-2, "max": 0.2} if case["optimizer"] == "mixed_muon_adamw" else {"rel": 3e-2}
    return {"eval": {"rel": 3e-2}, "moe": {"rel": 2e-2, "max": 0.7}, "attention": {"rel": 1e-2, "max": 0.3},
            "muon": {"rel": 1e-2, "max": 0.15}, "ops": {"rel": 2e-2, "max": 0.4}, "module": {"rel": 1e-2}}[kind]


# --------------------------------------------------------------------------------------------- in 64 bits
def _norm64(x, w, eps=1e-5):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _silu64(x):
    return x * torch.sigmoid(x)


def _head_attention64(q, k, v):
    """One head's [S, 128] rows; returns the output and the log-sum-exp of the scaled causal scores."""
    scores = q @ k.T / math.sqrt(q.shape[-1])
    scores = scores.masked_fill(torch.ones_like(scores, dtype=torch.bool).triu_(1), -math.inf)
    lse = torch.logsumexp(scores, -1)
    return torch.exp(scores - lse[:, None]) @ v, lse


def _attention64(qkv, batch, seq, heads):
    """``qkv``: [batch * seq, 3 * heads * 128]; one head at a time, recomputed in the backward pass."""
    parts = qkv.view(batch, seq, 3, heads, 128)
    outs, lses = [], []
    for b in range(batch):
        pairs = [torch.utils.checkpoint.checkpoint(_head_attention64, *(parts[b, :, i, n] for i in range(3)), use_reentrant=False)
                 for n in range(heads)]
        outs.append(torch.stack([o for o, _ in pairs], 1).reshape(seq, heads * 128))
        lses.append(torch.stack([l for _, l in pairs]))
    return torch.cat(outs), torch.stack(lses)


def _rope64(x, seq):
    """``x``: [batch, seq, heads, 128], pairs (i, i + 64)."""
    inv = 10000.0 ** (-torch.arange(0, 128, 2, device=x.device, dtype=torch.float64) / 128)
    angle = (torch.arange(seq, device=x.device, dtype=torch.float64)[:, None] * inv)[None, :, None, :]
    a, b = x[..., :64], x[..., 64:]
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], -1)


def _units64(units):
    """Per unit: the flat fp32 weights and, by name, 64-bit views of their bf16 values that take gradients."""
    flats, named = [], []
    for u in units:
        flat = u.flat_buffer.local_shard.detach().clone()
        leaf = flat.to(BF16).double().requires_grad_(True)
        flats.append((flat.double(), leaf))
        named.append({mp.fqn: leaf[mp.offset:mp.offset + mp.numel].view(mp.shape) for mp in u.registry})
    return flats, named


def _llama64(case, named, tokens):
    embed = next(n for n in named if set(n) == {"weight"})["weight"]
    head = next(n for n in named if any("lm_head" in k for k in n))
    blocks = [n for n in named if any("w_gate" in k for k in n)]
    assert len(blocks) == case["layers"]
    b, s, h = *tokens.shape, 128 * case["heads"]
    x = embed[tokens.reshape(-1)]
    for w in blocks:
        xn = _norm64(x, w["attn_norm.weight"])
        q, k, v = (xn @ w[n].T for n in ("wq.weight", "wk.weight", "wv.weight"))
        q, k = (_rope64(t.view(b, s, -1, 128), s).reshape(b * s, h) for t in (q, k))
        x = x + _attention64(torch.cat([q, k, v], 1), b, s, case["heads"])[0] @ w["wo.weight"].T
        xn = _norm64(x, w["mlp_norm.weight"])
        x = x + (_silu64(xn @ w["w_gate.weight"].T) * (xn @ w["w_up.weight"].T)) @ w["w_down.weight"].T
    return _norm64(x, head["final_norm.weight"]) @ head["lm_head.weight"].T


def _adamw64(flats, grads, lr=3e-4, decay=0.1, beta1=0.9, eps=1e-8):
    """First step: both moments are the gradient's after bias correction."""
    weights = [p * (1 - lr * decay) - lr * g / (g.abs() + eps) for (p, _), g in zip(flats, grads)]
    return dict(weights=weights, moments=[(1 - beta1) * g for g in grads])


def _exact_train(case, seed):
    s = _prepare_train(case, seed)
    flats, named = _units64(s["units"])
    loss, grads = 0.0, None
    for tokens, targets in s["batches"]:
        part = nn.functional.cross_entropy(_llama64(case, named, tokens), targets.reshape(-1), ignore_index=IGNORED) / len(s["batches"])
        got = torch.autograd.grad(part, [leaf for _, leaf in flats])
        grads = got if grads is None else [a + b for a, b in zip(grads, got)]
        loss = part.detach()
    _State(s)
    if s["muon"]:
        return dict(loss=loss, weights=[None] * len(flats))
    if case["clip"]:
        norm = torch.sqrt(sum((g * g).sum() for g in grads))
        grads = [g * torch.clamp(1.0 / (norm + 1e-6), max=1.0) for g in grads]
    return dict(loss=loss, **_adamw64(flats, grads))


def _exact_eval(case, seed):
    s = _prepare_eval(case, seed)
    with torch.no_grad():
        out = _llama64(case, _units64(s["units"])[1], s["tokens"]).view(*s["tokens"].shape, -1)
    _State(s)
    return out


def _exact_attention(case, seed):
    s = _prepare_attention(case, seed)
    qkv = s["qkv"].double().requires_grad_(True)
    out, lse = _attention64(qkv, *s["shape"][:3])
    return out.detach(), lse.detach(), torch.autograd.grad(out, qkv, s["dout"].double())[0]


def _exact_muon(case, seed):
    s = _prepare_muon(case, seed)
    params, moments = [], []
    for p in s["params"]:
        g = p.grad.double()
        m = 0.05 * g
        x = 0.05 * g + 0.95 * m if case["nesterov"] else m
        x = x / x.norm()
        for _ in range(case["steps"]):
            gram = x.T @ x if x.shape[0] > x.shape[1] else x @ x.T
            poly = -4.7750 * gram + 2.0315 * gram @ gram
            x = 3.4445 * x + (x @ poly if x.shape[0] > x.shape[1] else poly @ x)
        params.append(p.detach().double() * (1 - 0.02 * 0.1) - 0.02 * 0.2 * math.sqrt(max(p.shape)) * x)
        moments.append(m)
    return params, moments


def _exact_ops(case, seed):
    s = _prepare_ops(case, seed)
    w = {k: v.detach().double().requires_grad_(True) for k, v in s["w"].items()}
    x = s["x"].detach().double().requires_grad_(True)
    gate, up = (_norm64(x, w["norm1"]) @ w["gate_up"].T).chunk(2, -1)
    h = (_silu64(gate) * up) @ w["down"].T + x
    loss = nn.functional.cross_entropy(_norm64(h, w["norm2"]) @ w["head"].T, s["targets"], ignore_index=IGNORED)
    return loss.detach(), torch.autograd.grad(loss, [x, *w.values()])


def _exact_module(case, seed):
    s = _prepare_module(case, seed)
    flats, named = _units64(s["units"])
    x = s["x"].double()
    for w in named:
        y = nn.functional.layer_norm(x, (case["hidden"],), w["norm.weight"], w["norm.bias"])
        x = x + nn.functional.linear(nn.functional.gelu(nn.functional.linear(y, w["up.weight"], w["up.bias"])),
                                     w["down.weight"], w["down.bias"])
    loss = nn.functional.mse_loss(x, s["y"].double())
    grads = torch.autograd.grad(loss, [leaf for _, leaf in flats])
    _State(s)
    return dict(loss=loss.detach(), **_adamw64(flats, grads))


_EXACT = dict(train=_exact_train, eval=_exact_eval, attention=_exact_attention, muon=_exact_muon, ops=_exact_ops,
              module=_exact_module)


def exact(case, seed):
    """``None`` where 64 bits take too long (the largest products, the longest rows) and for the mixture of experts,
    where a rounding decides which expert a token goes to and the rest follows from that."""
    if case["kind"] == "moe" or work(case)["flops"] > 4e13 or case.get("seq", 0) > 4096:
        return None
    return _EXACT[case["kind"]](case, int(seed))
