"""Performance cases: the work a user of the framework has it do, through its public entry points.

Four kinds of case, each over the range of sizes it is used at:

``linear``     one fused (multi-)LoRA linear layer, forward and usually backward through autograd
               (``fused_linear_lora`` / ``fused_linear_multi_lora``), bf16 or NF4 base weight
``attention``  causal variable-length grouped-query attention on a packed batch
               (``packed_attention``), forward alone or forward and backward
``step``       one optimizer step of ``MultiLoRATrainer.train_step``: token arrays to the device,
               forward, backward, AdamW of every adapter, loss back to the host
``nf4``        quantising a base weight to NF4 (model loading) and expanding it again

Shapes are those of ``models/config.py`` and of the kernel and layer benchmarks under ``cli/``.
The layer stacks are cut to one to four layers, since all layers of a model do the same work.
"""

from __future__ import annotations

import math
import random

import torch

from lorafusion_b200.models.config import AdapterSpec, get_model_config
from lorafusion_b200.ops import (dequantize_nf4, fused_linear_lora, fused_linear_multi_lora,
                                 prepare_multi_lora_batch_info, quantize_nf4)
from lorafusion_b200.ops.attention import build_attn_tiles, packed_attention
from lorafusion_b200.train.data import LengthDistribution, MicroBatchSpec
from lorafusion_b200.train.trainer import MultiLoRATrainer, OptimizerConfig

DEVICE = "cuda"
HEAD_DIM = 128
TILE = 128


# ---------------------------------------------------------------------------- descriptions
def _linear(name, segments, k, n, ranks, dropout, backward=True, nf4=False, bias=False):
    """``segments``: tokens of each adapter's part of the microbatch, ``"512,300"``; one number
    is the single-adapter layer.  ``ranks`` / ``dropout``: one value per segment."""
    c = dict(kind="linear", segments=segments, k=k, n=n, ranks=ranks, dropout=dropout, backward=backward,
             nf4=nf4, bias=bias)
    return dict(c, name=name) if name else c


def _attention(name, tokens, median, heads, kv_heads, backward=True):
    """A packed batch of ``tokens`` tokens, sequence lengths lognormal around ``median``."""
    c = dict(kind="attention", tokens=tokens, median=median, heads=heads, kv_heads=kv_heads, backward=backward)
    return dict(c, name=name) if name else c


def _step(name, model, layers, tokens, medians, ranks, dropout, nf4=False, recompute="auto", microbatches=1):
    """``medians`` / ``ranks`` / ``dropout``: one value per adapter (its samples' median length)."""
    c = dict(kind="step", model=model, layers=layers, tokens=tokens, medians=medians, ranks=ranks, dropout=dropout,
             nf4=nf4, recompute=recompute, microbatches=microbatches)
    return dict(c, name=name) if name else c


def _nf4(name, n, k):
    c = dict(kind="nf4", n=n, k=k)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a single short sample through one small layer: launches and host work, nothing else
        _linear("linear-100", "100", 1024, 1536, "16", "0.1"),
        # one job's 16K-token microbatch split over two: the single-adapter layer of the kernel benchmark
        _linear("linear-8192", "8192", 4096, 4096, "16", "0.1"),
        # evaluation of an adapter: forward only, no dropout, q|k|v projection with bias, ragged token count
        _linear("linear-eval-1000", "1000", 5120, 7168, "16", "0", backward=False, bias=True),
        # four jobs packed into one ragged microbatch, ranks and dropout rates of their own
        _linear("linear-4jobs", "1700,3011,900,2500", 8192, 8192, "16,16,32,64", "0.1,0,0.05,0.1"),
        # the same on an NF4 base (the QLoRA configuration), a short microbatch of two jobs
        _linear("linear-nf4-2jobs", "700,1313", 8192, 10240, "16,16", "0.1,0.1", nf4=True),
        # attention of a small batch, forward only (evaluation)
        _attention("attention-600", 600, 200, 8, 2, backward=False),
        # attention of a training microbatch of short samples, where most query tiles see few key tiles
        _attention("attention-mixed-16k", 16384, 512, 64, 8),
        # ... and of long documents, where the inner loop dominates
        _attention("attention-long-8k", 8192, 8192, 32, 8),
        # a miniature model's step: every kernel is short, the host and the gaps between launches count
        _step("step-small", "small", 4, 1500, "256,512", "16,8", "0.1,0", recompute="False"),
        # two layers of the 8B shape with loss head, one adapter, full microbatch, activations kept
        _step("step-8b", "llama-3.1-8b", 2, 16384, "512", "16", "0.1"),
        # two layers of the 70B shape on an NF4 base, four jobs, full microbatch, layers recomputed
        _step("step-70b-nf4", "llama-3.1-70b", 2, 16384, "256,512,1024,2048", "16,16,16,16", "0.1,0.1,0.1,0.1",
              nf4=True, recompute="True"),
        # loading a base weight as NF4 and expanding it (the 8B gate|up projection)
        _nf4("nf4-gate-up", 28672, 4096),
    ]


def _log_int(rng, lo, hi, multiple=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi, max(lo, round(v / multiple) * multiple)))


def draw(rng):
    limit = _cost(listed()[-2])
    while True:
        c = _draw_any(rng)
        if _cost(c) <= limit:
            return c


def _draw_any(rng):
    kind = rng.choice(["linear"] * 5 + ["attention"] * 3 + ["step"] * 3 + ["nf4"])
    if kind == "linear":
        jobs = rng.choice([1, 1, 2, 3, 4])
        total = _log_int(rng, 64 * jobs, 16384)
        cuts = sorted(rng.sample(range(1, total), jobs - 1))
        segments = [b - a for a, b in zip([0] + cuts, cuts + [total])]
        rate = rng.choice([0.0, 0.05, 0.1])
        rates = [rate if rng.random() < 0.7 else rng.choice([0.0, 0.05, 0.1, 0.2]) for _ in range(jobs)]
        nf4 = rng.random() < 0.3
        step = 256 if nf4 else 8
        return _linear(None, ",".join(map(str, segments)), _log_int(rng, 512, 8192, step), _log_int(rng, 512, 28672, step),
                       ",".join(str(rng.choice([4, 8, 16, 16, 24, 32, 64])) for _ in range(jobs)),
                       ",".join("%g" % r for r in rates), backward=rng.random() < 0.75, nf4=nf4,
                       bias=rng.random() < 0.2)
    if kind == "attention":
        heads, kv = rng.choice([(4, 2), (8, 2), (32, 8), (40, 8), (64, 8)])
        tokens = _log_int(rng, 100, 16384)
        return _attention(None, tokens, min(tokens, _log_int(rng, 64, 8192)), heads, kv, backward=rng.random() < 0.7)
    if kind == "step":
        model, layers = rng.choice([("small", 4), ("small", 2), ("llama-3.1-8b", 1), ("llama-3.1-8b", 2),
                                    ("qwen2.5-32b", 1), ("llama-3.1-70b", 1)])
        jobs = rng.choice([1, 2, 4])
        return _step(None, model, layers, _log_int(rng, 512, 16384),
                     ",".join(rng.choice(["256", "512", "1024", "2048"]) for _ in range(jobs)),
                     ",".join(rng.choice(["8", "16", "16", "32"]) for _ in range(jobs)),
                     ",".join(rng.choice(["0", "0.1", "0.1"]) for _ in range(jobs)),
                     nf4=model != "small" and rng.random() < 0.5, recompute=rng.choice(["auto", "True", "False"]),
                     microbatches=rng.choice([1, 1, 2]))
    return _nf4(None, _log_int(rng, 512, 28672), _log_int(rng, 512, 8192, 64))


def _cost(case):
    w = work(case)
    return max(w["flops"] / 1e15, w["bytes"] / 6e12)


def _ints(text):
    return [int(v) for v in text.split(",")]


def _floats(text):
    return [float(v) for v in text.split(",")]


def _lengths(tokens, median, mix):
    """Sequence lengths of a packed batch: the same for every seed, summing to ``tokens``."""
    dist = LengthDistribution(median, 0.6, 32, 8192)
    out, left, i = [], tokens, 0
    while left > 0:
        n = min(left, int(dist.sample(1, 1000 * mix + i)[0]))
        if left - n < 32:   # no tail of a few tokens
            n = left if left <= 8192 else n
        out.append(n)
        left -= n
        i += 1
    return out


def _microbatches(case):
    """Host descriptions of the step's microbatches: every adapter gets an equal share of the
    tokens, filled with samples of its own length distribution."""
    medians = _ints(case["medians"])
    share = case["tokens"] // len(medians)
    return [MicroBatchSpec([(a, _lengths(share - share % 2 if a % 2 else share, m, 7 + 10 * i + a))
                            for a, m in enumerate(medians)]) for i in range(case["microbatches"])]


# ---------------------------------------------------------------------------- preparation
class _Source:
    """Values on the GPU, made from one seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEVICE).manual_seed(int(seed))

    def normal(self, *shape, std=1.0):
        t = torch.empty(*shape, dtype=torch.float32, device=DEVICE)
        return t.normal_(0.0, std, generator=self.g).to(torch.bfloat16)

    def uniform(self, *shape, bound):
        t = torch.empty(*shape, dtype=torch.float32, device=DEVICE)
        return t.uniform_(-bound, bound, generator=self.g).to(torch.bfloat16)


def prepare(case, seed):
    return {"linear": _prepare_linear, "attention": _prepare_attention, "step": _prepare_step,
            "nf4": _prepare_nf4}[case["kind"]](case, seed)


def _prepare_linear(case, seed):
    src = _Source(seed)
    seg, ranks, rates = _ints(case["segments"]), _ints(case["ranks"]), _floats(case["dropout"])
    k, n = case["k"], case["n"]
    padded = [(s + TILE - 1) // TILE * TILE for s in seg]
    rows = seg[0] if len(seg) == 1 else sum(padded)
    grad = case["backward"]
    w = src.normal(n, k, std=0.02)
    state = dict(
        case=case, seed=int(seed) & 0xFFFF,
        x=src.normal(rows, k).requires_grad_(grad),
        w=quantize_nf4(w) if case["nf4"] else w,
        bias=src.normal(n, std=0.02) if case["bias"] else None,
        a=[src.uniform(r, k, bound=1.0 / math.sqrt(k)).requires_grad_(grad) for r in ranks],
        b=[src.normal(n, r, std=0.01).requires_grad_(grad) for r in ranks],
        dy=src.normal(rows, n) if grad else None)
    if len(seg) > 1:   # made once per microbatch, used by every layer of the model
        state["info"] = prepare_multi_lora_batch_info(
            seg, list(range(len(seg))), ranks, rates, [32.0 / r for r in ranks], device=DEVICE,
            seed=state["seed"], num_adapters=len(seg))
    else:
        state["alpha"], state["rate"] = 32.0 / ranks[0], rates[0]
    return state


def _prepare_attention(case, seed):
    src = _Source(seed)
    tokens, heads, kv = case["tokens"], case["heads"], case["kv_heads"]
    cu = [0]
    for n in _lengths(tokens, case["median"], 1):
        cu.append(cu[-1] + n)
    return dict(case=case, tiles=build_attn_tiles(cu, DEVICE),
                qkv=src.normal(tokens, (heads + 2 * kv) * HEAD_DIM).requires_grad_(case["backward"]),
                d_out=src.normal(tokens, heads * HEAD_DIM) if case["backward"] else None)


def _prepare_step(case, seed):
    cfg = get_model_config(case["model"]).with_layers(case["layers"])
    adapters = [AdapterSpec("lora_%d" % i, r=r, lora_alpha=32.0, dropout=p)
                for i, (r, p) in enumerate(zip(_ints(case["ranks"]), _floats(case["dropout"])))]
    trainer = MultiLoRATrainer(cfg, adapters, torch.device(DEVICE, torch.cuda.current_device()), quantize=case["nf4"],
                               recompute={"True": True, "False": False, "auto": "auto"}[case["recompute"]],
                               optim=OptimizerConfig(lr=1e-4), seed=int(seed) & 0xFFFFFF, init_b_std=0.01,
                               max_tokens=16384)
    specs = _microbatches(case)
    trainer.stage.plan_activations(max(s.padded_total_tokens for s in specs))
    return dict(case=case, trainer=trainer, specs=specs, seed=int(seed) & 0xFFFF,
                host=trainer.stage_batches(specs, int(seed) & 0xFFFF))


def _prepare_nf4(case, seed):
    return dict(case=case, w=_Source(seed).normal(case["n"], case["k"], std=0.02))


# ---------------------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    if case["kind"] == "linear":
        if "info" in state:
            y = fused_linear_multi_lora(state["x"], state["w"], lora_a_list=state["a"], lora_b_list=state["b"],
                                        batch_info=state["info"], linear_bias=state["bias"], seed=state["seed"])
        else:
            y = fused_linear_lora(state["x"], state["w"], state["a"][0], state["b"][0], state["alpha"],
                                  seed=state["seed"], dropout_p=state["rate"], linear_bias=state["bias"])
        if not case["backward"]:
            return {"y": y}
        return {"y": y.detach(), "grads": torch.autograd.grad(y, [state["x"], *state["a"], *state["b"]], state["dy"])}
    if case["kind"] == "attention":
        out = packed_attention(state["qkv"], state["tiles"], case["heads"], case["kv_heads"])
        if not case["backward"]:
            return {"out": out}
        return {"out": out.detach(), "grads": torch.autograd.grad(out, [state["qkv"]], state["d_out"])}
    if case["kind"] == "step":
        t = state["trainer"]
        loss = t.train_step(state["specs"], state["seed"], host=state["host"])
        arena = t.stage.arena
        return {"loss": loss, "weights": arena.master, "m": arena.m, "v": arena.v}
    q = quantize_nf4(state["w"])
    return {"packed": q.packed, "scales": q.absmax_q, "nested": q.nested, "w": dequantize_nf4(q)}


# ---------------------------------------------------------------------------- work and tolerance
def _linear_work(tokens, k, n, rank, backward, weight_bytes):
    flops = 2.0 * tokens * (k * n + rank * (k + n))
    nbytes = 2.0 * (tokens * (k + n) + rank * (k + n)) + weight_bytes
    if backward:
        flops += 2.0 * tokens * (k * n + 2 * rank * (k + n))
        nbytes += 2.0 * (tokens * (k + n) + rank * (k + n))
    return flops, nbytes


def _causal_pairs(lengths):
    return sum(n * (n + 1) / 2.0 for n in lengths)


def work(case):
    if case["kind"] == "linear":
        seg, ranks = _ints(case["segments"]), _ints(case["ranks"])
        k, n = case["k"], case["n"]
        wb = k * n * (0.5 + 1.0 / 64) if case["nf4"] else 2.0 * k * n
        flops = nbytes = 0.0
        for s, r in zip(seg, ranks):
            f, b = _linear_work(s, k, n, r, case["backward"], 0.0)
            flops, nbytes = flops + f, nbytes + b
        return {"bytes": nbytes + wb, "flops": flops}
    if case["kind"] == "attention":
        tokens, heads, kv = case["tokens"], case["heads"], case["kv_heads"]
        flops = 4.0 * HEAD_DIM * heads * _causal_pairs(_lengths(tokens, case["median"], 1))
        nbytes = 2.0 * HEAD_DIM * tokens * ((heads + 2 * kv) + heads)
        return {"bytes": nbytes * (2 if case["backward"] else 1), "flops": flops * (3.5 if case["backward"] else 1)}
    if case["kind"] == "step":
        cfg = get_model_config(case["model"]).with_layers(case["layers"])
        h, i = cfg.hidden_size, cfg.intermediate_size
        per_weight = 0.5 + 1.0 / 64 if case["nf4"] else 2.0
        shapes = [(h, cfg.q_size), (h, cfg.kv_size), (h, cfg.kv_size), (cfg.q_size, h), (h, i), (h, i), (i, h)]
        ranks = _ints(case["ranks"])
        # frozen weights once, trained weights and their optimizer state once in and once out
        nbytes = sum(k * n for k, n in shapes) * per_weight * cfg.num_layers + 2.0 * cfg.vocab_size * h
        nbytes += sum(r * (k + n) for r in ranks for k, n in shapes) * cfg.num_layers * 24.0
        flops = 0.0
        for spec in _microbatches(case):
            for a, lens in spec.segments:
                t = sum(lens)
                for k, n in shapes:
                    flops += cfg.num_layers * _linear_work(t, k, n, ranks[a], True, 0.0)[0]
                flops += cfg.num_layers * 3.5 * 4.0 * HEAD_DIM * cfg.num_heads * _causal_pairs(lens)
                flops += 4.0 * t * h * cfg.vocab_size
        return {"bytes": nbytes, "flops": flops}
    e = float(case["n"]) * case["k"]
    return {"bytes": e * (2 + 0.5 + 1.0 / 64 + 2), "flops": 0}


def tolerance(case):
    """About four times what was measured on a B200: against the same path in 64 bits for a linear
    layer (y and dX 1.7e-3, dA and dB 3e-3, largest single error 1.2e-2 of the value or the rms) and
    for attention (2.5e-3, largest 8.5e-2); for a training step against itself with the sums of the
    large products in another order (m 5e-3, v 6e-3, largest 0.13).  NF4 codes are whole numbers;
    a mean summed in another order may move a scale across a rounding boundary."""
    kind = case["kind"]
    if kind == "linear":
        return {"rel": 1e-2, "max": 5e-2}
    if kind == "attention":
        return {"rel": 1e-2, "max": 0.35}
    if kind == "step":
        return {"rel": 2.5e-2, "max": 0.55}
    return {"rel": 1e-4, "max": 3e-2, "differ": 1e-4}


# ---------------------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    """What :func:`run` returns, in plain 64-bit torch: linear layers, attention and the double
    quantisation's scales.  A training step has no such value (a whole model with its optimizer),
    nor have whole codes and what hangs on the choice of one."""
    if case["kind"] == "step":
        return None
    state = prepare(case, seed)
    return {"linear": _exact_linear, "attention": _exact_attention, "nf4": _exact_nf4}[case["kind"]](case, state)


def _keep_mask(rows, cols, p, seed):
    """Philox4x32-7 with key ``seed`` over counters (row, column / 8, 0, 0): sixteen bits an element,
    kept where they reach ``round(p * 65536)``."""
    low = 0xFFFFFFFF
    c = [rows[:, None].expand(-1, cols // 8), torch.arange(cols // 8, device=DEVICE)[None, :].expand(len(rows), -1)]
    c += [torch.zeros_like(c[0]), torch.zeros_like(c[0])]
    k0, k1 = seed & low, seed >> 32 & low
    for _ in range(7):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [p1 >> 32 & low ^ c[1] ^ k0, p1 & low, p0 >> 32 & low ^ c[3] ^ k1, p0 & low]
        k0, k1 = (k0 + 0x9E3779B9) & low, (k1 + 0xBB67AE85) & low
    lanes = torch.stack([c[j // 2] >> 16 * (j % 2) & 0xFFFF for j in range(8)], dim=-1)
    return (lanes >= round(p * 65536)).reshape(len(rows), cols)


def _nf4_values(q):
    """64-bit values of a quantised weight: table value times the scale of its block of 64."""
    table = torch.tensor([-1.0, -0.6961928009986877, -0.5250730514526367, -0.39491748809814453, -0.28444138169288635,
                          -0.18477343022823334, -0.09105003625154495, 0.0, 0.07958029955625534, 0.16093020141124725,
                          0.24611230194568634, 0.33791524171829224, 0.44070982933044434, 0.5626170039176941,
                          0.7229568362236023, 1.0], dtype=torch.float64, device=DEVICE)
    codes = torch.stack([q.packed >> 4, q.packed & 15], dim=-1).reshape(-1, 64)
    nested = q.nested.double().repeat_interleave(256)[:len(codes)]
    scales = q.code256.double()[q.absmax_q.long()] * nested + float(q.offset)
    return (table[codes.long()] * scales[:, None]).reshape(q.shape)


def _exact_linear(case, state):
    seg, ranks, rates = _ints(case["segments"]), _ints(case["ranks"]), _floats(case["dropout"])
    w = _nf4_values(state["w"]) if case["nf4"] else state["w"].double()
    x = state["x"].detach().double()
    y = x @ w.t()
    if state["bias"] is not None:
        y += state["bias"].double()
    back = case["backward"]
    if back:
        dy = state["dy"].double()
        dx, da, db = dy @ w, [], []
    start = 0
    for i, s in enumerate(seg):
        rows = slice(start, start + (s if len(seg) == 1 else (s + TILE - 1) // TILE * TILE))
        start, alpha, p = rows.stop, 32.0 / ranks[i], rates[i]
        a, b = state["a"][i].detach().double(), state["b"][i].detach().double()
        keep = 1.0
        if p > 0:
            keep = _keep_mask(torch.arange(rows.start, rows.stop, device=DEVICE), case["k"], p, state["seed"]) / (1.0 - p)
        dropped = x[rows] * keep
        low = alpha * (dropped @ a.t())
        y[rows] += low @ b.t()
        if back:
            d_low = alpha * (dy[rows] @ b)
            db.append(dy[rows].t() @ low)
            da.append(d_low.t() @ dropped)
            dx[rows] += (d_low @ a) * keep
    return {"y": y, "grads": (dx, *da, *db)} if back else {"y": y}


def _exact_attention(case, state):
    heads, kv, d = case["heads"], case["kv_heads"], HEAD_DIM
    qkv = state["qkv"].detach().double()
    out = torch.empty(len(qkv), heads * d, dtype=torch.float64, device=DEVICE)
    grad = torch.zeros_like(qkv)
    start = 0
    for n in _lengths(case["tokens"], case["median"], 1):
        rows = slice(start, start + n)
        start += n
        above = torch.ones(n, n, dtype=torch.bool, device=DEVICE).triu(1)
        for h in range(heads):
            cols = [slice(c * d, (c + 1) * d) for c in (h, heads + h * kv // heads, heads + kv + h * kv // heads)]
            q, k, v = (qkv[rows, c] for c in cols)
            p = ((q @ k.t()) / math.sqrt(d)).masked_fill_(above, -math.inf).softmax(-1)
            out[rows, cols[0]] = p @ v
            if case["backward"]:
                do = state["d_out"][rows, cols[0]].double()
                grad[rows, cols[2]] += p.t() @ do
                ds = p * (do @ v.t() - (do * out[rows, cols[0]]).sum(-1, keepdim=True)) / math.sqrt(d)
                grad[rows, cols[0]] = ds @ k
                grad[rows, cols[1]] += ds.t() @ q
    return {"out": out, "grads": (grad,)} if case["backward"] else {"out": out}


def _exact_nf4(case, state):
    absmax = state["w"].double().reshape(-1, 64).abs().amax(1)
    off = absmax - absmax.mean()
    nested = torch.nn.functional.pad(off, (0, -len(off) % 256)).reshape(-1, 256).abs().amax(1)
    return {"packed": None, "scales": None, "nested": nested.clamp_min(1e-12), "w": None}
