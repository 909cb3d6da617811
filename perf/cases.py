"""Performance cases: the work this engine is run for, through its public entry points.

Five kinds, each over a range of sizes (`draw`) of which `listed` names the usual points:

  experts   `ops.moe.moe_experts`: the routed NVFP4 experts of one flagship layer, from one token to a prefill chunk
  linear    `ops.functional.linear`: one projection of the flagship, fp8 (128 x 128 blocks) or bf16, one token to a chunk
  attention `ops.attention.sparse_mla`: window rows and selected compressed rows per token, one token to a chunk
  flash     `Engine.open_sequence` / `feed` / `close_sequence`: prompts in chunks of 4096 and steps of one token per sequence
            through a flagship-shaped model (NVFP4 experts, fp8 cache, compressed and window layers)
  hybrid    the same through a layer-by-layer decoder (windowed attention and mLSTM in turns, bf16)

Inputs are random from the seed, with the value ranges of the model: normed activations, gaussian weights, routing with popular
and unpopular experts, distinct selected rows spread over the context.
"""
import math
import random

import torch

from stkernel_b200.config import EngineConfig, SchedulerConfig, YarnScaling, flash_config, hybrid_stack
from stkernel_b200.models.dsv4 import RandomSource, build_model_weights
from stkernel_b200.models.hybrid import build_hybrid_weights
from stkernel_b200.ops import attention as A
from stkernel_b200.ops import functional as Fn
from stkernel_b200.ops import moe as M
from stkernel_b200.ops.cache import PAGE, PagedCache
from stkernel_b200.runtime.engine import Engine

DEV = "cuda"
BF16, F32, F64, FP8 = torch.bfloat16, torch.float32, torch.float64, torch.float8_e4m3fn
HIDDEN, INTER, TOP = 4096, 2048, 6          # flagship: width, rows of an expert, experts per token
LATENT, ROPE, NOPE = 512, 64, 448           # cached latent row: 448 e4m3 values with a scale per 64, 64 bf16 rotated ones
WINDOW = 128
LIMIT = 10.0
CHUNK = 4096                                # tokens of a prefill step



def listed():
    return [
        # one request being decoded: six experts' weights are streamed for one token
        {"name": "experts_1_token", "kind": "experts", "tokens": 1, "experts": 256},
        # a busy decode batch: nearly every expert has a token or two, all weights are streamed
        {"name": "experts_64_tokens", "kind": "experts", "tokens": 64, "experts": 256},
        # a whole prefill chunk: about a hundred tokens per expert
        {"name": "experts_4096_tokens", "kind": "experts", "tokens": 4096, "experts": 256},
        # output projection of one decoded token
        {"name": "linear_fp8_1_token", "kind": "linear", "tokens": 1, "n": 4096, "k": 8192, "fp8": True},
        # query projection of a decode batch
        {"name": "linear_fp8_64_tokens", "kind": "linear", "tokens": 64, "n": 40960, "k": 1536, "fp8": True},
        # a short prompt of odd length in a bf16 model
        {"name": "linear_bf16_777_tokens", "kind": "linear", "tokens": 777, "n": 4096, "k": 4096, "fp8": False},
        # output projection of a prefill chunk
        {"name": "linear_fp8_4096_tokens", "kind": "linear", "tokens": 4096, "n": 4096, "k": 8192, "fp8": True},
        # attention of a decode batch over long contexts
        {"name": "attention_64_tokens", "kind": "attention", "tokens": 64, "heads": 64, "selected": 2048, "context": 32768},
        # attention of a prefill chunk deep in a long prompt
        {"name": "attention_4096_tokens", "kind": "attention", "tokens": 4096, "heads": 64, "selected": 2048, "context": 32768},
        # a long prompt, chunk after chunk
        {"name": "flash_prompt_16384", "kind": "flash", "prompts": 1, "length": 16384, "steps": 0},
        # a batch of short prompts of uneven lengths and the tokens that follow them
        {"name": "flash_32_prompts_8_steps", "kind": "flash", "prompts": 32, "length": 90, "steps": 8},
        # the same in the layer-by-layer decoder: a prompt of a chunk and a half, then a few tokens
        {"name": "hybrid_prompt_6000_4_steps", "kind": "hybrid", "prompts": 1, "length": 6000, "steps": 4},
    ]


def _log(rng: random.Random, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("experts", "linear", "attention", "flash", "hybrid"))
    if kind == "experts":
        return {"kind": kind, "tokens": _log(rng, 1, 4096), "experts": rng.randint(32, 256)}
    if kind == "linear":
        # from a narrow model's projections to the flagship's widest (40960 x 1536) and deepest (4096 x 8192)
        return {"kind": kind, "tokens": _log(rng, 1, 4096), "n": 128 * _log(rng, 8, 320), "k": 128 * _log(rng, 8, 64),
                "fp8": rng.random() < 0.6}
    if kind == "attention":
        return {"kind": kind, "tokens": _log(rng, 1, 4096), "heads": rng.choice((8, 16, 32, 64)),
                "selected": rng.choice((0, 512, 2048)), "context": _log(rng, 512, 32768)}
    if kind == "flash":
        n = rng.choice((1, 1, 2, 5, 16, 32))
        return {"kind": kind, "prompts": n, "length": _log(rng, 16, min(16384, 8192 // n)), "steps": rng.choice((0, 1, 4, 8))}
    n = rng.choice((1, 2, 7, 24))
    return {"kind": kind, "prompts": n, "length": _log(rng, 16, 8192 // n), "steps": rng.choice((0, 1, 4, 8))}


# ---- inputs ---------------------------------------------------------------------------------------------------------
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _lengths(case):
    """Prompt lengths around the case's: uneven, the same for every seed (the work is the case's)."""
    n, mean = case["prompts"], case["length"]
    return [mean] if n == 1 else [max(1, int(mean * (0.5 + (i * 7 % n) / (n - 1)))) for i in range(n)]


def _expert_inputs(case, seed):
    g = _gen(seed)
    t, e = case["tokens"], case["experts"]
    # A gaussian weight in NVFP4 meets every e2m1 code about equally often (a group's largest value is about 1.9 sigma and maps
    # to 6), so uniform nibbles stand for quantised gaussian weights; group scales spread as group maxima do.
    codes = lambda *s: torch.randint(0, 256, s, generator=g, device=DEV, dtype=torch.uint8)
    scales = lambda *s: (200 + 240 * torch.rand(s, generator=g, device=DEV)).to(FP8).view(torch.uint8)
    w = {"w13": codes(e, 2 * INTER, HIDDEN // 2), "s13": scales(e, 2 * INTER, HIDDEN // 16),
         "w2": codes(e, HIDDEN, INTER // 2), "s2": scales(e, HIDDEN, INTER // 16),
         "g13": 2e-5 * (0.9 + 0.2 * torch.rand(e, generator=g, device=DEV)), "g2": 2e-5 * (0.9 + 0.2 * torch.rand(e, generator=g, device=DEV))}
    x = torch.randn(t, HIDDEN, generator=g, device=DEV).to(BF16)
    popular = 0.5 * torch.randn(e, generator=g, device=DEV)
    score = torch.sigmoid(torch.randn(t, e, generator=g, device=DEV) + popular)
    top, ids = score.topk(TOP, 1)
    shared = torch.randn(t, HIDDEN, generator=g, device=DEV).to(BF16)
    return x, ids.to(torch.int32), (top / top.sum(1, keepdim=True)).contiguous(), w, shared


def _linear_inputs(case, seed):
    g = _gen(seed)
    t, n, k = case["tokens"], case["n"], case["k"]
    x = torch.randn(t, k, generator=g, device=DEV).to(BF16)
    w = 0.02 * torch.randn(n, k, generator=g, device=DEV)
    if not case["fp8"]:
        return x, w.to(BF16), None
    blocks = w.view(n // 128, 128, k // 128, 128)
    scale = blocks.abs().amax((1, 3)) / 448.0
    q = (blocks / scale[:, None, :, None]).to(FP8).view(n, k)
    return x, q.contiguous(), scale.contiguous()


def _latent_rows(g, rows: int):
    """Random latent rows as they lie in a cache page: e4m3 codes with a power-of-two scale per 64 values, bf16 rotated part."""
    pages = -(-rows // PAGE)
    v = torch.randn(pages * PAGE, NOPE // 64, 64, generator=g, device=DEV)
    exponent = torch.ceil(torch.log2(v.abs().amax(2) / 448.0))
    codes = (v / torch.exp2(exponent)[:, :, None]).to(FP8).view(torch.uint8).view(pages, PAGE, NOPE)
    rope = torch.randn(pages, PAGE, ROPE, generator=g, device=DEV).to(BF16).view(torch.uint8)
    tail = torch.zeros(pages, PAGE, 8, dtype=torch.uint8, device=DEV)
    tail[:, :, :NOPE // 64] = (exponent + 127).to(torch.uint8).view(pages, PAGE, -1)
    return torch.cat([torch.cat([codes, rope], 2).reshape(pages, -1), tail.reshape(pages, -1)], 1)


def _attention_inputs(case, seed):
    g = _gen(seed)
    t, nh, sel, ctx = case["tokens"], case["heads"], case["selected"], case["context"]
    rows = {"window": _latent_rows(g, max(PAGE, min(t, ctx) + WINDOW))}
    n_window = rows["window"].shape[0] * PAGE
    last = torch.arange(t, device=DEV) % (n_window - WINDOW) + WINDOW - 1
    slots = (last[:, None] - torch.arange(WINDOW, device=DEV)).to(torch.int32)
    lens = torch.full((t,), WINDOW, dtype=torch.int32, device=DEV)
    picked = picked_lens = None
    if sel:
        pool = max(PAGE, ctx // 4)
        rows["selected"] = _latent_rows(g, pool)
        n = min(sel, pool)
        picked = torch.full((t, sel), -1, dtype=torch.int32, device=DEV)
        for a in range(0, t, 512):
            b = min(t, a + 512)
            picked[a:b, :n] = torch.rand(b - a, pool, generator=g, device=DEV).topk(n, 1)[1].to(torch.int32)
        picked_lens = torch.full((t,), n, dtype=torch.int32, device=DEV)
    q = torch.randn(t, nh, LATENT, generator=g, device=DEV).to(BF16)
    sink = torch.randn(nh, generator=g, device=DEV)
    positions = torch.arange(t, device=DEV) % ctx + max(0, ctx - t)
    inv_freq = 10000.0 ** (-torch.arange(0, ROPE, 2, device=DEV, dtype=F32) / ROPE)
    return q, rows, slots, lens, picked, picked_lens, sink, positions, inv_freq


def _cache(pages: torch.Tensor) -> PagedCache:
    c = PagedCache.allocate(pages.shape[0], LATENT, ROPE, True, "latent", DEV)
    c.buf[:, :pages.shape[1]] = pages
    return c


def _flash_config():
    # One compressed and one window layer of the flagship with 64 experts, chosen by token id as its first layers do.  The dense
    # weights are the configuration's bf16 ones: activations rounded to fp8 (cases of their own above) turn a difference in a
    # value's last bit into one of several percent of a whole model's logits, which would hide any error worth finding.
    return flash_config(2, n_routed_experts=64, num_hash_layers=2, dense_dtype="bf16")


class _FlashSource(RandomSource):
    """Random weights whose stream mixes are those of a model that uses all of its streams: read, write and combine weights near
    one another (without this nearly every token's mixes would be saturated at 0 or 1, and a few at the border between)."""

    def get(self, name, shape, device):
        t = super().get(name, shape, device)
        return 0.25 * (t - 0.5) if name.endswith(("hc_attn_fn", "hc_ffn_fn")) else t


def _hybrid_config():
    return hybrid_stack(4, 2048, heads=16, kv_heads=4, dim=128, window=2048, ff=5632, vocab=32768, mlstm_heads=4, mlstm_dim=256,
                        mlstm_vdim=512, yarn=YarnScaling(4.0, 4096, 32.0, 1.0))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "experts":
        x, ids, wts, w, shared = _expert_inputs(case, seed)
        return {"case": case, "x": x, "ids": ids, "wts": wts, "shared": shared,
                "experts": M.ExpertWeights(w["w13"], w["w2"], w["s13"], w["s2"], w["g13"], w["g2"])}
    if kind == "linear":
        x, w, scale = _linear_inputs(case, seed)
        return {"case": case, "x": x, "weight": Fn.LinearWeight(w, scale)}
    if kind == "attention":
        q, rows, slots, lens, picked, picked_lens, sink, positions, inv_freq = _attention_inputs(case, seed)
        return {"case": case, "args": (q, _cache(rows["window"]), slots, lens, _cache(rows["selected"]) if case["selected"] else None,
                                       picked, picked_lens, sink, LATENT ** -0.5, (positions, inv_freq))}
    cfg = _flash_config() if kind == "flash" else _hybrid_config()
    lengths = _lengths(case)
    limit = max(lengths) + case["steps"] + 64
    sched = SchedulerConfig(max_model_len=limit, max_num_seqs=max(2, case["prompts"]), max_num_batched_tokens=CHUNK)
    if kind == "flash":
        weights = build_model_weights(cfg, _FlashSource(seed), DEV)
    else:
        weights = build_hybrid_weights(cfg, RandomSource(seed), DEV)
    engine = Engine(EngineConfig(model=cfg, sched=sched).validate(), weights, torch.device(DEV, torch.cuda.current_device()), max_context=limit)
    g = torch.Generator().manual_seed(int(seed))
    token_lists = [torch.randint(0, cfg.vocab_size, (n + case["steps"],), generator=g).tolist() for n in lengths]
    return {"case": case, "engine": engine, "tokens": token_lists, "lengths": lengths}


# ---- one pass ---------------------------------------------------------------------------------------------------------
def run(state):
    kind = state["case"]["kind"]
    if kind == "experts":
        return M.moe_experts(state["x"], state["ids"], state["wts"], state["experts"], LIMIT, state["shared"], state["experts"].num_local)
    if kind == "linear":
        return Fn.linear(state["x"], state["weight"])
    if kind == "attention":
        q, window, slots, lens, selected, picked, picked_lens, sink, scale, rope = state["args"]
        return A.sparse_mla(q, window, slots, lens, selected, picked, picked_lens, sink, scale, inv_rope=rope)
    # prompts in steps of at most CHUNK tokens with the logits of every 64th and each prompt's last token, then steps of one given
    # token per sequence with the logits of each
    engine, tokens, lengths = state["engine"], state["tokens"], state["lengths"]
    seqs = [engine.open_sequence() for _ in lengths]
    done = [0] * len(seqs)
    logits = []
    while any(d < n for d, n in zip(done, lengths)):
        spans, room = [], CHUNK
        for i, s in enumerate(seqs):
            n = min(room, lengths[i] - done[i])
            if n > 0:
                want = sorted(set(range(63, n, 64)) | {n - 1})
                spans.append((s, tokens[i][done[i]:done[i] + n], want))
                done[i] += n
                room -= n
        logits.append(engine.feed(spans))
    for k in range(state["case"]["steps"]):
        logits.append(engine.feed([(s, [tokens[i][lengths[i] + k]], [0]) for i, s in enumerate(seqs)]))
    for s in seqs:
        engine.close_sequence(s)
    return logits


# ---- what a pass cannot do without ------------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "experts":
        t, e = case["tokens"], case["experts"]
        per = 3 * HIDDEN * INTER
        touched = e * (1.0 - (1.0 - TOP / e) ** t)
        return {"bytes": touched * per * 9 / 16 + 3 * 2 * t * HIDDEN, "flops": 2.0 * t * TOP * per}
    if kind == "linear":
        t, n, k = case["tokens"], case["n"], case["k"]
        return {"bytes": n * k * (1 if case["fp8"] else 2) + 2 * t * (n + k), "flops": 2.0 * t * n * k}
    if kind == "attention":
        t, nh, pool = case["tokens"], case["heads"], max(PAGE, case["context"] // 4)
        n = min(case["selected"], pool)
        rows = WINDOW + n
        # distinct cached rows, their lists, queries and outputs
        distinct = min(t, case["context"]) + WINDOW + (pool * (1.0 - (1.0 - n / pool) ** t) if n else 0)
        return {"bytes": distinct * 584 + 4 * t * rows + 4 * t * nh * LATENT, "flops": 4.0 * t * rows * nh * LATENT}
    tokens = sum(_lengths(case)) + case["prompts"] * case["steps"]
    feeds = -(-sum(_lengths(case)) // CHUNK) + case["steps"]
    wanted = sum(n // 64 + 1 for n in _lengths(case)) + case["prompts"] * case["steps"]
    per_step = tokens / feeds
    mean = case["length"]
    if kind == "flash":
        cfg = _flash_config()
        qkv = HIDDEN * (1536 + LATENT) + 1536 * 64 * LATENT + 8 * 1024 * HIDDEN + HIDDEN * 8192
        dense = 2 * (qkv + 3 * HIDDEN * INTER + 64 * HIDDEN) + 1536 * 64 * 128
        sides = HIDDEN * (4 * LATENT + 64 + 4 * 128) + 2 * 2 * 24 * 4 * HIDDEN
        expert = 3 * HIDDEN * INTER
        touched = 2 * 64 * (1.0 - (1.0 - TOP / 64) ** per_step)
        head = cfg.vocab_size * HIDDEN
        flops = 2.0 * tokens * (dense + sides + 2 * TOP * expert) + 2.0 * wanted * head
        rows = 2 * min(WINDOW, mean) + min(2048, mean / 8)
        flops += tokens * (4.0 * rows * 64 * LATENT + 2.0 * 64 * 128 * mean / 8)
        size = 2 * (dense + sides + head) + touched * expert * 9 / 16
        return {"bytes": feeds * size + tokens * 2 * 2 * 4 * HIDDEN * 4 + wanted * 4 * cfg.vocab_size, "flops": flops}
    cfg = _hybrid_config()
    width, ff = 2048, 5632
    rec = width * (4 * (256 * 2 + 512) + 2 * 4 + 4 * 512) + 4 * 512 * width
    att = width * (16 * 128 + 4 * 128) + 16 * 128 * width
    dense = 2 * (rec + att) + 4 * 3 * width * ff
    head = cfg.vocab_size * width
    flops = 2.0 * tokens * dense + 2.0 * wanted * head + 2 * tokens * (4.0 * min(2048, mean / 2) * 16 * 128 + 4.0 * 4 * 256 * 512)
    return {"bytes": feeds * 2 * (dense + head) + tokens * 4 * 2 * 4 * width + wanted * 4 * cfg.vocab_size, "flops": flops}


def tolerance(case):
    # Four times what two correct paths differ by.  One product: results are rounded to bf16 (2^-9 relative at most, 0.0017 in the
    # 2-norm), intermediates of the experts to 16 bits once more.  fp8 projections round the activation to e4m3 first; a value at
    # the border of two codes may go either way in another order of the same arithmetic.  Whole models carry those roundings
    # through every layer of the residual stream, and the fp8 cache rows of the flagship amplify them.
    if case["kind"] in ("flash", "hybrid"):
        return {"rel": 0.03, "max": 0.5}
    return {"rel": 0.01, "max": 0.1}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------
_E2M1 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0, -0.0, -0.5, -1.0, -1.5, -2.0, -3.0, -4.0, -6.0)


def _nvfp4(codes, scales, global_scale):
    table = torch.tensor(_E2M1, dtype=F64, device=DEV)
    v = torch.stack([table[(codes & 15).long()], table[(codes >> 4).long()]], -1).view(codes.shape[0], -1, 16)
    return (v * scales.view(FP8).to(F64)[:, :, None]).view(codes.shape[0], -1) * global_scale.to(F64)


def _exact_experts(case, seed):
    x, ids, wts, w, shared = _expert_inputs(case, seed)
    x64, out = x.to(F64), shared.to(F64)
    for e in range(case["experts"]):
        tok, place = (ids == e).nonzero(as_tuple=True)
        if tok.numel() == 0:
            continue
        h = x64[tok] @ _nvfp4(w["w13"][e], w["s13"][e], w["g13"][e]).t()
        gate, up = h[:, :INTER].clamp(max=LIMIT), h[:, INTER:].clamp(-LIMIT, LIMIT)
        y = (gate * torch.sigmoid(gate) * up) @ _nvfp4(w["w2"][e], w["s2"][e], w["g2"][e]).t()
        out.index_add_(0, tok, y * wts[tok, place].to(F64)[:, None])
    return out


def _exact_linear(case, seed):
    x, w, scale = _linear_inputs(case, seed)
    a, b = x.to(F64), w.to(F64)
    if scale is not None:
        n, k = w.shape
        b = (b.view(n // 128, 128, k // 128, 128) * scale.to(F64)[:, None, :, None]).view(n, k)
        if case["tokens"] > 8:
            # larger batches quantise the activation: one scale per token and 128 values, e4m3 codes
            v = x.float().view(-1, k // 128, 128)
            s = (v.abs().amax(2) / 448.0).clamp(min=1e-10)
            a = ((v / s[:, :, None]).to(FP8).to(F64) * s.to(F64)[:, :, None]).view(-1, k)
    return a @ b.t()


def _unpack(pages):
    n = pages.shape[0]
    data = pages[:, :PAGE * 576].reshape(n * PAGE, 576)
    tail = pages[:, PAGE * 576:PAGE * 584].reshape(n * PAGE, 8)
    nope = data[:, :NOPE].contiguous().view(FP8).to(F64).view(-1, NOPE // 64, 64) * torch.exp2(tail[:, :NOPE // 64].to(F64) - 127)[:, :, None]
    return torch.cat([nope.view(-1, NOPE), data[:, NOPE:].contiguous().view(BF16).to(F64)], 1)


def _exact_attention(case, seed):
    q, rows, slots, lens, picked, picked_lens, sink, positions, inv_freq = _attention_inputs(case, seed)
    window = _unpack(rows["window"])
    chosen = _unpack(rows["selected"]) if case["selected"] else None
    n = int(picked_lens[0]) if picked is not None else 0
    out = torch.empty(q.shape, dtype=F64, device=DEV)
    for a in range(0, q.shape[0], 64):
        b = min(q.shape[0], a + 64)
        kv = window[slots[a:b].long()]
        if n:
            kv = torch.cat([kv, chosen[picked[a:b, :n].long()]], 1)
        s = q[a:b].to(F64) @ kv.transpose(1, 2) * LATENT ** -0.5
        p = torch.softmax(torch.cat([s, sink.to(F64)[None, :, None].expand(b - a, -1, 1)], 2), 2)[:, :, :-1]
        out[a:b] = p @ kv
    angle = positions.to(F64)[:, None] * inv_freq.to(F64)[None]
    cos, sin = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
    even, odd = out[..., NOPE::2].clone(), out[..., NOPE + 1::2].clone()
    out[..., NOPE::2] = even * cos + odd * sin
    out[..., NOPE + 1::2] = odd * cos - even * sin
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "experts":
        return _exact_experts(case, seed)
    if kind == "linear":
        return _exact_linear(case, seed)
    if kind == "attention":
        return _exact_attention(case, seed)
    return None     # whole models: token by token in 64 bits (recurrences, caches, per-token selections) takes minutes
