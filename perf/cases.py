"""The work this framework is measured on: what one GPU does while it serves.

Nine kinds of case, each through the entry points that the serving engine itself calls:

* ``decode``   a decode step of a Llama-3-8B slice (two of its layers, embedding, LM head), replayed from a CUDA graph as ``ModelRunner`` does:
  embedding gather, norms, QKV / output / MLP projections, rotary + paged KV write, paged attention over ragged contexts, logits.
* ``prefill``  an extend step of the same slice over ragged prompts, some of which continue a cached prefix; logits of the last rows.
* ``chunk``    paged attention of one long prompt's chunk against its cached context (chunked prefill).
* ``context``  paged attention of a decode batch over long, uneven contexts (split-KV).
* ``moe``      a mixture-of-experts block: routing and the routed expert MLPs (Mixtral-8x7B and Qwen3-30B-A3B sizes).
* ``fp8``      a block-scaled fp8 gated MLP (activation quantiser, two block-scaled products, SiLU * mul).
* ``sample``   sampling a batch whose rows ask for different settings (greedy, top-k, top-p, min-p, plain), with log-probabilities.
* ``scan``     the Mamba-2 recurrence over ragged prompt portions or single decode tokens.

``listed()`` has the twelve that stand for them, ``draw()`` gives more of the same ranges.  Lengths of a batch follow from the case's own numbers
(log-normal, as chat traffic is), values from the seed.
"""
from __future__ import annotations

import math
import random
from types import SimpleNamespace

import torch

import sglang_b200  # noqa: F401
from sglang_b200 import ops
from sglang_b200.configs.model_config import load_model_config
from sglang_b200.managers.schedule_batch import ForwardMode
from sglang_b200.mem_cache.memory_pool import KVPool
from sglang_b200.model_executor.forward_batch import ForwardBatch
from sglang_b200.model_loader.loader import build_model
from sglang_b200.ops import moe_ops, quant_ops

ops.load_native()                           # (what the model runner does first)

DEV = "cuda"
PAGE = 32                                   # the benchmark's page size
HEADS, KV_HEADS, HEAD = 32, 8, 128          # Llama-3-8B attention
HIDDEN, INTER, VOCAB, LAYERS = 4096, 14336, 128256, 2
EPS, THETA = 1e-5, 500000.0
#: expert blocks by name: experts, chosen per token, width, expert width
MOE = {"mixtral-8x7b": (8, 2, 4096, 14336), "qwen3-30b-a3b": (128, 8, 2048, 768)}
#: fp8 MLPs: width, inner width (Llama-3-8B whole; one rank of Llama-3-70B at TP = 8)
FP8 = {"llama-3-8b": (4096, 14336), "llama-3-70b-tp8": (8192, 3584)}
#: Mamba-2 mixers: heads, head width, state width, groups
SCAN = {"h64": (64, 64, 128, 8), "h16": (16, 128, 128, 16)}


def listed():
    return [
        # one user, one token: latency, launches, weights read once
        {"name": "decode_single", "kind": "decode", "batch": 1, "mean": 611, "shape": 1},
        # a busy server's decode step at chat lengths
        {"name": "decode_batch", "kind": "decode", "batch": 128, "mean": 600, "shape": 2},
        # one scheduler step of ragged prompts (odd total), a few with a cached prefix
        {"name": "prefill_prompts", "kind": "prefill", "tokens": 5003, "batch": 17, "shape": 3},
        # the last chunk of a long document
        {"name": "chunk_long", "kind": "chunk", "tokens": 4096, "context": 15011},
        # a handful of long conversations
        {"name": "context_long", "kind": "context", "batch": 6, "mean": 24000, "shape": 4},
        # expert block: a small decode batch, a prompt chunk, and fine-grained experts at a larger decode batch
        {"name": "moe_decode", "kind": "moe", "model": "mixtral-8x7b", "tokens": 20},
        {"name": "moe_prompt", "kind": "moe", "model": "mixtral-8x7b", "tokens": 4001},
        {"name": "moe_fine", "kind": "moe", "model": "qwen3-30b-a3b", "tokens": 333},
        # block-scaled fp8 MLP: decode batch and prompt chunk
        {"name": "fp8_decode", "kind": "fp8", "model": "llama-3-70b-tp8", "tokens": 9},
        {"name": "fp8_prompt", "kind": "fp8", "model": "llama-3-8b", "tokens": 3001},
        # a decode batch's sampler over the full vocabulary
        {"name": "sample_batch", "kind": "sample", "batch": 121, "vocab": 128256},
        # hybrid models' recurrence over prompts
        {"name": "scan_prompts", "kind": "scan", "model": "h64", "tokens": 3001, "batch": 5, "shape": 5},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["decode", "decode", "prefill", "chunk", "context", "moe", "moe", "moe", "fp8", "fp8", "sample", "scan"])
    shape = rng.randrange(1, 1000)
    if kind == "decode":
        return {"kind": kind, "batch": log(1, 192), "mean": log(64, 900), "shape": shape}
    if kind == "prefill":
        tokens = log(64, 5000)
        return {"kind": kind, "tokens": tokens, "batch": rng.randint(1, max(1, min(24, tokens // 16))), "shape": shape}
    if kind == "chunk":
        tokens = log(64, 4096)
        return {"kind": kind, "tokens": tokens, "context": rng.randint(tokens, 15000)}
    if kind == "context":
        mean = log(2000, 40000)
        return {"kind": kind, "batch": rng.randint(1, max(1, min(32, 140000 // mean))), "mean": mean, "shape": shape}
    if kind == "moe":
        return {"kind": kind, "model": rng.choice(sorted(MOE)), "tokens": log(1, 4000)}
    if kind == "fp8":
        return {"kind": kind, "model": rng.choice(sorted(FP8)), "tokens": log(1, 3000)}
    if kind == "sample":
        return {"kind": kind, "batch": log(1, 256), "vocab": rng.choice([32000, 128256, 151936])}
    batch = rng.randint(1, 12)
    return {"kind": kind, "model": rng.choice(sorted(SCAN)), "tokens": max(batch, log(8, 3000)), "batch": batch, "shape": shape}


# ------------------------------------------------------------------ sizes that follow from a case
def _spread(n, total, seed, sigma):
    """n positive lengths that sum to ``total``, log-normally uneven"""
    r = random.Random(seed * 7919 + n)
    raw = [math.exp(r.gauss(0.0, sigma)) for _ in range(n)]
    left = total - n
    cut = [int(left * x / sum(raw)) for x in raw]
    cut[0] += left - sum(cut)
    return [1 + c for c in cut]


def _lengths(case):
    """(tokens fed, tokens cached before them) of every request"""
    k = case["kind"]
    if k == "decode":
        return [1] * case["batch"], [max(1, x - 1) for x in _spread(case["batch"], case["batch"] * case["mean"], case["shape"], 0.7)]
    if k == "prefill":
        q = _spread(case["batch"], case["tokens"], case["shape"], 0.8)
        return q, [(37 * i) % 512 if i % 3 == 2 else 0 for i in range(len(q))]
    if k == "chunk":
        return [case["tokens"]], [case["context"] - case["tokens"]]
    if k == "context":
        return [1] * case["batch"], [max(1, x - 1) for x in _spread(case["batch"], case["batch"] * case["mean"], case["shape"], 0.6)]
    if k == "scan":
        q = _spread(case["batch"], case["tokens"], case["shape"], 0.8)
        return q, [0 if i % 2 == 0 else 100 for i in range(len(q))]
    raise KeyError(k)


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _randn(g, *shape, std=1.0, dtype=torch.bfloat16):
    return torch.randn(*shape, generator=g, device=DEV, dtype=dtype).mul_(std)


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


# ------------------------------------------------------------------ inputs, from the seed alone (shared by prepare and exact)
def _paged(case, g, layers):
    """KV pages of every request, in random order, filled with earlier tokens' keys and values"""
    q, past = _lengths(case)
    need = [(a + b + PAGE - 1) // PAGE for a, b in zip(q, past)]
    pages = sum(need) + 1                                             # page 0 stays unused, as in the engine
    order = (torch.randperm(pages - 1, generator=g, device=DEV) + 1).to(torch.int32)
    table = torch.zeros(len(q) + 1, max(need), dtype=torch.int32, device=DEV)
    off = 0
    for i, n in enumerate(need):
        table[i + 1, :n] = order[off:off + n]
        off += n
    kv = torch.randn(layers, 2, pages * PAGE, KV_HEADS, HEAD, generator=g, device=DEV, dtype=torch.bfloat16)
    return q, past, table, kv


def _slots(table, row, first, last):
    p = torch.arange(first, last, device=DEV)
    return table[row + 1].long()[p // PAGE] * PAGE + p % PAGE


def _slice_weights(g):
    w = {"model.embed_tokens.weight": _randn(g, VOCAB, HIDDEN), "lm_head.weight": _randn(g, VOCAB, HIDDEN, std=HIDDEN ** -0.5),
         "model.norm.weight": 1 + _randn(g, HIDDEN, std=0.1)}
    for i in range(LAYERS):
        p = f"model.layers.{i}."
        w[p + "self_attn.qkv_proj.weight"] = _randn(g, (HEADS + 2 * KV_HEADS) * HEAD, HIDDEN, std=HIDDEN ** -0.5)
        w[p + "self_attn.o_proj.weight"] = _randn(g, HIDDEN, HEADS * HEAD, std=HIDDEN ** -0.5)
        w[p + "mlp.gate_up_proj.weight"] = _randn(g, 2 * INTER, HIDDEN, std=HIDDEN ** -0.5)
        w[p + "mlp.down_proj.weight"] = _randn(g, HIDDEN, INTER, std=INTER ** -0.5)
        w[p + "input_layernorm.weight"] = 1 + _randn(g, HIDDEN, std=0.1)
        w[p + "post_attention_layernorm.weight"] = 1 + _randn(g, HIDDEN, std=0.1)
    return w


def _slice_inputs(case, seed):
    g = _gen(seed)
    q, past, table, kv = _paged(case, g, LAYERS)
    ids = torch.randint(0, VOCAB, (sum(q),), generator=g, device=DEV, dtype=torch.int32)
    return g, q, past, table, kv, ids


def _moe_inputs(case, seed):
    E, K, H, I = MOE[case["model"]]
    g = _gen(seed)
    x = _randn(g, case["tokens"], H)
    # routers prefer some experts: a common bias beside what the token itself asks for
    logits = _randn(g, case["tokens"], E, dtype=torch.float32) + _randn(g, 1, E, std=0.7, dtype=torch.float32)
    return x, logits.to(torch.bfloat16), _randn(g, E, 2 * I, H, std=H ** -0.5), _randn(g, E, H, I, std=I ** -0.5)


def _fp8_weight(g, n, k):
    """e4m3 weights with one scale per 128 x 128 block, as such checkpoints hold them"""
    w = torch.randn(n, k, generator=g, device=DEV).mul_(k ** -0.5)
    b = w.view(n // 128, 128, k // 128, 128)
    s = b.abs().amax(dim=(1, 3)).clamp(min=1e-10) / 448.0
    return (b / s[:, None, :, None]).clamp(-448, 448).to(torch.float8_e4m3fn).view(n, k), s


def _fp8_inputs(case, seed):
    H, I = FP8[case["model"]]
    g = _gen(seed)
    # activations with the uneven channels that make block scales worth having
    x = _randn(g, case["tokens"], H) * torch.exp(0.5 * _randn(g, 1, H))
    return x, _fp8_weight(g, 2 * I, H), _fp8_weight(g, H, I)


def _scan_inputs(case, seed):
    H, P, N, G = SCAN[case["model"]]
    g = _gen(seed)
    q, past = _lengths(case)
    T, n = sum(q), len(q)
    u = torch.nn.functional.silu(_randn(g, T, H * P + 2 * G * N, dtype=torch.float32))
    z = _randn(g, T, H * P)
    dt = _randn(g, T, H)
    dt_bias = torch.log(torch.expm1(torch.empty(H, device=DEV).uniform_(0.001, 0.1, generator=g)))
    A_log = torch.log(torch.empty(H, device=DEV).uniform_(1.0, 16.0, generator=g))
    D = 1 + _randn(g, H, std=0.1, dtype=torch.float32)
    state = _randn(g, n + 1, H, N, P, dtype=torch.float32)
    return u, z, dt, dt_bias, A_log, D, state


# ------------------------------------------------------------------ prepare
def _splits(batch, longest):
    """KV splits of a decode batch, as the engine's runner picks them for its attention launches"""
    ctas, tiles, sms = batch * KV_HEADS, (longest + 127) // 128, torch.cuda.get_device_properties(0).multi_processor_count
    return 1 if ctas >= sms or tiles <= 2 else int(max(1, min(tiles, 8, (sms * 2) // max(1, ctas))))


def _workspace(splits, tokens):
    if splits == 1:
        return None
    return (torch.empty(splits, tokens, HEADS, HEAD, dtype=torch.float32, device=DEV), torch.empty(splits, tokens, HEADS, dtype=torch.float32, device=DEV))


def _prepare_slice(case, seed):
    g, q, past, table, kv, ids = _slice_inputs(case, seed)
    cfg = load_model_config("dummy:llama-3-8b", {"num_hidden_layers": LAYERS})
    model = build_model(cfg, torch.device(DEV))
    params = dict(model.named_parameters())
    for name, t in _slice_weights(g).items():
        params.pop(name).data = t
    assert not params, sorted(params)
    pool = KVPool(1, PAGE, 1, KV_HEADS, HEAD, torch.bfloat16, DEV)
    pool.num_pages, pool.num_layers, pool.num_slots, pool.buf = kv.shape[2] // PAGE, LAYERS, kv.shape[2], kv
    n, decode = len(q), case["kind"] == "decode"
    longest = max(a + b for a, b in zip(q, past))
    positions = torch.cat([torch.arange(b, a + b, device=DEV) for a, b in zip(q, past)]).to(torch.int32)
    loc = torch.cat([_slots(table, i, b, a + b) for i, (a, b) in enumerate(zip(q, past))]).to(torch.int32)
    rows = _i32(list(range(1, n + 1)))
    fb = ForwardBatch(mode=ForwardMode.DECODE if decode else ForwardMode.EXTEND, batch_size=n, num_tokens=sum(q), input_ids=None if decode else ids,
                      positions=positions, out_cache_loc=loc, req_slots=rows, seq_lens=_i32([a + b for a, b in zip(q, past)]), cu_q=None, q_lens=None,
                      last_idx=None, sample_slots=rows, page_table=table, page_size=PAGE, kv_pool=pool, max_kv_len=longest)
    if decode:
        fb.next_token_buf = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
        fb.next_token_buf[1:] = ids
        fb.num_splits = _splits(n, 4096)                      # graphs are captured for the longest context the bucket may see
        fb.attn_workspace = _workspace(fb.num_splits, n)
    else:
        cu = [0]
        for a in q:
            cu.append(cu[-1] + a)
        fb.cu_q, fb.q_lens, fb.max_q_len, fb.last_idx = _i32(cu), _i32(q), max(q), _i32([c - 1 for c in cu[1:]])
    s = SimpleNamespace(kind=case["kind"], model=model, fb=fb)
    if decode:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _slice_forward(s)
            s.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s.graph, stream=side):
                s.logits = _slice_forward(s)
        torch.cuda.current_stream().wait_stream(side)
    return s


def _slice_forward(s):
    h = s.model(s.fb)
    return s.model.compute_logits(h if s.fb.last_idx is None else ops.gather_rows(h, s.fb.last_idx))


def prepare(case, seed):
    k = case["kind"]
    if k in ("decode", "prefill"):
        return _prepare_slice(case, seed)
    if k in ("chunk", "context"):
        g = _gen(seed)
        q, past, table, kv = _paged(case, g, 1)
        lens = [a + b for a, b in zip(q, past)]
        s = SimpleNamespace(kind=k, q=_randn(g, sum(q), HEADS, HEAD), k=kv[0, 0], v=kv[0, 1], table=table, rows=_i32(list(range(1, len(q) + 1))),
                            lens=_i32(lens), cu=None, ql=None, most=max(q), splits=1, work=None)
        if k == "chunk":
            s.cu, s.ql = _i32([0, q[0]]), _i32(q)
        else:
            s.splits = _splits(len(q), max(lens))
            s.work = _workspace(s.splits, len(q))
        return s
    if k == "moe":
        x, logits, w13, w2 = _moe_inputs(case, seed)
        return SimpleNamespace(kind=k, x=x, logits=logits, w13=w13, w2=w2, top=MOE[case["model"]][1])
    if k == "fp8":
        x, up, down = _fp8_inputs(case, seed)
        return SimpleNamespace(kind=k, x=x, up=up, down=down)
    if k == "sample":
        g = _gen(seed)
        B, V = case["batch"], case["vocab"]
        # next-token logits: a few candidates far above a broad tail
        logits = _randn(g, B, V, std=1.5, dtype=torch.float32)
        best = torch.randint(0, V, (B, 60), generator=g, device=DEV)
        logits.scatter_add_(1, best, 14.0 + 2.0 * _randn(g, B, 60, dtype=torch.float32))
        # settings in turn: greedy, nucleus, top-k within a nucleus, min-p, plain
        i = torch.arange(B, device=DEV) % 5
        pick = lambda *v: torch.tensor(v, device=DEV)[i]  # noqa: E731
        return SimpleNamespace(kind=k, logits=logits.to(torch.bfloat16), temperature=pick(1.0, 0.7, 0.8, 1.0, 1.0),
                               top_k=pick(1, 1 << 30, 50, 1 << 30, 1 << 30).to(torch.int32), top_p=pick(1.0, 0.9, 0.95, 1.0, 1.0),
                               min_p=pick(0.0, 0.0, 0.0, 0.05, 0.0), seed=seed, slots=torch.arange(1, B + 1, device=DEV, dtype=torch.int32),
                               next=torch.zeros(B + 1, dtype=torch.int32, device=DEV), lp=torch.empty(B, device=DEV))
    if k == "scan":
        q, past = _lengths(case)
        u, z, dt, dt_bias, A_log, D, state = _scan_inputs(case, seed)
        cu = [0]
        for a in q:
            cu.append(cu[-1] + a)
        return SimpleNamespace(kind=k, u=u, z=z, dt=dt, dt_bias=dt_bias, A_log=A_log, D=D, state=state, rows=_i32(list(range(1, len(q) + 1))),
                               lens=_i32([a + b for a, b in zip(q, past)]), cu=_i32(cu), ql=_i32(q), dims=SCAN[case["model"]])
    raise KeyError(k)


# ------------------------------------------------------------------ run
def run(s):
    if s.kind == "decode":
        s.graph.replay()
        return s.logits
    if s.kind == "prefill":
        return _slice_forward(s)
    if s.kind in ("chunk", "context"):
        return ops.paged_attention(s.q, s.k, s.v, s.table, s.rows, s.lens, s.cu, s.ql, s.most, PAGE, HEAD ** -0.5, num_splits=s.splits, workspace=s.work)
    if s.kind == "moe":
        w, ids = moe_ops.topk_softmax(s.logits, s.top, True)
        return moe_ops.fused_moe(s.x, s.w13, s.w2, w, ids)
    if s.kind == "fp8":
        h = ops.silu_and_mul(quant_ops.fp8_block_linear(s.x, *s.up))
        return quant_ops.fp8_block_linear(h, *s.down)
    if s.kind == "sample":
        tokens = ops.sample(s.logits, s.temperature, s.top_k, s.top_p, s.min_p, out_slots=s.slots, next_token_buf=s.next, out_logprobs=s.lp,
                            global_seed=s.seed, step=7)
        return {"tokens": tokens, "logprobs": s.lp, "next": s.next}
    H, P, N, G = s.dims
    y = ops.mamba2_scan(s.u, s.z, s.dt, s.dt_bias, s.A_log, s.D, s.state, s.rows, s.lens, s.cu, s.ql, H, P, N, G)
    return {"y": y, "state": s.state}


# ------------------------------------------------------------------ what a pass cannot do without
def _attended(q, past):
    """(query, key) pairs a causal mask leaves"""
    return sum(a * b + a * (a + 1) // 2 for a, b in zip(q, past))


def work(case):
    k = case["kind"]
    row = KV_HEADS * HEAD * 2                                                   # bytes of one token's keys (or values) in a layer
    if k in ("decode", "prefill"):
        q, past = _lengths(case)
        T, n = sum(q), len(q)
        per = (HEADS + 2 * KV_HEADS) * HEAD * HIDDEN + HIDDEN * HEADS * HEAD + 3 * INTER * HIDDEN
        weights = 2 * (LAYERS * (per + 2 * HIDDEN) + HIDDEN + VOCAB * HIDDEN)
        kv = 2 * row * LAYERS * (sum(past) + T)
        flops = 2 * T * LAYERS * per + 2 * n * VOCAB * HIDDEN + 4 * HEADS * HEAD * LAYERS * _attended(q, past)
        return {"bytes": weights + kv + 2 * T * HIDDEN + 2 * n * VOCAB, "flops": flops}
    if k in ("chunk", "context"):
        q, past = _lengths(case)
        T = sum(q)
        return {"bytes": 2 * row * (sum(past) + T) + 4 * T * HEADS * HEAD, "flops": 4 * HEADS * HEAD * _attended(q, past)}
    if k == "moe":
        E, K, H, I = MOE[case["model"]]
        T = case["tokens"]
        hit = E * (1 - (1 - K / E) ** T)                                         # experts that any token chose, if all were alike
        return {"bytes": hit * 3 * H * I * 2 + 4 * T * H + 2 * T * E, "flops": 6 * T * K * H * I}
    if k == "fp8":
        H, I = FP8[case["model"]]
        T = case["tokens"]
        return {"bytes": 3 * H * I + 4 * T * H, "flops": 6 * T * H * I}
    if k == "sample":
        return {"bytes": 2 * case["batch"] * case["vocab"] + 24 * case["batch"], "flops": 0}
    H, P, N, G = SCAN[case["model"]]
    T, n = case["tokens"], case["batch"]
    old = sum(1 for b in _lengths(case)[1] if b)
    return {"bytes": T * (4 * (2 * H * P + 2 * G * N) + 2 * H * P + 2 * H) + 4 * (n + old) * H * N * P, "flops": 6 * T * H * N * P}


def tolerance(case):
    # measured against exact(): bf16 model slices 0.006 (a value of 4e8 is up to 0.06 rms off), bf16 attention 0.0027, experts 0.0035,
    # fp8 MLP 0.004 (values that round to another e4m3 step), fp32 scan 4e-7
    return {"decode": {"rel": 0.024, "max": 0.3}, "prefill": {"rel": 0.024, "max": 0.3}, "chunk": {"rel": 0.012, "max": 0.3}, "context": {"rel": 0.012, "max": 0.3},
            "moe": {"rel": 0.015, "max": 0.3}, "fp8": {"rel": 0.02, "max": 0.4}, "sample": {"rel": 1e-4, "max": 1e-3, "differ": 0.01},
            "scan": {"rel": 1e-5, "max": 1e-3}}[case["kind"]]


# ------------------------------------------------------------------ the same in 64 bits, plain torch
def _rope_table(positions):
    f = THETA ** (-torch.arange(0, HEAD, 2, device=DEV, dtype=torch.float64) / HEAD)
    a = torch.arange(positions, device=DEV, dtype=torch.float64)[:, None] * f[None]
    return torch.cat([a.cos(), a.sin()], dim=-1)


def _rotate(x, table):
    c, s = (t[:, None, :] for t in table.chunk(2, dim=-1))
    a, b = x.chunk(2, dim=-1)
    return torch.cat([a * c - b * s, b * c + a * s], dim=-1)


def _attend(q, k, v, past):
    """q [n, heads, d] at positions past.., k / v [past + n, kv heads, d]"""
    n, out = q.shape[0], torch.empty_like(q)
    seen = torch.arange(k.shape[0], device=DEV)[None] <= past + torch.arange(n, device=DEV)[:, None]
    for h in range(HEADS):
        g = h * KV_HEADS // HEADS
        for a in range(0, n, 1024):
            p = (q[a:a + 1024, h] @ k[:, g].T * HEAD ** -0.5).masked_fill_(~seen[a:a + 1024], -math.inf).softmax(-1)
            out[a:a + 1024, h] = p @ v[:, g]
    return out


def _norm(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w.double()


def _exact_slice(case, seed):
    g, q, past, table, kv, ids = _slice_inputs(case, seed)
    w = _slice_weights(g)
    rope = _rope_table(max(a + b for a, b in zip(q, past)))
    pos = torch.cat([torch.arange(b, a + b, device=DEV) for a, b in zip(q, past)])
    mul = lambda x, name: x @ w[name].double().T  # noqa: E731
    h = w["model.embed_tokens.weight"][ids.long()].double()
    for i in range(LAYERS):
        p = f"model.layers.{i}."
        y = mul(_norm(h, w[p + "input_layernorm.weight"]), p + "self_attn.qkv_proj.weight").view(-1, HEADS + 2 * KV_HEADS, HEAD)
        qq, kk, vv = y.split([HEADS, KV_HEADS, KV_HEADS], dim=1)
        qq, kk, o, off = _rotate(qq, rope[pos]), _rotate(kk, rope[pos]), [], 0
        for r, (a, b) in enumerate(zip(q, past)):
            old = _slots(table, r, 0, b)
            o.append(_attend(qq[off:off + a], torch.cat([kv[i, 0][old].double(), kk[off:off + a]]), torch.cat([kv[i, 1][old].double(), vv[off:off + a]]), b))
            off += a
        h = h + mul(torch.cat(o).view(-1, HEADS * HEAD), p + "self_attn.o_proj.weight")
        gate, up = mul(_norm(h, w[p + "post_attention_layernorm.weight"]), p + "mlp.gate_up_proj.weight").chunk(2, dim=-1)
        h = h + mul(torch.nn.functional.silu(gate) * up, p + "mlp.down_proj.weight")
    last = torch.tensor(q, device=DEV).cumsum(0) - 1
    return mul(_norm(h[last], w["model.norm.weight"]), "lm_head.weight")


def _fp8_product(x, weight):
    """x quantised in groups of 128 (what the path is defined to do), the products and sums in 64 bits"""
    q, s = weight
    n, k = q.shape
    g = x.double().view(-1, k // 128, 128)
    xs = (g.abs().amax(-1, keepdim=True).clamp(min=1e-10) / 448.0).float().double()
    xq = (g / xs).to(torch.float8_e4m3fn).double() * xs
    w = q.double().view(n // 128, 128, k // 128, 128) * s.double()[:, None, :, None]
    return xq.view(-1, k) @ w.view(n, k).T


def exact(case, seed):
    k = case["kind"]
    if k in ("decode", "prefill"):
        return _exact_slice(case, seed)
    if k in ("chunk", "context"):
        g = _gen(seed)
        q, past, table, kv = _paged(case, g, 1)
        x, o, off = _randn(g, sum(q), HEADS, HEAD).double(), [], 0
        for r, (a, b) in enumerate(zip(q, past)):
            at = _slots(table, r, 0, a + b)
            o.append(_attend(x[off:off + a], kv[0, 0][at].double(), kv[0, 1][at].double(), b))
            off += a
        return torch.cat(o)
    if k == "moe":
        E, K, H, I = MOE[case["model"]]
        x, logits, w13, w2 = _moe_inputs(case, seed)
        x, p = x.double(), logits.double().softmax(-1)
        # equal scores: the lower expert first
        ids = (p + torch.arange(E, 0, -1, device=DEV, dtype=torch.float64) * 1e-12).topk(K, dim=-1).indices
        wt = p.gather(1, ids)
        wt, out = wt / wt.sum(-1, keepdim=True), torch.zeros_like(x)
        for e in range(E):
            t, j = (ids == e).nonzero(as_tuple=True)
            if t.numel():
                gate, up = (x[t] @ w13[e].double().T).chunk(2, dim=-1)
                out.index_add_(0, t, (torch.nn.functional.silu(gate) * up) @ w2[e].double().T * wt[t, j][:, None])
        return out
    if k == "fp8":
        x, up, down = _fp8_inputs(case, seed)
        gate, u = _fp8_product(x, up).to(torch.bfloat16).double().chunk(2, dim=-1)          # the path hands bf16 from product to product
        return _fp8_product((torch.nn.functional.silu(gate) * u).to(torch.bfloat16), down)
    if k == "sample":
        return None                                  # which token is drawn follows from the sampler's own generator
    H, P, N, G = SCAN[case["model"]]
    q, past = _lengths(case)
    u, z, dt, dt_bias, A_log, D, state = (t.double() for t in _scan_inputs(case, seed))
    dt = torch.log1p(torch.exp(dt + dt_bias))
    x, b, c = u.split([H * P, G * N, G * N], dim=-1)
    x, b, c = x.view(-1, H, P), b.view(-1, G, N).repeat_interleave(H // G, 1), c.view(-1, G, N).repeat_interleave(H // G, 1)
    decay, y, off = torch.exp(-A_log.exp() * dt), torch.empty_like(x), 0
    for r, (a, old) in enumerate(zip(q, past)):
        S = state[r + 1] if old else torch.zeros_like(state[r + 1])
        for t in range(off, off + a):
            S = S * decay[t][:, None, None] + (dt[t][:, None] * b[t])[:, :, None] * x[t][:, None, :]
            y[t] = torch.einsum("hnp,hn->hp", S, c[t])
        state[r + 1] = S
        off += a
    y = (y + D[None, :, None] * x).view(-1, H * P) * torch.nn.functional.silu(z)
    return {"y": y, "state": state}
