"""The work that users of this package have it do, as cases that can be timed.

Every case goes through a public entry point with the arguments that nano-vllm's engine gives it:

  layer        ``Attention.forward`` called eagerly (``plugin.install()``): store of the new K/V rows, then prefill
               (packed, or through the block table when prompts share cached blocks) or decode
  step         ``decode_step``: store of the new token and decode attention in one call
  graph        a captured decode step replayed: per layer ``qk_norm_rope_store`` and ``Attention.forward(kv_stored=True)``
               (``plugin.fuse_pre_attention()``), the way the engine runs every decode step up to 512 sequences
  pre          ``qk_norm_rope_store`` on a prefill chunk's qkv activation
  sample       ``sample_tokens`` on the logits of a step (``plugin.fuse_sampler()``)
  inputs       ``DecodeInputStager.stage`` of a decode step (``plugin.fuse_decode_inputs()``)

Lengths belong to a case (they follow from its own numbers); all values, block placements and tokens follow from
the seed of ``prepare``.
"""
from __future__ import annotations

import random

import torch

from nano_vllm_b200 import attention, context, decode_inputs, workloads
from nano_vllm_b200.attention import Attention

BLOCK = workloads.BLOCK_SIZE
DEVICE = "cuda"
MAX_MODEL_LEN = 4096     # of the engine's benchmark: its decode tables are 16 blocks wide
MAX_BATCHED_TOKENS = 16384  # tokens of one prefill step
GEOMETRIES = {"qwen3-0.6b": workloads.QWEN3_06B, "qwen3-8b": workloads.QWEN3_8B, "qwen2-0.5b": workloads.QWEN2_05B}


def _heads(case):
    """Query heads, KV heads and head_dim of one rank's shard."""
    g, tp = GEOMETRIES[case["model"]], case.get("tp", 1)
    return g["hq"] // tp, g["hkv"] // tp, g["d"]


def _lengths(case):
    r = random.Random(case["lengths"])
    return [r.randint(case["lo"], case["hi"]) for _ in range(case["batch"])]


def _shared_blocks(case, lens):
    """Cached blocks of each prompt: every 4th shares 1 to 3 whole blocks with the one before it, where it can."""
    r = random.Random(case["lengths"] + 1)
    shared = [0] * len(lens)
    if case["shared"]:
        for i in range(3, len(lens), 4):
            shared[i] = min(r.randint(1, 3), (lens[i] - 1) // BLOCK, lens[i - 1] // BLOCK)
    return shared


def listed():
    return [
        # one user waiting for tokens with the graphs off: launches and host time are everything
        dict(name="layer-decode-1", kind="layer", phase="decode", model="qwen3-0.6b", batch=1, lo=317, hi=317, lengths=1),
        # a handful of concurrent requests of the benchmark's lengths (the single-layer decode configuration)
        dict(name="layer-decode-8", kind="layer", phase="decode", model="qwen3-0.6b", batch=8, lo=100, hi=1024, lengths=2),
        # long-context serving at head_dim 64: few KV heads, 128 scattered blocks a sequence
        dict(name="layer-decode-48-long", kind="layer", phase="decode", model="qwen2-0.5b", batch=48, lo=32768, hi=32768,
             lengths=3),
        # the largest decode step: the benchmark's headline workload, 5.5 GB of K/V
        dict(name="step-decode-256", kind="step", model="qwen3-8b", tp=1, batch=256, lo=2048, hi=8192, lengths=4),
        # a small batch decoding from a captured graph, all 28 layers: what the engine does between two prefills
        dict(name="graph-decode-16", kind="graph", model="qwen3-0.6b", layers=28, batch=16, lo=100, hi=1024, lengths=5),
        # one short prompt arrives: time to first token
        dict(name="layer-prompt-1", kind="layer", phase="prefill", model="qwen3-0.6b", batch=1, lo=201, hi=201, lengths=6,
             shared=False),
        # a full prefill step of the benchmark: ragged prompts, a quarter of them with cached prefixes
        dict(name="layer-prompts-64", kind="layer", phase="prefill", model="qwen3-0.6b", batch=64, lo=100, hi=1024,
             lengths=7, shared=True),
        # the same prompts in the head_dim 64 geometry (7 query heads to a KV head)
        dict(name="layer-prompts-64-d64", kind="layer", phase="prefill", model="qwen2-0.5b", batch=64, lo=100, hi=1024,
             lengths=7, shared=True),
        # long documents: the engine's largest prefill step, also its warm-up shape
        dict(name="layer-prompts-4x4096", kind="layer", phase="prefill", model="qwen3-0.6b", batch=4, lo=4096, hi=4096,
             lengths=8, shared=False),
        # the fused pre-attention step on that many tokens
        dict(name="pre-16384", kind="pre", model="qwen3-0.6b", tokens=16384),
        # sampling for the benchmark's full batch: bf16 logits over the whole vocabulary, T = 0.6
        dict(name="sample-256", kind="sample", batch=256, vocab=151936, dtype="bf16", temperature=0.6, spread=3.0),
        # host and device side of the inputs of that batch's decode step
        dict(name="inputs-256", kind="inputs", batch=256, lo=100, hi=2048, lengths=9),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prefill", "prefill", "step", "graph", "pre", "sample", "inputs"])
    model = rng.choice(sorted(GEOMETRIES))
    lengths = rng.randrange(1 << 30)
    if kind in ("decode", "step"):
        case = dict(kind="layer", phase="decode", model=model, lengths=lengths) if kind == "decode" else \
            dict(kind="step", model=model, tp=rng.choice([1, 2]) if model == "qwen2-0.5b" else rng.choice([1, 2, 4, 8]),
                 lengths=lengths)
        hi = _log_int(rng, 16, 32768)
        _, hkv, d = _heads(case)
        fits = int(3.5e9 / (hi * hkv * d * 4))  # K/V bytes of the batch
        return dict(case, batch=_log_int(rng, 1, max(1, min(512, fits))), lo=max(1, int(hi * rng.uniform(0.1, 1.0))), hi=hi)
    if kind == "prefill":
        hi = _log_int(rng, 8, 4096)
        lo = max(1, int(hi * rng.uniform(0.1, 1.0)))
        tokens = MAX_BATCHED_TOKENS if GEOMETRIES[model]["hq"] <= 16 else MAX_BATCHED_TOKENS // 2
        return dict(kind="layer", phase="prefill", model=model, batch=_log_int(rng, 1, max(1, min(256, tokens // hi))), lo=lo,
                    hi=hi, lengths=lengths, shared=rng.random() < 0.5)
    if kind == "graph":
        hi = _log_int(rng, 64, MAX_MODEL_LEN)
        batch = rng.choice([1, 2, 4, 8] + list(range(16, 513, 16)))
        layers = {"qwen3-0.6b": 28, "qwen3-8b": 36, "qwen2-0.5b": 24}[model]
        _, hkv, d = _heads(dict(model=model))
        while batch > 1 and batch * (hi + BLOCK) * hkv * d * 4 * layers > 4e9:
            batch = batch - 16 if batch > 16 else batch // 2
        return dict(kind="graph", model=model, layers=layers, batch=batch, lo=max(1, hi // 8), hi=hi, lengths=lengths)
    if kind == "pre":
        return dict(kind="pre", model=model, tokens=_log_int(rng, 1, MAX_BATCHED_TOKENS))
    if kind == "sample":
        return dict(kind="sample", batch=_log_int(rng, 1, 512), vocab=rng.choice([151936, 151643, 50257, 32000]),
                    dtype=rng.choice(["bf16", "bf16", "fp32"]), temperature=rng.choice([0.0, 0.6, 1.0]),
                    spread=rng.choice([1.0, 3.0]))
    return dict(kind="inputs", batch=_log_int(rng, 1, 512), lo=32, hi=_log_int(rng, 64, MAX_MODEL_LEN), lengths=lengths)


# ---- what a program holds before the call ------------------------------------------------------

class _Sequence:
    """What the stager reads of nano-vllm's Sequence."""

    def __init__(self, last_token, num_tokens, block_table, temperature):
        self.last_token, self.num_tokens = last_token, num_tokens
        self.block_table, self.temperature = block_table, temperature


def _rope_table(d):
    inv = 1.0 / (1e6 ** (torch.arange(0, d, 2, dtype=torch.float32, device=DEVICE) / d))
    f = torch.outer(torch.arange(MAX_MODEL_LEN, dtype=torch.float32, device=DEVICE), inv)
    return torch.cat([f.cos(), f.sin()], dim=1)


def _norm_weight(case, d, gen):
    if case["model"] == "qwen2-0.5b":  # no q/k norm in that model
        return None
    return (1 + 0.1 * torch.randn(d, generator=gen, device=DEVICE)).bfloat16()


def _prepare_layer(case, seed):
    hq, hkv, d = _heads(case)
    lens = _lengths(case)
    attn = Attention(hq, d, d ** -0.5, hkv)
    if case["phase"] == "decode":
        c = workloads.make_decode_case(seed, len(lens), 1, 1, hq, hkv, d, device=DEVICE, context_lens=lens).to(DEVICE)
        ctx = dict(is_prefill=False, slot_mapping=c.slot_mapping, context_lens=c.context_lens, block_tables=c.block_tables)
        new_k, new_v = c.k_new, c.v_new
    else:
        c = workloads.make_prefill_case(seed, len(lens), 1, 1, hq, hkv, d, device=DEVICE, lengths=lens,
                                        shared_blocks=_shared_blocks(case, lens)).to(DEVICE)
        ctx = dict(is_prefill=True, cu_seqlens_q=c.cu_seqlens_q, cu_seqlens_k=c.cu_seqlens_k, max_seqlen_q=c.max_seqlen_q,
                   max_seqlen_k=c.max_seqlen_k, slot_mapping=c.slot_mapping, block_tables=c.block_tables)
        new_k, new_v = c.k, c.v
    # the engine's activations: q, k and v are slices of the qkv projection's output
    n = c.q.shape[0]
    qkv = torch.cat([c.q.reshape(n, -1), new_k.reshape(n, -1), new_v.reshape(n, -1)], dim=1)
    q, k, v = qkv.split([hq * d, hkv * d, hkv * d], dim=1)
    attn.k_cache, attn.v_cache = c.k_cache, c.v_cache
    return dict(kind="layer", attn=attn, q=q, k=k, v=v, ctx=ctx)


def _prepare_step(case, seed):
    hq, hkv, d = _heads(case)
    lens = _lengths(case)
    c = workloads.make_decode_case(seed, len(lens), 1, 1, hq, hkv, d, device=DEVICE, context_lens=lens).to(DEVICE)
    return dict(kind="step", c=c)


def _prepare_graph(case, seed):
    hq, hkv, d = _heads(case)
    lens, layers = _lengths(case), case["layers"]
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    one = workloads.make_decode_case(seed, len(lens), 1, 1, 1, 1, 64, device=DEVICE, context_lens=lens,
                                     table_width=MAX_MODEL_LEN // BLOCK).to(DEVICE)  # lengths, tables, slots
    kv = torch.randn(2, layers, one.k_cache.shape[0], BLOCK, hkv, d, generator=gen, dtype=torch.bfloat16, device=DEVICE)
    qkv = torch.randn(layers, len(lens), (hq + 2 * hkv) * d, generator=gen, dtype=torch.bfloat16, device=DEVICE)
    positions = (one.context_lens - 1).long()
    qw, kw, rope = _norm_weight(case, d, gen), _norm_weight(case, d, gen), _rope_table(d)
    stack = []
    for i in range(layers):
        attn = Attention(hq, d, d ** -0.5, hkv)
        attn.k_cache, attn.v_cache = kv[0, i], kv[1, i]
        stack.append(attn)

    def forward(n):
        context.set_context(False, slot_mapping=one.slot_mapping, context_lens=one.context_lens, block_tables=one.block_tables)
        outs = []
        for i in range(n):
            attention.qk_norm_rope_store(qkv[i], positions, qw, kw, rope, 1e-6, one.slot_mapping, stack[i].k_cache,
                                         stack[i].v_cache, hq, hkv, d)
            q, k, v = qkv[i].split([hq * d, hkv * d, hkv * d], dim=1)
            outs.append(stack[i](q, k, v, kv_stored=True))
        context.reset_context()
        return outs

    forward(1)  # warm-up outside capture, as the engine does
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs = forward(layers)
    return dict(kind="graph", graph=graph, outs=outs, qkv=qkv, kv=kv, keep=(one, positions, qw, kw, rope, stack))


def _prepare_pre(case, seed):
    hq, hkv, d = _heads(case)
    n = case["tokens"]
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    blocks = (n + BLOCK - 1) // BLOCK + 3
    perm = torch.randperm(blocks, generator=gen, device=DEVICE)
    at = torch.arange(n, device=DEVICE)
    qkv = torch.randn(n, (hq + 2 * hkv) * d, generator=gen, dtype=torch.bfloat16, device=DEVICE)
    kv = torch.zeros(2, blocks, BLOCK, hkv, d, dtype=torch.bfloat16, device=DEVICE)
    return dict(kind="pre", qkv=qkv, kv=kv, positions=at % MAX_MODEL_LEN,
                slots=(perm[at // BLOCK] * BLOCK + at % BLOCK).int(), qw=_norm_weight(case, d, gen), kw=_norm_weight(case, d, gen),
                rope=_rope_table(d), heads=(hq, hkv, d))


def _prepare_sample(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    dtype = torch.float32 if case["dtype"] == "fp32" else torch.bfloat16
    logits = torch.randn(case["batch"], case["vocab"], generator=gen, dtype=torch.float32, device=DEVICE).mul_(case["spread"])
    temperatures = torch.full((case["batch"],), case["temperature"], dtype=torch.float32, device=DEVICE)
    return dict(kind="sample", logits=logits.to(dtype), temperatures=temperatures, seed=seed, step=0)


def _prepare_inputs(case, seed):
    r = random.Random(seed)
    lens = _lengths(case)
    width = MAX_MODEL_LEN // BLOCK
    pool = list(range(sum((n + BLOCK - 1) // BLOCK for n in lens)))
    r.shuffle(pool)
    seqs = [_Sequence(r.randrange(151936), n, [pool.pop() for _ in range((n + BLOCK - 1) // BLOCK)], 0.6) for n in lens]
    sizes = [1, 2, 4, 8] + list(range(16, 513, 16))
    graph_bs = next(x for x in sizes if x >= len(seqs))
    i64 = dict(dtype=torch.int64, device=DEVICE)
    i32 = dict(dtype=torch.int32, device=DEVICE)
    graph_vars = {"input_ids": torch.zeros(graph_bs, **i64), "positions": torch.zeros(graph_bs, **i64),
                  "slot_mapping": torch.zeros(graph_bs, **i32), "context_lens": torch.zeros(graph_bs, **i32),
                  "block_tables": torch.zeros(graph_bs, width, **i32)}
    stager = decode_inputs.DecodeInputStager(512, width, torch.device(DEVICE, torch.cuda.current_device()))
    return dict(kind="inputs", seqs=seqs, graph_bs=graph_bs, graph_vars=graph_vars, stager=stager)


def prepare(case, seed):
    make = {"layer": _prepare_layer, "step": _prepare_step, "graph": _prepare_graph, "pre": _prepare_pre,
            "sample": _prepare_sample, "inputs": _prepare_inputs}[case["kind"]]
    return make(case, seed)


# ---- one pass ----------------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "layer":
        attn = state["attn"]
        context.set_context(**state["ctx"])
        o = attn(state["q"], state["k"], state["v"])
        context.reset_context()
        return {"o": o, "k_cache": attn.k_cache, "v_cache": attn.v_cache}
    if kind == "step":
        c = state["c"]
        o = attention.decode_step(c.q, c.k_new, c.v_new, c.k_cache, c.v_cache, c.slot_mapping, c.context_lens, c.block_tables,
                                  c.scale)
        return {"o": o, "k_cache": c.k_cache, "v_cache": c.v_cache}
    if kind == "graph":
        state["graph"].replay()
        return {"o": state["outs"], "qkv": state["qkv"], "kv": state["kv"]}
    if kind == "pre":
        hq, hkv, d = state["heads"]
        attention.qk_norm_rope_store(state["qkv"], state["positions"], state["qw"], state["kw"], state["rope"], 1e-6,
                                     state["slots"], state["kv"][0], state["kv"][1], hq, hkv, d)
        return {"qkv": state["qkv"], "kv": state["kv"]}
    if kind == "sample":
        state["step"] += 1
        return attention.sample_tokens(state["logits"], state["temperatures"], seed=state["seed"], step=state["step"])
    temperatures = state["stager"].stage(state["seqs"], state["graph_bs"], state["graph_vars"])
    return {**state["graph_vars"], "temperatures": temperatures}


# ---- what a pass cannot do without, and how far another implementation may be off ----------------

def _pre_bytes(n, hq, hkv, d):
    """qkv read, q and k rewritten, k and v rows put into the cache; position and slot of each token."""
    return n * (2 * d * ((hq + 2 * hkv) + (hq + hkv) + 2 * hkv) + 12)


def work(case):
    kind = case["kind"]
    if kind == "sample":
        size = 4 if case["dtype"] == "fp32" else 2
        return {"bytes": case["batch"] * (case["vocab"] * size + 12), "flops": 2 * case["batch"] * case["vocab"]}
    if kind == "inputs":
        blocks = sum((n + BLOCK - 1) // BLOCK for n in _lengths(case))
        staged = case["batch"] * 20 + 4 + 4 * blocks  # host block read; the static tensors written
        return {"bytes": staged + case["batch"] * (24 + 4 * (MAX_MODEL_LEN // BLOCK)), "flops": 0}
    hq, hkv, d = _heads(case)
    if kind == "pre":
        n = case["tokens"]
        return {"bytes": _pre_bytes(n, hq, hkv, d), "flops": 10 * n * (hq + hkv) * d}
    lens = _lengths(case)
    if kind == "layer" and case["phase"] == "prefill":
        lq = [n - BLOCK * s for n, s in zip(lens, _shared_blocks(case, lens))]
        n = sum(lq)
        return {"bytes": workloads.store_bytes(n, hkv * d) + 2 * (2 * n * hq * d) + 2 * (2 * (sum(lens) - n) * hkv * d),
                "flops": workloads.prefill_flops(lq, lens, hq, d)}
    # decode: the new rows are stored and everything cached is read
    byts = workloads.decode_bytes(lens, hq, hkv, d) + workloads.store_bytes(len(lens), hkv * d)
    flops = 4 * hq * d * sum(lens)
    if kind == "graph":
        byts = case["layers"] * (workloads.decode_bytes(lens, hq, hkv, d) + _pre_bytes(len(lens), hq, hkv, d))
        flops *= case["layers"]
    return {"bytes": byts, "flops": flops}


def tolerance(case):
    if case["kind"] in ("sample", "inputs"):
        return "exact"  # whole numbers, and temperatures copied
    # bf16 probabilities and bf16 outputs; copied rows do not differ at all
    return {"rel": 6e-3, "max": 5e-2}
