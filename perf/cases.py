"""The attention work of a serving step, as a program that uses this library has it done.

A case is one pass of one kind:

  decode         one layer of a decode step: the step's new K / V rows go into the paged cache (by the fused prologue from
                 the packed qkv rows, or by a store of finished rows), then paged decode attention over the whole context
  layers         one replay of the CUDA graph that holds a decode step's attention blocks, layer after layer: QKV projection
                 with prologue and store, decode attention, output projection, every layer with its own weights and cache
  prefill        one layer of a prefill step: prologue or store, then varlen causal attention over dense or paged keys
  prefill_layer  the same between its two projections (QKV with prologue and store, attention, output projection)
  mixed          one layer of a continuous-batching step with prompts and decode rows: two stores, one attention call

Heads are those of the 32 / 8 and 16 / 8 head configurations and of their tensor-parallel shards, head_dim 128, cache blocks
of 256 tokens.  Lengths are spread evenly over their range, in an order that comes from the seed, so that a case is the
same amount of work for every seed.
"""
from __future__ import annotations

import importlib
import math
import random

import numpy as np
import torch

nvk = importlib.import_module("nano-vllm-cpp_b200")

D, BS = 128, 256
EPS, ROPE_BASE = 1e-6, 1.0e6
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
HEADS = ((32, 8), (16, 4), (8, 2), (4, 1), (16, 8), (8, 4))


def listed():
    return [
        # One user, a short conversation: what a call costs when there is next to nothing to read.
        decode("decode-1", 32, 8, 1, 300, 300),
        # A few dozen users with mixed context lengths, the bulk of a server's day.
        decode("decode-37", 32, 8, 37, 100, 2048, table_blocks=16),
        # The largest: the repository's headline configuration (batch 256, context 1024 to 8192, store + decode).
        decode("decode-256", 32, 8, 256, 1024, 8192, write="store"),
        # A handful of long documents: few sequences, tens of thousands of keys each, 64-bit indices.
        decode("decode-long-3", 16, 8, 3, 9000, 40000, dtype="fp16", index="i64"),
        # The int8 cache: quantising store and decode.
        decode("decode-int8-100", 32, 8, 100, 500, 4096, kv="int8", write="store"),
        # The e4m3 cache on one of eight tensor-parallel ranks (one KV head).
        decode("decode-fp8-rank", 4, 1, 256, 100, 2048, kv="fp8", write="store"),
        # The fp32 configuration of the CPU reference.
        decode("decode-fp32-8", 16, 8, 8, 64, 1024, dtype="fp32", write="store"),
        # A captured decode step of eight attention blocks with their projections.
        layers("layers-64", 32, 8, 64, 100, 2048, num_layers=8, hidden=4096, table_blocks=8),
        # A short question on top of a cached prompt: the smallest prefill.
        prefill("prefill-1", 32, 8, 1, 77, 77, prefix=512),
        # A batch of short prompts of ragged length, whole attention block.
        prefill_layer("prefill-layer-24", 32, 8, 24, 20, 600, hidden=4096),
        # The largest prefill: 16 prompts of 512 to 4096 tokens, half of them behind a cached prefix.
        prefill("prefill-16", 32, 8, 16, 512, 4096, prefix=768, prefix_share=0.5, write="store"),
        # Prompts and decode rows in one step.
        mixed("mixed-3-90", 32, 8, 3, 500, 2048, 90, 500, 8192),
    ]


def decode(name, q_heads, kv_heads, batch, ctx_lo, ctx_hi, dtype="bf16", kv="same", index="i32", write="prologue", table_blocks=0):
    return dict(name=name, kind="decode", q_heads=q_heads, kv_heads=kv_heads, batch=batch, ctx_lo=ctx_lo, ctx_hi=ctx_hi, dtype=dtype, kv=kv,
                index=index, write=write, table_blocks=table_blocks)


def layers(name, q_heads, kv_heads, batch, ctx_lo, ctx_hi, num_layers, hidden, table_blocks, dtype="bf16"):
    return dict(name=name, kind="layers", q_heads=q_heads, kv_heads=kv_heads, batch=batch, ctx_lo=ctx_lo, ctx_hi=ctx_hi, layers=num_layers,
                hidden=hidden, dtype=dtype, index="i32", table_blocks=table_blocks)


def prefill(name, q_heads, kv_heads, seqs, q_lo, q_hi, prefix=0, prefix_share=1.0, dtype="bf16", index="i32", write="prologue", keys="paged"):
    return dict(name=name, kind="prefill", q_heads=q_heads, kv_heads=kv_heads, seqs=seqs, q_lo=q_lo, q_hi=q_hi, prefix=prefix,
                prefix_share=prefix_share, dtype=dtype, index=index, write=write, keys=keys)


def prefill_layer(name, q_heads, kv_heads, seqs, q_lo, q_hi, hidden, dtype="bf16"):
    return dict(name=name, kind="prefill_layer", q_heads=q_heads, kv_heads=kv_heads, seqs=seqs, q_lo=q_lo, q_hi=q_hi, prefix=0, prefix_share=0.0,
                hidden=hidden, dtype=dtype, index="i32", keys="paged")


def mixed(name, q_heads, kv_heads, seqs, q_lo, q_hi, batch, ctx_lo, ctx_hi, dtype="bf16"):
    return dict(name=name, kind="mixed", q_heads=q_heads, kv_heads=kv_heads, seqs=seqs, q_lo=q_lo, q_hi=q_hi, prefix=0, prefix_share=0.0,
                batch=batch, ctx_lo=ctx_lo, ctx_hi=ctx_hi, dtype=dtype, index="i32", keys="paged")


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the same ranges; none is more work than the largest listed one of its kind."""
    kind = rng.choice(("decode", "decode", "decode", "decode8", "decode32", "layers", "prefill", "prefill", "prefill_layer", "mixed"))
    hq, hkv = rng.choice(HEADS)
    dtype = rng.choice(("bf16", "bf16", "fp16"))
    index = rng.choice(("i32", "i32", "i64"))
    if kind.startswith("decode"):
        batch = _log(rng, 1, 8 if kind == "decode32" else 256)
        hi = _log(rng, 64, min(40000, 256 * 8192 // batch))
        lo = rng.randint(max(1, hi // 20), hi)
        table = rng.choice((0, -(-hi // BS) + rng.randint(0, 16)))
        if kind == "decode":
            c = decode("", hq, hkv, batch, lo, hi, dtype, "same", index, rng.choice(("prologue", "store")), table)
        elif kind == "decode8":
            c = decode("", hq, hkv, batch, lo, hi, dtype, rng.choice(("int8", "fp8")), index, "store", table)
        else:
            hi = min(hi, 4096)
            c = decode("", hq, hkv, batch, min(lo, hi), hi, "fp32", "same", index, "store", table)
    elif kind == "layers":
        batch, hi = _log(rng, 1, 128), _log(rng, 64, 2048)
        c = layers("", hq, hkv, batch, rng.randint(max(1, hi // 20), hi), hi, rng.randint(4, 8), rng.choice((2048, 4096)),
                   -(-hi // BS) + rng.randint(0, 8), dtype)
    elif kind == "mixed":
        seqs, hi, batch, ctx = _log(rng, 1, 6), _log(rng, 40, 2048), _log(rng, 4, 128), _log(rng, 200, 8192)
        c = mixed("", hq, hkv, seqs, rng.randint(max(1, hi // 8), hi), hi, batch, rng.randint(max(1, ctx // 16), ctx), ctx, dtype)
    else:
        seqs = _log(rng, 1, 32)
        hi = _log(rng, 8, min(8192, 40000 // seqs, int(10000 / seqs ** 0.5)))
        lo = rng.randint(max(1, hi // 8), hi)
        if kind == "prefill_layer":
            c = prefill_layer("", hq, hkv, seqs, min(lo, 1 + 7000 // seqs), min(hi, 1 + 7000 // seqs), rng.choice((2048, 4096)), dtype)
        else:
            keys = rng.choice(("paged", "paged", "dense"))
            prefix, share = (rng.randint(1, 4) * BS, rng.choice((0.0, 0.5, 1.0))) if keys == "paged" else (0, 0.0)
            c = prefill("", hq, hkv, seqs, lo, hi, prefix, share, dtype, index, "store" if keys == "dense" else rng.choice(("prologue", "store")), keys)
    del c["name"]
    return c


# ---- lengths and sizes ------------------------------------------------------------------------------------------------------

def _spread(lo, hi, n):
    """n lengths over [lo, hi], the middles of n equal parts."""
    return [lo + int((hi - lo) * (i + 0.5) / n) for i in range(n)]


def _prompts(c):
    """(new tokens, cached prefix) of every prompt."""
    q = _spread(c["q_lo"], c["q_hi"], c["seqs"])
    hits = round(c["seqs"] * c["prefix_share"])
    return [(n, c["prefix"] if (i * hits) // len(q) != ((i + 1) * hits) // len(q) else 0) for i, n in enumerate(q)]


def work(c):
    es = 4 if c["dtype"] == "fp32" else 2
    hq, hkv, nbytes, flops = c["q_heads"], c["kv_heads"], 0, 0
    row = (hq + 2 * hkv) * D * es                     # a token's q, k and v
    if "batch" in c:                                  # decode rows
        ctx, n = _spread(c["ctx_lo"], c["ctx_hi"], c["batch"]), c.get("layers", 1)
        kv = 2 * D * es if c.get("kv", "same") == "same" else 2 * (D + 2)
        nbytes += n * (sum(ctx) * hkv * kv + c["batch"] * hq * D * es + sum(-(-t // BS) for t in ctx) * 4)
        flops += n * 4 * hq * D * sum(ctx)
        if c["kind"] == "layers":
            wide = (2 * hq + 2 * hkv) * D * c["hidden"]
            nbytes += n * (wide * es + c["batch"] * (2 * c["hidden"] + hq * D) * es)
            flops += n * 2 * wide * c["batch"]
        else:
            nbytes += c["batch"] * (row + hkv * kv + (D * 4 if c.get("write") == "prologue" else 0))
    if "seqs" in c:                                   # prompts
        lens = _prompts(c)
        rows, cached = sum(n for n, _ in lens), sum(p for _, p in lens)
        flops += sum(4 * hq * D * (n * p + n * (n + 1) // 2) for n, p in lens)
        nbytes += cached * hkv * 2 * D * es + rows * (hq + 2 * hkv) * D * es   # cached keys in; result and the new K / V rows out
        if c["kind"] == "prefill_layer":
            wide = (2 * hq + 2 * hkv) * D * c["hidden"]
            nbytes += wide * es + rows * (2 * c["hidden"] + hq * D) * es
            flops += 2 * wide * rows
        else:
            nbytes += rows * (row + (D * 4 if c.get("write") == "prologue" else 0))
    return {"bytes": nbytes, "flops": flops}


def tolerance(c):
    # Attention in 16-bit types rounds its probabilities and its results; cache bytes of the 8-bit formats stay as they are
    # (no share of them may differ).
    return {"rel": 1e-5} if c["dtype"] == "fp32" else {"rel": 1e-2}


# ---- inputs -----------------------------------------------------------------------------------------------------------------

class _Maker:
    """Seeded inputs on the GPU and the host-side metadata of a step."""

    def __init__(self, c, seed):
        self.c, self.rng, self.order = c, np.random.default_rng(seed), random.Random(seed)
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)
        self.dtype = DTYPES[c["dtype"]]
        self.index = torch.int64 if c["index"] == "i64" else torch.int32

    def normal(self, *shape, std=1.0, mean=0.0):
        return torch.empty(shape, device="cuda", dtype=self.dtype).normal_(mean, std, generator=self.gen)

    def up(self, a, dtype=torch.int32):
        return torch.from_numpy(np.ascontiguousarray(a)).to("cuda", dtype)

    def shuffled(self, v):
        v = list(v)
        self.order.shuffle(v)
        return v

    def tables(self, lens, width=0):
        """Block tables of sequences of these lengths, a random permutation of the pool: (tables, blocks in the pool)."""
        need = [-(-n // BS) for n in lens]
        perm, at = self.rng.permutation(sum(need)), 0
        out = np.zeros((len(lens), max(width, max(need))), np.int64)
        for i, n in enumerate(need):
            out[i, :n] = perm[at:at + n]
            at += n
        return out, sum(need)

    def cache(self, blocks, lead=()):
        return self.normal(*lead, blocks, BS, self.c["kv_heads"], D)

    def rope(self, positions):
        at = torch.arange(positions, device="cuda", dtype=torch.float64)
        ang = at[:, None] / ROPE_BASE ** (torch.arange(0, D, 2, device="cuda", dtype=torch.float64) / D)
        return torch.cat([ang.cos(), ang.sin()], 1).float()

    def norms(self):
        return self.normal(D, std=0.1, mean=1.0), self.normal(D, std=0.1, mean=1.0)


def _slots(tables, seq, pos):
    return tables[seq, pos // BS] * BS + pos % BS


def _decode_rows(m, s, offset=0):
    """Context lengths, tables, slots and positions of the decode rows; returns the blocks their caches take."""
    c = m.c
    ctx = np.array(m.shuffled(_spread(c["ctx_lo"], c["ctx_hi"], c["batch"])))
    tables, pool = m.tables(ctx, c.get("table_blocks", 0))
    slots = _slots(tables, np.arange(len(ctx)), ctx - 1)
    s.ctx, s.tables = m.up(ctx, m.index), m.up(tables + offset, m.index)
    s.slots, s.positions = m.up(slots + offset * BS), m.up(ctx - 1)
    need = nvk.decode_attention_workspace_bytes(c["batch"], c["q_heads"], c["kv_heads"], D, tables.shape[1], BS)
    s.workspace = torch.empty(max(16, need), dtype=torch.uint8, device="cuda")
    return pool, int(ctx.max())


def _prompt_rows(m, s):
    """The same for the rows of the prompts."""
    lens = m.shuffled(_prompts(m.c))
    n, p = np.array([x for x, _ in lens]), np.array([x for _, x in lens])
    tables, pool = m.tables(n + p)
    seq = np.repeat(np.arange(len(n)), n)
    pos = np.concatenate([np.arange(a, a + b) for a, b in zip(p, n)])
    s.cu_q, s.cu_k = (m.up(np.concatenate([[0], np.cumsum(v)]), m.index) for v in (n, n + p))
    s.p_tables, s.p_slots, s.p_positions = m.up(tables, m.index), m.up(_slots(tables, seq, pos)), m.up(pos)
    return pool, int(n.sum()), int((n + p).max())


class _State:
    pass


def prepare(case, seed):
    c, m, s = case, _Maker(case, seed), _State()
    s.c, s.scale = c, 1.0 / math.sqrt(D)
    hq, hkv = c["q_heads"], c["kv_heads"]
    packed = (hq + 2 * hkv) * D
    if c["kind"] == "decode":
        pool, longest = _decode_rows(m, s)
        b = c["batch"]
        if c["write"] == "prologue":
            s.qkv, (s.q_norm, s.k_norm), s.rope = m.normal(b, packed), m.norms(), m.rope(longest)
            s.q = torch.empty((b, hq, D), device="cuda", dtype=m.dtype)
        else:
            s.q, s.k, s.v = m.normal(b, hq, D), m.normal(b, hkv, D), m.normal(b, hkv, D)
        s.k_cache, s.v_cache = m.cache(pool), m.cache(pool)
        if c["kv"] != "same":
            full = s.k_cache, s.v_cache
            s.k_cache, s.v_cache = (torch.empty(x.shape, device="cuda", dtype=torch.int8 if c["kv"] == "int8" else torch.uint8) for x in full)
            s.k_scale, s.v_scale = (torch.empty(x.shape[:-1], device="cuda", dtype=torch.float16) for x in full)
            rows = torch.arange(pool * BS, device="cuda", dtype=torch.int32)
            _store8(c)(*(x.view(-1, hkv, D) for x in full), s.k_cache, s.v_cache, s.k_scale, s.v_scale, rows)
        s.out = torch.empty_like(s.q)
    elif c["kind"] == "layers":
        pool, longest = _decode_rows(m, s)
        n, b, hidden = c["layers"], c["batch"], c["hidden"]
        s.x, s.w_qkv, s.w_o = m.normal(n, b, hidden), m.normal(n, packed, hidden, std=hidden ** -0.5), m.normal(n, hidden, hq * D, std=(hq * D) ** -0.5)
        (s.q_norm, s.k_norm), s.rope = m.norms(), m.rope(longest)
        s.k_cache, s.v_cache = m.cache(pool, (n,)), m.cache(pool, (n,))
        s.q = torch.empty((n, b, hq, D), device="cuda", dtype=m.dtype)
        s.attn, s.out = torch.empty_like(s.q), torch.empty_like(s.x)
        _decode_layers(s, 1)                              # everything is loaded before the capture
        torch.cuda.synchronize()
        s.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s.graph):
            _decode_layers(s, n)
    else:
        pool, rows, longest = _prompt_rows(m, s)
        if c["kind"] == "mixed":
            d_pool, d_longest = _decode_rows(m, s, offset=pool)
            pool += d_pool
            s.d_q, s.d_k, s.d_v = m.normal(c["batch"], hq, D), m.normal(c["batch"], hkv, D), m.normal(c["batch"], hkv, D)
            s.d_out = torch.empty_like(s.d_q)
        s.k_cache, s.v_cache = m.cache(pool), m.cache(pool)
        if c["kind"] == "prefill_layer":
            s.x = m.normal(rows, c["hidden"])
            s.w_qkv, s.w_o = m.normal(packed, c["hidden"], std=c["hidden"] ** -0.5), m.normal(c["hidden"], hq * D, std=(hq * D) ** -0.5)
            s.y = torch.empty_like(s.x)
        elif c.get("write") == "prologue":
            s.qkv = m.normal(rows, packed)
        if c["kind"] == "prefill_layer" or c.get("write") == "prologue":
            (s.q_norm, s.k_norm), s.rope = m.norms(), m.rope(longest)
            s.q = torch.empty((rows, hq, D), device="cuda", dtype=m.dtype)
        else:
            s.q, s.k, s.v = m.normal(rows, hq, D), m.normal(rows, hkv, D), m.normal(rows, hkv, D)
        s.out = torch.empty_like(s.q)
    return s


# ---- one pass ---------------------------------------------------------------------------------------------------------------

def _store8(c):
    return nvk.store_kvcache_int8 if c["kv"] == "int8" else nvk.store_kvcache_fp8


def _decode_layers(s, n):
    c = s.c
    hq, hkv = c["q_heads"], c["kv_heads"]
    for i in range(n):
        nvk.qkv_linear_norm_rope_store(s.x[i], s.w_qkv[i], s.positions, s.q_norm, s.k_norm, EPS, s.rope, s.slots, s.k_cache[i], s.v_cache[i],
                                       hq, hkv, D, s.q[i])
        nvk.launch_decode_attention_paged(s.q[i], s.k_cache[i], s.v_cache[i], s.ctx, s.tables, hkv, D, BS, s.scale, s.attn[i], s.workspace)
        nvk.linear(s.attn[i].view(c["batch"], hq * D), s.w_o[i], s.out[i])


def _run_decode(s):
    c = s.c
    hq, hkv = c["q_heads"], c["kv_heads"]
    if c["kv"] != "same":
        _store8(c)(s.k, s.v, s.k_cache, s.v_cache, s.k_scale, s.v_scale, s.slots)
        attend = nvk.launch_decode_attention_paged_int8 if c["kv"] == "int8" else nvk.launch_decode_attention_paged_fp8
        attend(s.q, s.k_cache, s.v_cache, s.k_scale, s.v_scale, s.ctx, s.tables, hkv, D, BS, s.scale, s.out, s.workspace)
        return s.out, s.k_cache, s.v_cache, s.k_scale, s.v_scale
    if c["write"] == "prologue":
        nvk.fused_split_norm_rope_store(s.qkv, s.positions, s.q_norm, s.k_norm, EPS, s.rope, s.slots, s.k_cache, s.v_cache, hq, hkv, D, s.q)
    else:
        nvk.store_kvcache(s.k, s.v, s.k_cache, s.v_cache, s.slots)
    nvk.launch_decode_attention_paged(s.q, s.k_cache, s.v_cache, s.ctx, s.tables, hkv, D, BS, s.scale, s.out, s.workspace)
    return s.out, s.k_cache, s.v_cache


def _run_prefill(s):
    c = s.c
    hq, hkv = c["q_heads"], c["kv_heads"]
    if c["kind"] == "prefill_layer":
        nvk.qkv_linear_norm_rope_store(s.x, s.w_qkv, s.p_positions, s.q_norm, s.k_norm, EPS, s.rope, s.p_slots, s.k_cache, s.v_cache, hq, hkv, D, s.q)
    elif c["write"] == "prologue":
        nvk.fused_split_norm_rope_store(s.qkv, s.p_positions, s.q_norm, s.k_norm, EPS, s.rope, s.p_slots, s.k_cache, s.v_cache, hq, hkv, D, s.q)
    else:
        nvk.store_kvcache(s.k, s.v, s.k_cache, s.v_cache, s.p_slots)
    if c["keys"] == "dense":
        nvk.launch_prefill_attention_dense(s.q, s.cu_q, s.k, s.v, s.cu_k, hkv, D, s.scale, s.out)
    else:
        nvk.launch_prefill_attention_paged(s.q, s.cu_q, s.k_cache, s.v_cache, s.cu_k, s.p_tables, hkv, D, BS, s.scale, s.out)
    if c["kind"] == "prefill_layer":
        nvk.linear(s.out.view(s.out.shape[0], hq * D), s.w_o, s.y)
        return s.y, s.q, s.out, s.k_cache, s.v_cache
    return s.out, s.k_cache, s.v_cache


def run(s):
    kind = s.c["kind"]
    if kind == "decode":
        return _run_decode(s)
    if kind == "layers":
        s.graph.replay()
        return s.out, s.q, s.attn, s.k_cache, s.v_cache
    if kind == "mixed":
        nvk.store_kvcache(s.k, s.v, s.k_cache, s.v_cache, s.p_slots)
        nvk.store_kvcache(s.d_k, s.d_v, s.k_cache, s.v_cache, s.slots)
        nvk.attention_mixed_step(s.q, s.cu_q, None, None, s.cu_k, s.p_tables, s.out, s.d_q, s.ctx, s.tables, s.d_out, s.k_cache, s.v_cache,
                                 s.c["kv_heads"], D, BS, s.scale, s.workspace)
        return s.out, s.d_out, s.k_cache, s.v_cache
    return _run_prefill(s)
