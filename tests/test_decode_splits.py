"""Tensor-core paged decode at the edges of how a sequence is shared out: clusters of 1 to 8 blocks, chunks with few and with many
partial results, no workspace, whole contexts taken
longest first, contexts around a tile, a round of the four warps' tiles, a chunk and a part, equal and empty ones among them."""
import numpy as np
import pytest

import oracle
from util import assert_attention_close, nvk, to_dev, to_np, workloads

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

EDGES = [0, 1, 15, 16, 17, 63, 64, 65, 127, 129, 255, 256, 257, 511, 513]


def _workspace(batch, hq, hkv, blocks, bs):
    return torch.empty(max(16, nvk().decode_attention_workspace_bytes(batch, hq, hkv, 128, blocks, bs)), dtype=torch.uint8, device="cuda")


@pytest.mark.parametrize("hq,hkv,bs,lens,table_blocks", [
    (8, 2, 256, [300], 2),                                  # eight blocks per (sequence, KV head)
    (32, 8, 256, [700, 0, 33], 4),
    (16, 8, 16, EDGES[:9], 9),                              # four, two and one
    (4, 4, 256, EDGES, 3),
    (8, 8, 32, EDGES * 3, 17),
    (4, 1, 256, (EDGES * 3)[:33], 3),                       # as many clusters of eight as are resident, and one more
    (4, 1, 256, (EDGES * 3)[:34], 3),
    (4, 1, 256, (EDGES * 5)[:71], 4),                       # the same for clusters of four
    (4, 1, 256, (EDGES * 5)[:72], 4),
    (4, 1, 256, (EDGES[:12] * 4)[:40], 2),                  # tables of 512 keys in one block each
    (8, 1, 256, [2047, 2048, 2049, 1, 9000], 80),           # chunks: up to 36 parts of one context
    (16, 8, 256, EDGES * 3 + [4096, 2500, 2048], 16),       # whole contexts, 4096-key tables
    (16, 8, 256, EDGES * 2 + [4096, 2500, 2048, 9, 99, 1, 2, 3], 16),   # and just past a wave: chunks, longest first
    (4, 1, 256, (EDGES * 15)[:221] + [2048], 8),            # 2048-key tables, whole
    (4, 1, 256, (EDGES * 15)[:220] + [2048], 8),            # and in two chunks
    (8, 2, 256, [300] * 170 + EDGES * 3 + [1024], 4),       # longest first with most in one class of length
    (16, 8, 256, [4097, 8192, 5000] + EDGES * 3, 33),       # chunks: up to 5 parts
    (16, 8, 256, [300, 0, 2500, 17], 128),                  # most chunks empty, chunk after chunk
    (8, 1, 256, [300, 17, 9000] + [40] * 34, 80),           # merged by a block per head, 296 rows
    (8, 1, 256, [300, 17, 9000] + [40] * 35, 80),           # and by warps, 304
    (8, 8, 256, EDGES * 5, 20),                             # most chunks empty, sequence after sequence
])
def test_every_way_to_share_out_a_context_matches_the_oracle(hq, hkv, bs, lens, table_blocks):
    w = workloads().make_decode_workload(len(lens), hq, hkv, 128, bs, 0, 0, seed=len(lens) + hq, context_lens=np.array(lens, np.int32),
                                         pad_blocks_to=table_blocks)
    bf = torch.bfloat16
    q, kc, vc, ctx, bt = to_dev(w["q"], bf), to_dev(w["k_cache"], bf), to_dev(w["v_cache"], bf), to_dev(w["context_lens"]), to_dev(w["block_tables"])
    ref = oracle.decode_attention_paged(w["q"], w["k_cache"], w["v_cache"], w["context_lens"], w["block_tables"], hkv, 128, bs, w["scale"])
    for ws in (_workspace(len(lens), hq, hkv, bt.shape[1], bs), None):
        out = torch.full_like(q, float("nan"))
        nvk().launch_decode_attention_paged(q, kc, vc, ctx, bt, hkv, 128, bs, w["scale"], out, ws)
        assert_attention_close(to_np(out), ref)


@pytest.mark.parametrize("fmt", ["int8", "fp8"])
@pytest.mark.parametrize("hq,hkv,lens,table_blocks", [(8, 2, [300, 17], 2), (16, 8, EDGES * 4, 3), (8, 1, [5000, 1, 2049], 40), (8, 8, EDGES * 4, 20),
                                                     (4, 1, (EDGES * 18)[:263] + [1024], 4), (4, 1, (EDGES * 25)[:369] + [2048], 8)])
def test_8_bit_caches_do_not_depend_on_how_a_context_is_shared_out(fmt, hq, hkv, lens, table_blocks):
    w = workloads().make_decode_workload(len(lens), hq, hkv, 128, 256, 0, 0, seed=5, context_lens=np.array(lens, np.int32), pad_blocks_to=table_blocks)
    bf, lib = torch.bfloat16, nvk()
    store, decode = ((lib.store_kvcache_int8, lib.launch_decode_attention_paged_int8) if fmt == "int8" else
                     (lib.store_kvcache_fp8, lib.launch_decode_attention_paged_fp8))
    k16, v16 = to_dev(w["k_cache"], bf), to_dev(w["v_cache"], bf)
    kc, vc = (torch.empty(k16.shape, dtype=torch.int8 if fmt == "int8" else torch.uint8, device="cuda") for _ in range(2))
    ks, vs = (torch.empty(k16.shape[:-1], dtype=torch.float16, device="cuda") for _ in range(2))
    rows = torch.arange(ks.numel() // hkv, dtype=torch.int32, device="cuda")
    store(k16.view(-1, hkv, 128), v16.view(-1, hkv, 128), kc, vc, ks, vs, rows)
    q, ctx, bt = to_dev(w["q"], bf), to_dev(w["context_lens"]), to_dev(w["block_tables"])
    a, b = torch.full_like(q, float("nan")), torch.full_like(q, float("nan"))
    decode(q, kc, vc, ks, vs, ctx, bt, hkv, 128, 256, w["scale"], a, _workspace(len(lens), hq, hkv, bt.shape[1], 256))
    decode(q, kc, vc, ks, vs, ctx, bt, hkv, 128, 256, w["scale"], b, None)
    ref = oracle.decode_attention_paged(w["q"], w["k_cache"], w["v_cache"], w["context_lens"], w["block_tables"], hkv, 128, 256, w["scale"])
    assert float((a.float() - b.float()).abs().max()) <= 1e-2
    assert np.abs(to_np(a) - ref).max() <= (5e-2 if fmt == "int8" else 2.5e-1) and not torch.isnan(b.float()).any()


@pytest.mark.parametrize("hq,hkv,bs,lens,table_blocks", [
    (24, 3, 48, EDGES[:7] + [700], 15),                     # clusters of four, eight heads a group, blocks and heads that are no power of two
    (3, 3, 48, [300, 47, 48, 49], 7),                       # of eight, one head a group
    (7, 7, 16, [1024, 513, 16], 64),                        # of four, more table entries than lanes
    (40, 5, 80, (EDGES * 4)[:45] + [2500, 3999], 50),       # chunks: groups of eight by warps of four heads
    (16, 8, 256, [9000, 300, 5000] + [40] * 34, 36),        # more than four parts: a warp per head
    (32, 4, 256, [4000, 2049] + [40] * 127, 33),            # the same as far as it goes (4128 rows: four heads a warp)
])
def test_parts_come_together_without_what_is_not_there(hq, hkv, bs, lens, table_blocks):
    """Every merge form; an infinity in V stays in its column: parts that do not exist add nothing, not even zero times infinity."""
    w = workloads().make_decode_workload(len(lens), hq, hkv, 128, bs, 0, 0, seed=len(lens) + hq, context_lens=np.array(lens, np.int32),
                                         pad_blocks_to=table_blocks)
    bf = torch.bfloat16
    q, kc, vc, ctx, bt = to_dev(w["q"], bf), to_dev(w["k_cache"], bf), to_dev(w["v_cache"], bf), to_dev(w["context_lens"]), to_dev(w["block_tables"])
    ref = oracle.decode_attention_paged(w["q"], w["k_cache"], w["v_cache"], w["context_lens"], w["block_tables"], hkv, 128, bs, w["scale"])
    for ws in (_workspace(len(lens), hq, hkv, bt.shape[1], bs), None):
        out = torch.full_like(q, float("nan"))
        nvk().launch_decode_attention_paged(q, kc, vc, ctx, bt, hkv, 128, bs, w["scale"], out, ws)
        assert_attention_close(to_np(out), ref)
    last = [int(w["block_tables"][i, (n - 1) // bs]) * bs + (n - 1) % bs for i, n in enumerate(lens) if n]
    vc.view(-1, hkv, 128)[torch.tensor(last, device="cuda"), :, 5] = float("inf")
    live = torch.tensor(lens, device="cuda") > 0
    for ws in (_workspace(len(lens), hq, hkv, bt.shape[1], bs), None):
        out = torch.full_like(q, float("nan"))
        nvk().launch_decode_attention_paged(q, kc, vc, ctx, bt, hkv, 128, bs, w["scale"], out, ws)
        assert bool((out[live][..., 5] == float("inf")).all())
        rest = torch.cat([out[..., :5], out[..., 6:]], -1)
        assert_attention_close(to_np(rest), np.concatenate([ref[..., :5], ref[..., 6:]], -1))


@pytest.mark.parametrize("kv,hq,hkv,bs,batch,table_blocks", [
    ("same", 8, 1, 256, 72, 3), ("same", 16, 8, 256, 18, 5), ("same", 6, 2, 48, 37, 43), ("same", 4, 4, 256, 37, 32),     # fewest and most pairs, odd and widest tables
    ("int8", 8, 1, 256, 105, 5), ("fp8", 4, 2, 64, 111, 24), ("int8", 8, 8, 256, 14, 8),
])
def test_halves_of_a_table_in_clusters_of_two(kv, hq, hkv, bs, batch, table_blocks):
    """Contexts that end in the first half, with it, in the second and with the table, and none."""
    half, full = (table_blocks + 1) // 2 * bs, table_blocks * bs
    edges = [0, 1, half - 1, half, half + 1, half + 17, full - 1, full]
    lens = [min(edges[i % 8], 3000) for i in range(batch)]
    w = workloads().make_decode_workload(batch, hq, hkv, 128, bs, 0, 0, seed=batch, context_lens=np.array(lens, np.int32), pad_blocks_to=table_blocks)
    bf, lib = torch.bfloat16, nvk()
    q, ctx, bt = to_dev(w["q"], bf), to_dev(w["context_lens"]), to_dev(w["block_tables"])
    kc, vc = to_dev(w["k_cache"], bf), to_dev(w["v_cache"], bf)
    ws, out = _workspace(batch, hq, hkv, bt.shape[1], bs), torch.full_like(q, float("nan"))
    if kv == "same":
        lib.launch_decode_attention_paged(q, kc, vc, ctx, bt, hkv, 128, bs, w["scale"], out, ws)
        k, v, tol = w["k_cache"], w["v_cache"], None
    else:
        store, decode = ((lib.store_kvcache_int8, lib.launch_decode_attention_paged_int8) if kv == "int8" else
                         (lib.store_kvcache_fp8, lib.launch_decode_attention_paged_fp8))
        k8, v8 = (torch.empty(kc.shape, dtype=torch.int8 if kv == "int8" else torch.uint8, device="cuda") for _ in range(2))
        ks, vs = (torch.empty(kc.shape[:-1], dtype=torch.float16, device="cuda") for _ in range(2))
        store(kc.view(-1, hkv, 128), vc.view(-1, hkv, 128), k8, v8, ks, vs, torch.arange(ks.numel() // hkv, dtype=torch.int32, device="cuda"))
        decode(q, k8, v8, ks, vs, ctx, bt, hkv, 128, bs, w["scale"], out, ws)
        plain = (lambda x: x.float()) if kv == "int8" else (lambda x: x.view(torch.float8_e4m3fn).float())
        k, v = ((plain(x) * s.float()[..., None]).cpu().numpy() for x, s in ((k8, ks), (v8, vs)))   # on the same quantised cache
    ref = oracle.decode_attention_paged(w["q"], k, v, w["context_lens"], w["block_tables"], hkv, 128, bs, w["scale"])
    assert_attention_close(to_np(out), ref)


@pytest.mark.parametrize("kv,hq,hkv,bs,batch,table_blocks", [
    ("same", 4, 1, 256, 149, 7), ("same", 8, 4, 64, 56, 41), ("same", 8, 1, 256, 295, 16), ("same", 4, 2, 256, 52, 12), ("same", 16, 8, 16, 10, 160),   # 1024- and 512-key chunks
    ("same", 4, 1, 256, 72, 9), ("same", 4, 1, 256, 103, 12), ("same", 6, 3, 48, 34, 43), ("same", 8, 8, 256, 18, 26), ("same", 2, 1, 256, 149, 6),   # beside halves; whole
    ("same", 6, 2, 48, 37, 41), ("same", 8, 8, 256, 18, 12), ("same", 4, 1, 16, 104, 192),                                                           # halves as far as they go
    ("int8", 4, 1, 256, 223, 4), ("fp8", 8, 1, 256, 240, 6), ("int8", 8, 8, 64, 30, 20), ("fp8", 4, 4, 256, 74, 5), ("int8", 2, 1, 256, 106, 7), ("fp8", 6, 1, 256, 223, 3),
])
def test_contexts_of_unequal_length_in_chunks(kv, hq, hkv, bs, batch, table_blocks):
    """Contexts that end at the edges of 256-, 512- and 1024-key chunks and with the table, among short and empty ones."""
    full = table_blocks * bs
    edges = [min(n, full) for n in (full, 5, 0, 511, 512, 17, 513, full - 1, 40, 1023, 1024, 1, 1025, 255, 257, 3)]
    lens = [edges[i % 16] for i in range(batch)]
    w = workloads().make_decode_workload(batch, hq, hkv, 128, bs, 0, 0, seed=batch + 1, context_lens=np.array(lens, np.int32), pad_blocks_to=table_blocks)
    bf, lib = torch.bfloat16, nvk()
    q, ctx, bt = to_dev(w["q"], bf), to_dev(w["context_lens"]), to_dev(w["block_tables"])
    kc, vc = to_dev(w["k_cache"], bf), to_dev(w["v_cache"], bf)
    ws, out = _workspace(batch, hq, hkv, bt.shape[1], bs), torch.full_like(q, float("nan"))
    if kv == "same":
        lib.launch_decode_attention_paged(q, kc, vc, ctx, bt, hkv, 128, bs, w["scale"], out, ws)
        k, v = w["k_cache"], w["v_cache"]
    else:
        store, decode = ((lib.store_kvcache_int8, lib.launch_decode_attention_paged_int8) if kv == "int8" else
                         (lib.store_kvcache_fp8, lib.launch_decode_attention_paged_fp8))
        k8, v8 = (torch.empty(kc.shape, dtype=torch.int8 if kv == "int8" else torch.uint8, device="cuda") for _ in range(2))
        ks, vs = (torch.empty(kc.shape[:-1], dtype=torch.float16, device="cuda") for _ in range(2))
        store(kc.view(-1, hkv, 128), vc.view(-1, hkv, 128), k8, v8, ks, vs, torch.arange(ks.numel() // hkv, dtype=torch.int32, device="cuda"))
        decode(q, k8, v8, ks, vs, ctx, bt, hkv, 128, bs, w["scale"], out, ws)
        plain = (lambda x: x.float()) if kv == "int8" else (lambda x: x.view(torch.float8_e4m3fn).float())
        k, v = ((plain(x) * s.float()[..., None]).cpu().numpy() for x, s in ((k8, ks), (v8, vs)))   # on the same quantised cache
    assert_attention_close(to_np(out), oracle.decode_attention_paged(w["q"], k, v, w["context_lens"], w["block_tables"], hkv, 128, bs, w["scale"]))
