"""fp32-arithmetic paged decode (clusters of blocks over a sequence's keys) at the edges of its tiling: contexts around a
warp's trip and a block's round of trips, every group remainder, cluster sizes 1 to 8, odd block sizes, ids outside the cache."""
import math

import numpy as np
import pytest

from util import nvk, to_dev, to_np, workloads

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _reference(w, hkv, bs):
    q, out = w["q"].astype(np.float64), np.zeros(w["q"].shape)
    d = q.shape[2]
    kc, vc = (np.concatenate([w[n].reshape(-1, hkv, d), np.zeros((1, hkv, d))]).astype(np.float64) for n in ("k_cache", "v_cache"))
    for b, n in enumerate(w["context_lens"]):
        pos = np.arange(max(int(n), 0))
        if not len(pos):
            continue
        rows = w["block_tables"][b, pos // bs].astype(np.int64) * bs + pos % bs
        rows[(rows < 0) | (rows >= len(kc) - 1)] = -1                    # ids outside the cache read as zeros
        for h in range(q.shape[1]):
            kv = h * hkv // q.shape[1]
            s = kc[rows, kv] @ q[b, h] * w["scale"]
            p = np.exp(s - s.max())
            out[b, h] = p @ vc[rows, kv] / p.sum()
    return out


@pytest.mark.parametrize("dtype,head_dim,block_size", [("f32", 128, 256), ("f32", 64, 16), ("f32", 256, 7), ("bf16", 64, 16), ("f16", 256, 3)])
@pytest.mark.parametrize("num_heads,num_kv_heads,batch", [(2, 2, 1), (6, 2, 5), (5, 1, 9), (8, 1, 3), (16, 8, 8), (4, 2, 160)])
def test_decode_simt_matches_a_float64_reference(dtype, head_dim, block_size, num_heads, num_kv_heads, batch):
    ctx = np.array(([0, 1, 7, 8, 9, 63, 64, 65, 127, 129, 300, 511, 513, 640] * 12)[:batch], np.int32)
    ctx[-1] = 641
    w = workloads().make_decode_workload(batch, num_heads, num_kv_heads, head_dim, block_size, 0, 0, seed=batch + head_dim, context_lens=ctx,
                                         value_scale=0.5, rounded=dtype != "f32")
    if dtype == "f16":
        for n in ("q", "k_cache", "v_cache"):
            w[n] = w[n].astype(np.float16).astype(np.float32)
    w["block_tables"][-1, 1] = w["k_cache"].shape[0] + 5
    td = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}[dtype]
    q = to_dev(w["q"], td)
    out = torch.full_like(q, float("nan"))
    nvk().launch_decode_attention_paged(q, to_dev(w["k_cache"], td), to_dev(w["v_cache"], td), to_dev(ctx), to_dev(w["block_tables"]), num_kv_heads,
                                        head_dim, block_size, w["scale"], out)
    err = np.abs(to_np(out) - _reference(w, num_kv_heads, block_size))
    assert err.max() <= (2e-6 if dtype == "f32" else 1e-2), err.max()
    assert math.isfinite(float(out.float().abs().max()))


@pytest.mark.parametrize("dtype,head_dim", [("f32", 128), ("f16", 64)])
@pytest.mark.parametrize("batch", [1, 6, 10, 20])   # 8 KV heads: clusters of 8, 4, 2 and 1
def test_infinite_values_stay_infinite(dtype, head_dim, batch):
    """A visible V row with infinities: these elements of the output are infinite with its sign, all others as without it."""
    ctx = np.array([(300, 77, 1000, 520, 64)[i % 5] for i in range(batch)], np.int32)
    w = workloads().make_decode_workload(batch, 16, 8, head_dim, 16, 0, 0, seed=batch, context_lens=ctx, value_scale=0.5)
    td = torch.float32 if dtype == "f32" else torch.float16
    for n in ("q", "k_cache", "v_cache"):
        w[n] = torch.from_numpy(w[n]).to(td).float().numpy()
    for b in range(batch):
        for pos, at, value in ((0, 3, np.inf), (int(ctx[b]) - 1, 5, -np.inf), (int(ctx[b]) // 2, head_dim - 1, np.inf)):
            w["v_cache"][w["block_tables"][b, pos // 16], pos % 16, b % 8, at] = value
    q = to_dev(w["q"], td)
    out = torch.full_like(q, float("nan"))
    nvk().launch_decode_attention_paged(q, to_dev(w["k_cache"], td), to_dev(w["v_cache"], td), to_dev(ctx), to_dev(w["block_tables"]), 8, head_dim, 16,
                                        w["scale"], out)
    ref, got = _reference(w, 8, 16), to_np(out)
    assert np.isinf(ref).sum() == 3 * 2 * batch
    assert np.array_equal(got[np.isinf(ref)], ref[np.isinf(ref)])
    assert np.abs(got[np.isfinite(ref)] - ref[np.isfinite(ref)]).max() <= (2e-6 if dtype == "f32" else 1e-2)


@pytest.mark.parametrize("dtype,head_dim,block_size", [("f32", 128, 256), ("f32", 64, 48), ("bf16", 256, 16)])
@pytest.mark.parametrize("num_heads,num_kv_heads,lens,keys", [
    (8, 2, [511, 3], 511), (8, 2, [512, 1, 0], 512),      # tables on both sides of where few clusters take blocks of eight warps
    (15, 15, [700], 768), (16, 16, [700], 768),           # as many clusters of those as fit, and one more
    (3, 1, [5000, 9], 5120),                              # rounds of a ring, more table entries than lanes
])
def test_decode_simt_block_sizes_and_keys_without_weight(dtype, head_dim, block_size, num_heads, num_kv_heads, lens, keys):
    ctx = np.array(lens, np.int32)
    w = workloads().make_decode_workload(len(lens), num_heads, num_kv_heads, head_dim, block_size, 0, 0, seed=len(lens) + head_dim, context_lens=ctx,
                                         value_scale=0.5, rounded=dtype != "f32", pad_blocks_to=-(-keys // block_size))
    td = {"f32": torch.float32, "bf16": torch.bfloat16}[dtype]
    w["q"] = np.abs(w["q"]) + 0.01 if dtype == "f32" else np.ones_like(w["q"])
    args = [to_dev(w["q"], td), to_dev(w["k_cache"], td), to_dev(w["v_cache"], td), to_dev(ctx), to_dev(w["block_tables"])]
    tail = (num_kv_heads, head_dim, block_size, w["scale"])
    out = torch.full_like(args[0], float("nan"))
    nvk().launch_decode_attention_paged(*args, *tail, out)
    err = np.abs(to_np(out) - _reference(w, num_kv_heads, block_size))
    assert err.max() <= (2e-6 if dtype == "f32" else 1e-2), err.max()
    # the first and a later key score minus infinity: no weight, nothing else changes
    for b, n in enumerate(lens):
        for key in {0, n // 2} if n > 2 else ():
            row = int(w["block_tables"][b, key // block_size]) * block_size + key % block_size
            w["k_cache"].reshape(-1, num_kv_heads, head_dim)[row] = -np.inf
    args[1] = to_dev(w["k_cache"], td)
    nvk().launch_decode_attention_paged(*args, *tail, out)
    err = np.abs(to_np(out) - _reference(w, num_kv_heads, block_size))
    assert err.max() <= (2e-6 if dtype == "f32" else 1e-2), err.max()


@pytest.mark.parametrize("dtype,head_dim", [("f32", 128), ("f32", 64), ("bf16", 256)])
@pytest.mark.parametrize("num_heads,num_kv_heads,batch,keys", [
    (4, 1, 15, 1024), (4, 1, 16, 1024), (4, 1, 18, 2304), (8, 1, 16, 1024), (4, 1, 34, 768), (4, 1, 55, 768), (4, 1, 56, 768), (4, 1, 75, 768), (4, 1, 112, 768),
    (3, 1, 149, 768), (4, 1, 223, 512), (4, 1, 223, 768), (4, 1, 297, 512), (4, 1, 1185, 768),                    # four heads: clusters of 8, 4, 2 and 1, of both kinds of blocks
    (2, 1, 33, 768), (2, 1, 34, 768), (1, 1, 297, 768), (2, 1, 297, 512), (2, 1, 445, 512),                      # one and two
])
def test_decode_simt_blocks_of_four_and_of_eight_warps(dtype, head_dim, num_heads, num_kv_heads, batch, keys):
    """Both sides of the lines between them; contexts around one and two steps of a block's warps, a few of them long; what was left in shared memory by
    others (infinities) does not matter."""
    per = 8 * 512 // head_dim                                            # keys of a step of eight warps
    ctx = np.array(([1, 0, per // 2, per - 1, per, per + 1, 2 * per - 1, 2 * per, 2 * per + 1, 3 * per, 5] * (batch // 11 + 1))[:batch], np.int32)
    ctx[0], ctx[-1] = keys, keys - 1
    w = workloads().make_decode_workload(batch, num_heads, num_kv_heads, head_dim, 256, 0, 0, seed=batch + head_dim, context_lens=ctx,
                                         value_scale=0.5, rounded=dtype != "f32")
    td = {"f32": torch.float32, "bf16": torch.bfloat16}[dtype]
    q, kc, vc, lens, bt = to_dev(w["q"], td), to_dev(w["k_cache"], td), to_dev(w["v_cache"], td), to_dev(ctx), to_dev(w["block_tables"])
    out = torch.full_like(q, float("nan"))
    inf = torch.full_like(vc, float("inf"))
    nvk().launch_decode_attention_paged(q, kc, inf, lens, bt, num_kv_heads, head_dim, 256, w["scale"], out)
    out.fill_(float("nan"))
    nvk().launch_decode_attention_paged(q, kc, vc, lens, bt, num_kv_heads, head_dim, 256, w["scale"], out)
    err = np.abs(to_np(out) - _reference(w, num_kv_heads, 256))
    assert err.max() <= (2e-6 if dtype == "f32" else 1e-2), err.max()
