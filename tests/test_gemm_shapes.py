"""The linears at the edges of their two kernels' tilings: parts of K in clusters of 1, 2, 4 and 8 blocks, one and two row tiles, pairs of
blocks with one and with several tiles, a last column tile of half width, remainders of rows and of K."""
import numpy as np
import pytest

import oracle
from util import nvk, to_dev, to_np, workloads

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,out_features,in_features", [
    (1, 128, 8), (8, 768, 4096), (9, 768, 1032), (64, 4096, 1024), (128, 6144, 520), (129, 768, 4096), (200, 6144, 512), (256, 2048, 2048),
    (257, 4096, 512), (500, 6144, 512), (513, 9472, 128), (1030, 1408, 264), (3000, 384, 2048), (5000, 4096, 72),
    (32, 4096, 128), (33, 4096, 128), (97, 12288, 256), (161, 6144, 256), (700, 512, 64),          # blocks with all of K, few rows and many
])
def test_linear_at_tile_edges(dtype, rows, out_features, in_features):
    gen = torch.Generator(device="cuda").manual_seed(rows + out_features)
    x = torch.randn((rows, in_features), generator=gen, device="cuda").to(dtype)
    w = (torch.randn((out_features, in_features), generator=gen, device="cuda") / in_features ** 0.5).to(dtype)
    guard = torch.full((rows + 1, out_features), float("nan"), device="cuda", dtype=dtype)
    nvk().linear(x, w, guard[:rows])
    torch.cuda.synchronize()
    assert nvk().gemm_status() == 0
    want = x.float() @ w.float().t()
    err = (guard[:rows].float() - want).abs()
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert bool((err <= want.abs().clamp_min(0.05) * 2 * ulp + 1e-3).all()), float(err.max())
    assert bool(torch.isnan(guard[rows].float()).all())          # nothing past the last row


@pytest.mark.parametrize("num_q_heads,num_kv_heads,rows,hidden", [(4, 1, 3, 2048), (32, 8, 200, 512), (16, 8, 700, 1024), (6, 3, 2100, 256), (32, 8, 1500, 128)])
def test_qkv_prologue_at_tile_edges(num_q_heads, num_kv_heads, rows, hidden):
    bf, d, max_pos, heads = torch.bfloat16, 128, 400, num_q_heads + 2 * num_kv_heads
    gen = torch.Generator(device="cuda").manual_seed(heads + rows)
    x = torch.randn((rows, hidden), generator=gen, device="cuda").to(bf)
    w = (torch.randn((heads * d, hidden), generator=gen, device="cuda") / hidden ** 0.5).to(bf)
    cache_rows = rows + 100
    pw = workloads().make_prologue_workload(rows, num_q_heads, num_kv_heads, d, cache_rows, max_pos, seed=rows)
    pw["slot_mapping"][rows // 2] = -1
    pw["positions"][0] = max_pos
    table = oracle.build_cos_sin_cache(max_pos, d, pw["rope_base"])
    kc = torch.zeros(cache_rows, num_kv_heads, d, dtype=bf, device="cuda")
    vc, q_out = torch.zeros_like(kc), torch.full((rows, num_q_heads, d), float("nan"), dtype=bf, device="cuda")
    nvk().qkv_linear_norm_rope_store(x, w, to_dev(pw["positions"]), to_dev(pw["q_norm_weight"], bf), to_dev(pw["k_norm_weight"], bf), pw["eps"],
                                     to_dev(table), to_dev(pw["slot_mapping"]), kc, vc, num_q_heads, num_kv_heads, d, q_out)
    qkv = torch.empty((rows, heads * d), dtype=bf, device="cuda")
    nvk().linear(x, w, qkv)
    torch.cuda.synchronize()
    assert nvk().gemm_status() == 0
    kc_ref, vc_ref = np.zeros((cache_rows, num_kv_heads, d), np.float32), np.zeros((cache_rows, num_kv_heads, d), np.float32)
    q_ref = oracle.fused_split_norm_rope_store(to_np(qkv), pw["positions"], pw["q_norm_weight"], pw["k_norm_weight"], pw["eps"], table,
                                               pw["slot_mapping"], kc_ref, vc_ref, num_q_heads, num_kv_heads, d)
    assert np.array_equal(to_np(vc), vc_ref)                      # V: the rounded product, copied
    for got, ref in ((to_np(q_out), q_ref), (to_np(kc), kc_ref)):
        assert (np.abs(got - ref) <= np.maximum(np.abs(ref), 1e-3) * 2.0 ** -7).all()


@pytest.mark.parametrize("rows,hidden", [(37, 2048), (200, 512), (700, 1024)])     # summed over a cluster, a block each, pairs
def test_qkv_prologue_takes_a_rotary_table_at_any_address(rows, hidden):
    bf, d, hq, hkv = torch.bfloat16, 128, 16, 8
    gen = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn((rows, hidden), generator=gen, device="cuda").to(bf)
    w = (torch.randn(((hq + 2 * hkv) * d, hidden), generator=gen, device="cuda") / hidden ** 0.5).to(bf)
    table, norm = to_dev(oracle.build_cos_sin_cache(rows, d, 1e6)), torch.ones(d, dtype=bf, device="cuda")
    pos = torch.arange(rows, dtype=torch.int32, device="cuda")
    flat = torch.zeros(table.numel() + 4, device="cuda")
    got = []
    for offset in (0, 1, 2):
        t = flat[offset:offset + table.numel()].view(rows, d)
        t.copy_(table)
        out = [torch.full((rows, h, d), float("nan"), dtype=bf, device="cuda") for h in (hq, hkv, hkv)]
        nvk().qkv_linear_norm_rope_store(x, w, pos, norm, norm, 1e-6, t, pos, out[1], out[2], hq, hkv, d, out[0])
        got.append(out)
    torch.cuda.synchronize()
    assert nvk().gemm_status() == 0
    for o in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(o, got[0])) and not any(torch.isnan(a.float()).any() for a in o)


@pytest.mark.parametrize("rows,hidden", [(37, 2048), (200, 512), (700, 1024)])     # summed over a cluster, a block each, pairs
def test_rows_of_a_warp_that_go_different_ways(rows, hidden):
    """Neighbouring rows with and without a slot, with and without a rotary row: each comes out as in a call where all rows are alike."""
    bf, d, hq, hkv = torch.bfloat16, 128, 16, 8
    gen = torch.Generator(device="cuda").manual_seed(rows + 1)
    x = torch.randn((rows, hidden), generator=gen, device="cuda").to(bf)
    w = (torch.randn(((hq + 2 * hkv) * d, hidden), generator=gen, device="cuda") / hidden ** 0.5).to(bf)
    table, norm = to_dev(oracle.build_cos_sin_cache(rows, d, 1e6)), torch.ones(d, dtype=bf, device="cuda")
    every = torch.arange(rows, dtype=torch.int32, device="cuda")

    def run(pos, slots):
        q, k, v = (torch.zeros((rows, h, d), dtype=bf, device="cuda") for h in (hq, hkv, hkv))
        nvk().qkv_linear_norm_rope_store(x, w, pos, norm, norm, 1e-6, table, slots, k, v, hq, hkv, d, q)
        return q, k, v

    turned, plain = run(every, every), run(torch.full_like(every, rows), every)
    slot, rope = every % 2 == 0, every % 3 != 0
    q, k, v = run(torch.where(rope, every, rows + 5), torch.where(slot, every, -1))
    torch.cuda.synchronize()
    assert nvk().gemm_status() == 0
    pick = rope[:, None, None]
    assert torch.equal(q, torch.where(pick, turned[0], plain[0]))
    assert torch.equal(k, torch.where(pick, turned[1], plain[1]) * slot[:, None, None])
    assert torch.equal(v, turned[2] * slot[:, None, None])


@pytest.mark.parametrize("num_q_heads,num_kv_heads,hidden", [(4, 1, 2048), (8, 2, 512), (24, 4, 1024), (32, 8, 640)])   # clusters of 8, 4, 4 and 2
@pytest.mark.parametrize("rows", [1, 31, 33, 57, 64, 65, 121, 128, 129, 250])                # runs of rows, with and without the ring's last stage
def test_sums_pushed_through_a_cluster(num_q_heads, num_kv_heads, hidden, rows):
    """Plain products against fp32, and with norm, rotation and store against the oracle on that product; without norm weights and slots as well."""
    bf, d, max_pos, heads = torch.bfloat16, 128, 300, num_q_heads + 2 * num_kv_heads
    gen = torch.Generator(device="cuda").manual_seed(heads * rows)
    x = torch.randn((rows, hidden), generator=gen, device="cuda").to(bf)
    w = (torch.randn((heads * d, hidden), generator=gen, device="cuda") / hidden ** 0.5).to(bf)
    qkv = torch.full((rows, heads * d), float("nan"), dtype=bf, device="cuda")
    nvk().linear(x, w, qkv)
    want = x.float() @ w.float().t()
    err = (qkv.float() - want).abs()                                # half a unit of the result, and the order of the sums
    assert bool((err <= want.abs().clamp_min(0.05) * 2.0 ** -8 + 1e-3).all()), float(err.max())
    cache_rows = rows + 10
    pw = workloads().make_prologue_workload(rows, num_q_heads, num_kv_heads, d, cache_rows, max_pos, seed=rows)
    pw["slot_mapping"][rows // 2] = -1
    pw["positions"][rows // 3] = max_pos
    table = oracle.build_cos_sin_cache(max_pos, d, pw["rope_base"])
    for normed in (True, False):
        qw, kw = (pw["q_norm_weight"], pw["k_norm_weight"]) if normed else (None, None)
        slots = pw["slot_mapping"] if normed else np.arange(rows, dtype=np.int32)
        kc = torch.zeros(cache_rows, num_kv_heads, d, dtype=bf, device="cuda")
        vc, q_out = torch.zeros_like(kc), torch.full((rows, num_q_heads, d), float("nan"), dtype=bf, device="cuda")
        nvk().qkv_linear_norm_rope_store(x, w, to_dev(pw["positions"]), to_dev(qw, bf) if normed else None, to_dev(kw, bf) if normed else None, pw["eps"],
                                         to_dev(table), to_dev(slots) if normed else None, kc, vc, num_q_heads, num_kv_heads, d, q_out)
        torch.cuda.synchronize()
        assert nvk().gemm_status() == 0
        if normed:
            kc_ref, vc_ref = np.zeros((cache_rows, num_kv_heads, d), np.float32), np.zeros((cache_rows, num_kv_heads, d), np.float32)
            q_ref = oracle.fused_split_norm_rope_store(to_np(qkv), pw["positions"], qw, kw, pw["eps"], table, slots, kc_ref, vc_ref, num_q_heads, num_kv_heads, d)
        else:
            parts = to_np(qkv).reshape(rows, heads, d)
            inside = (pw["positions"] >= 0) & (pw["positions"] < max_pos)
            t = table[np.where(inside, pw["positions"], 0)][:, None]
            lo, hi, cs, sn = parts[..., :64], parts[..., 64:], t[..., :64], t[..., 64:]
            turned = np.where(inside[:, None, None], np.concatenate([lo * cs - hi * sn, hi * cs + lo * sn], -1), parts)
            q_ref = turned[:, :num_q_heads]
            kc_ref, vc_ref = np.zeros((cache_rows, num_kv_heads, d), np.float32), np.zeros((cache_rows, num_kv_heads, d), np.float32)
            kc_ref[:rows], vc_ref[:rows] = turned[:, num_q_heads:num_q_heads + num_kv_heads], parts[:, num_q_heads + num_kv_heads:]
        assert np.array_equal(to_np(vc), vc_ref)
        for got, ref in ((to_np(q_out), q_ref), (to_np(kc), kc_ref)):
            assert (np.abs(got - ref) <= np.maximum(np.abs(ref), 1e-3) * 2.0 ** -7 + 2.0 ** -9 * (not normed)).all()   # (cancelling terms of a rotation, 16-bit inputs)


@pytest.mark.parametrize("normed", [True, False])
@pytest.mark.parametrize("num_q_heads,num_kv_heads,hidden", [(32, 8, 4096), (32, 8, 3080), (16, 8, 4096)])   # pairs with several tiles each, and one or two
def test_qkv_prologue_of_many_rows_does_not_depend_on_the_place_of_a_row(num_q_heads, num_kv_heads, hidden, normed):
    """Large K: a pair's tiles but the last finish under the next one's MMAs, in a form of their own.  Equal rows have equal bits in all tiles, and the
    first ones are what the oracle makes of the product."""
    dt, d, max_pos, heads, rows, period = torch.float16, 128, 300, num_q_heads + 2 * num_kv_heads, 1900, 256
    gen = torch.Generator(device="cuda").manual_seed(heads + hidden)
    at = torch.arange(rows, device="cuda") % period
    x = torch.randn((period, hidden), generator=gen, device="cuda").to(dt)[at].contiguous()
    w = (torch.randn((heads * d, hidden), generator=gen, device="cuda") / hidden ** 0.5).to(dt)
    pw = workloads().make_prologue_workload(rows, num_q_heads, num_kv_heads, d, rows, max_pos, seed=hidden)
    table = oracle.build_cos_sin_cache(max_pos, d, pw["rope_base"])
    pos, slots = np.arange(rows) % period + 20, np.arange(rows)[::-1].copy()
    pos[7::period], slots[rows // 2] = max_pos, -1                       # outside the table; not stored
    pos, slots = pos.astype(np.int32), slots.astype(np.int32)
    qw, kw = ((1 + 0.1 * torch.randn(d, generator=gen, device="cuda")).to(dt) for _ in range(2))
    q = torch.full((rows, num_q_heads, d), float("nan"), dtype=dt, device="cuda")
    kc, vc = (torch.zeros((rows, num_kv_heads, d), dtype=dt, device="cuda") for _ in range(2))
    nvk().qkv_linear_norm_rope_store(x, w, to_dev(pos), qw if normed else None, kw if normed else None, pw["eps"], to_dev(table), to_dev(slots), kc, vc,
                                     num_q_heads, num_kv_heads, d, q)
    qkv = torch.empty((rows, heads * d), dtype=dt, device="cuda")
    nvk().linear(x, w, qkv)
    torch.cuda.synchronize()
    assert nvk().gemm_status() == 0
    k, v = kc.flip(0), vc.flip(0)                                        # in the order of the rows
    stored = torch.ones(rows, dtype=torch.bool, device="cuda")
    stored[rows // 2] = False
    assert bool((k[rows // 2] == 0).all()) and bool((v[rows // 2] == 0).all())
    assert torch.equal(q, q[at]) and torch.equal(k[stored], k[at][stored]) and torch.equal(v[stored], v[at][stored])
    n = period
    if normed:
        kc_ref, vc_ref = np.zeros((n, num_kv_heads, d), np.float32), np.zeros((n, num_kv_heads, d), np.float32)
        q_ref = oracle.fused_split_norm_rope_store(to_np(qkv[:n]), pos[:n], to_np(qw), to_np(kw), pw["eps"], table, np.arange(n, dtype=np.int32), kc_ref, vc_ref,
                                                   num_q_heads, num_kv_heads, d, oracle.ROUND_NONE)
    else:
        parts = to_np(qkv[:n]).reshape(n, heads, d)
        inside = pos[:n] < max_pos
        t = table[np.where(inside, pos[:n], 0)][:, None]
        lo, hi, cs, sn = parts[..., :64], parts[..., 64:], t[..., :64], t[..., 64:]
        turned = np.where(inside[:, None, None], np.concatenate([lo * cs - hi * sn, hi * cs + lo * sn], -1), parts)
        q_ref, kc_ref, vc_ref = turned[:, :num_q_heads], turned[:, num_q_heads:num_q_heads + num_kv_heads], parts[:, num_q_heads + num_kv_heads:]
    assert np.array_equal(to_np(v[:n]), vc_ref)
    for got, ref in ((to_np(q[:n]), q_ref), (to_np(k[:n]), kc_ref)):
        # half a unit of an fp16 result and the fp32 steps before it; where a rotation's terms cancel, those of the terms (at most some 6)
        assert (np.abs(got - ref) <= np.abs(ref) * 2.0 ** -10 + 2.0 ** -18).all(), np.abs(got - ref).max()
