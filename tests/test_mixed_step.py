"""A continuous-batching step with prefill rows AND decode rows as one launch (``nvk_attention_mixed_step``): the
prefill rows against the oracle's paged / dense prefill, the decode rows against the oracle's paged decode, and both
bit for bit against the two single-purpose entry points (same kernels' arithmetic, same split policy), for several
divisions of the SMs between the two kinds of work and for int64 index tensors."""
import numpy as np
import pytest

import oracle
from util import assert_attention_close, nvk, to_dev, to_np, workloads

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

HQ, HKV, D, BS = 8, 2, 128, 256


def _case(paged, seed):
    wl = workloads()
    rng = np.random.default_rng(seed)
    # prefill part
    q_lens, prefix = ([300, 70, 129], [256, 0, 512]) if paged else ([200, 65, 130], [0, 0, 0])
    p = wl.make_prefill_workload(q_lens, prefix, HQ, HKV, D, BS, seed=seed, paged=paged)
    # decode part: its own sequences, in the same cache when the prefill part is paged
    ctx = rng.integers(1, 3000, size=9).astype(np.int32)
    ctx[3] = 0                                                        # an inactive row of a padded batch
    d = wl.make_decode_workload(len(ctx), HQ, HKV, D, BS, 0, 0, seed=seed + 1, context_lens=ctx, pad_blocks_to=14)
    if paged:   # one pool: decode blocks first, prefill blocks shifted behind them
        shift = d["k_cache"].shape[0]
        k_cache = np.concatenate([d["k_cache"], p["k_cache"]])
        v_cache = np.concatenate([d["v_cache"], p["v_cache"]])
        p_tables = (p["block_tables"] + shift).astype(np.int32)
    else:
        k_cache, v_cache, p_tables = d["k_cache"], d["v_cache"], None
    return p, d, k_cache, v_cache, p_tables


@pytest.mark.parametrize("paged", [True, False])
@pytest.mark.parametrize("prefill_blocks", [0, 1, 40, 1000])
def test_mixed_step_matches_oracle_and_the_two_single_purpose_calls(paged, prefill_blocks):
    bf = torch.bfloat16
    p, d, k_cache, v_cache, p_tables = _case(paged, seed=50 + prefill_blocks % 7)
    lib = nvk()
    kc, vc = to_dev(k_cache, bf), to_dev(v_cache, bf)
    pq, dq = to_dev(p["q"], bf), to_dev(d["q"], bf)
    cu_q, cu_k = to_dev(p["cu_q"]), to_dev(p["cu_k"])
    pt = to_dev(p_tables) if paged else None
    pk = None if paged else to_dev(p["k"], bf)
    pv = None if paged else to_dev(p["v"], bf)
    ctx, dt = to_dev(d["context_lens"]), to_dev(d["block_tables"])
    ws = torch.empty(max(16, lib.decode_attention_workspace_bytes(dq.shape[0], HQ, HKV, D, dt.shape[1], BS)), dtype=torch.uint8, device="cuda")
    p_out, d_out = torch.full_like(pq, float("nan")), torch.full_like(dq, float("nan"))
    lib.attention_mixed_step(pq, cu_q, pk, pv, cu_k, pt, p_out, dq, ctx, dt, d_out, kc, vc, HKV, D, BS, p["scale"], ws, prefill_blocks)
    torch.cuda.synchronize()
    assert lib.prefill_status() == 0
    assert not torch.isnan(p_out.float()).any() and not torch.isnan(d_out.float()).any()
    # the oracle
    if paged:
        want_p = oracle.prefill_attention_paged(p["q"], k_cache, v_cache, p["cu_q"], p["cu_k"], p_tables, HKV, D, BS, p["scale"])
    else:
        want_p = oracle.prefill_attention_dense(p["q"], p["k"], p["v"], p["cu_q"], p["cu_k"], HKV, D, p["scale"])
    want_d = oracle.decode_attention_paged(d["q"], k_cache, v_cache, d["context_lens"], d["block_tables"], HKV, D, BS, d["scale"])
    assert_attention_close(to_np(p_out), want_p)
    assert_attention_close(to_np(d_out), want_d)
    assert not to_np(d_out)[3].any()                                   # the inactive row is zeros
    # the single-purpose entry points
    p_ref, d_ref = torch.empty_like(pq), torch.empty_like(dq)
    if paged:
        lib.launch_prefill_attention_paged(pq, cu_q, kc, vc, cu_k, pt, HKV, D, BS, p["scale"], p_ref)
    else:
        lib.launch_prefill_attention_dense(pq, cu_q, pk, pv, cu_k, HKV, D, p["scale"], p_ref)
    lib.launch_decode_attention_paged(dq, kc, vc, ctx, dt, HKV, D, BS, d["scale"], d_ref, ws)
    torch.cuda.synchronize()
    assert torch.equal(p_out, p_ref)
    assert torch.equal(d_out, d_ref)


def test_mixed_step_repeats_with_int64_indices_and_from_a_graph():
    bf = torch.bfloat16
    p, d, k_cache, v_cache, p_tables = _case(True, seed=61)
    lib = nvk()
    L = torch.int64
    kc, vc = to_dev(k_cache, bf), to_dev(v_cache, bf)
    pq, dq = to_dev(p["q"], bf), to_dev(d["q"], bf)
    cu_q, cu_k, pt = to_dev(p["cu_q"]).to(L), to_dev(p["cu_k"]), to_dev(p_tables).to(L)
    ctx, dt = to_dev(d["context_lens"]).to(L), to_dev(d["block_tables"])
    ws = torch.empty(max(16, lib.decode_attention_workspace_bytes(dq.shape[0], HQ, HKV, D, dt.shape[1], BS)), dtype=torch.uint8, device="cuda")
    outs = []

    def step(p_out, d_out):
        lib.attention_mixed_step(pq, cu_q, None, None, cu_k, pt, p_out, dq, ctx, dt, d_out, kc, vc, HKV, D, BS, p["scale"], ws, 30)

    for _ in range(3):                                                 # the ticket counters re-arm between launches
        o = (torch.full_like(pq, float("nan")), torch.full_like(dq, float("nan")))
        step(*o)
        outs.append(o)
    torch.cuda.synchronize()
    gp, gd = torch.empty_like(pq), torch.empty_like(dq)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step(gp, gd)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step(gp, gd)
    for _ in range(2):
        gp.fill_(float("nan"))
        gd.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(gp, outs[0][0]) and torch.equal(gd, outs[0][1])
    for o in outs[1:]:
        assert torch.equal(o[0], outs[0][0]) and torch.equal(o[1], outs[0][1])
    assert lib.prefill_status() == 0


def _fp32_rows(q, k, v, scale, seen):
    """Attention of q [rows, heads, d] over the keys of one sequence in fp32; row r sees the first seen[r] keys."""
    group = q.shape[1] // k.shape[1]
    k, v = k.float().repeat_interleave(group, 1), v.float().repeat_interleave(group, 1)
    s = torch.einsum("qhd,khd->hqk", q.float(), k) * scale
    s.masked_fill_(torch.arange(k.shape[0], device="cuda")[None, None, :] >= seen[None, :, None], float("-inf"))
    return torch.einsum("hqk,khd->qhd", s.softmax(-1), v)


def test_two_hundred_steps_of_many_items_a_block_are_each_the_two_calls_bit_for_bit():
    """3 prompts of 500 to 2048 tokens beside 90 decode rows of 500 to 8192 keys, 32 / 8 heads: several items for every block, so that the
    warps of a block are items apart (an output row staged where a faster warp writes showed in one pass of seven, by up to 7)."""
    bf, lib, hq, hkv, scale = torch.bfloat16, nvk(), 32, 8, D ** -0.5
    gen = torch.Generator(device="cuda").manual_seed(5)
    rng = np.random.default_rng(5)
    q_lens, ctx_lens = np.array([1210, 500, 2048]), rng.permutation(np.linspace(500, 8192, 90).astype(np.int64))
    need = [-(-int(n) // BS) for n in (*q_lens, *ctx_lens)]
    ids, at = rng.permutation(sum(need)), 0
    pt, dt = np.zeros((3, max(need[:3])), np.int32), np.zeros((90, max(need[3:])), np.int32)
    for i, n in enumerate(need):
        (pt[i] if i < 3 else dt[i - 3])[:n] = ids[at:at + n]
        at += n

    def normal(*shape):
        return torch.empty(shape, dtype=bf, device="cuda").normal_(generator=gen)

    kc, vc = normal(sum(need), BS, hkv, D), normal(sum(need), BS, hkv, D)
    pq, dq = normal(int(q_lens.sum()), hq, D), normal(90, hq, D)
    cu, ctx, pt, dt = (to_dev(a.astype(np.int32)) for a in (np.concatenate([[0], np.cumsum(q_lens)]), ctx_lens, pt, dt))
    ws = torch.empty(lib.decode_attention_workspace_bytes(90, hq, hkv, D, dt.shape[1], BS), dtype=torch.uint8, device="cuda")
    want_p, want_d, p_out, d_out = torch.empty_like(pq), torch.empty_like(dq), torch.empty_like(pq), torch.empty_like(dq)
    lib.launch_prefill_attention_paged(pq, cu, kc, vc, cu, pt, hkv, D, BS, scale, want_p)
    lib.launch_decode_attention_paged(dq, kc, vc, ctx, dt, hkv, D, BS, scale, want_d, ws)
    for i in range(3):                                                 # the two calls against fp32
        n, r0 = int(q_lens[i]), int(q_lens[:i].sum())
        k, v = (c[pt[i, :need[i]].long()].view(-1, hkv, D)[:n] for c in (kc, vc))
        ref = _fp32_rows(pq[r0:r0 + n], k, v, scale, torch.arange(1, n + 1, device="cuda"))
        assert_attention_close(to_np(want_p[r0:r0 + n]), to_np(ref))
    for i in range(90):
        n = int(ctx_lens[i])
        k, v = (c[dt[i, :need[3 + i]].long()].view(-1, hkv, D)[:n] for c in (kc, vc))
        assert_attention_close(to_np(want_d[i:i + 1]), to_np(_fp32_rows(dq[i:i + 1], k, v, scale, torch.tensor([n], device="cuda"))))
    wrong = torch.zeros(200, dtype=torch.bool, device="cuda")
    for i in range(200):
        p_out.fill_(float("nan"))
        d_out.fill_(float("nan"))
        lib.attention_mixed_step(pq, cu, None, None, cu, pt, p_out, dq, ctx, dt, d_out, kc, vc, hkv, D, BS, scale, ws, (0, 0, 0, 1, 60, 148)[i % 6])
        wrong[i] = (p_out.view(torch.int16) != want_p.view(torch.int16)).any() | (d_out.view(torch.int16) != want_d.view(torch.int16)).any()
    assert lib.prefill_status() == 0
    assert not wrong.any(), wrong.nonzero().flatten().tolist()


def test_mixed_step_refuses_what_it_cannot_run():
    lib = nvk()
    f32 = torch.float32
    q = torch.zeros(4, 2, 128, device="cuda", dtype=f32)
    kc = torch.zeros(1, 256, 2, 128, device="cuda", dtype=f32)
    cu = torch.tensor([0, 4], device="cuda", dtype=torch.int32)
    ws = torch.zeros(1 << 20, device="cuda", dtype=torch.uint8)
    with pytest.raises(ValueError):                                    # fp32 takes the general paths: two calls
        lib.attention_mixed_step(q, cu, q, q, cu, None, q.clone(), q[:1], torch.ones(1, device="cuda", dtype=torch.int32),
                                 torch.zeros(1, 1, device="cuda", dtype=torch.int32), q[:1].clone(), kc, kc, 2, 128, 256, 0.1, ws, 0)


@pytest.mark.parametrize("batch,longest", [(4, 300), (40, 3000)])   # decode in clusters of blocks, and in chunks with a merge
def test_a_small_prefill_beside_decode_is_done_when_the_next_kernel_starts(batch, longest):
    """The two halves run side by side; a kernel queued right behind them sees both results, every time, eager and replayed."""
    wl, lib, bf = workloads(), nvk(), torch.bfloat16
    p = wl.make_prefill_workload([300], [0], 4, 1, 128, 256, seed=9, paged=True)
    ctx = np.linspace(1, longest, batch).astype(np.int32)
    d = wl.make_decode_workload(batch, 4, 1, 128, 256, 0, 0, seed=10, context_lens=ctx)
    shift = d["k_cache"].shape[0]
    kc, vc = (to_dev(np.concatenate([d[n], p[n]]), bf) for n in ("k_cache", "v_cache"))
    pq, dq, cu_q, cu_k, pt, cl, dt = (to_dev(p["q"], bf), to_dev(d["q"], bf), to_dev(p["cu_q"]), to_dev(p["cu_k"]),
                                      to_dev((p["block_tables"] + shift).astype(np.int32)), to_dev(ctx), to_dev(d["block_tables"]))
    ws = torch.empty(max(16, lib.decode_attention_workspace_bytes(batch, 4, 1, 128, dt.shape[1], 256)), dtype=torch.uint8, device="cuda")
    p_ref, d_ref = torch.empty_like(pq), torch.empty_like(dq)
    lib.launch_prefill_attention_paged(pq, cu_q, kc, vc, cu_k, pt, 1, 128, 256, p["scale"], p_ref)
    lib.launch_decode_attention_paged(dq, kc, vc, cl, dt, 1, 128, 256, d["scale"], d_ref, ws)
    p_out, d_out = torch.empty_like(pq), torch.empty_like(dq)
    right = torch.ones((), dtype=torch.bool, device="cuda")

    def step():
        p_out.fill_(float("nan"))
        d_out.fill_(float("nan"))
        lib.attention_mixed_step(pq, cu_q, None, None, cu_k, pt, p_out, dq, cl, dt, d_out, kc, vc, 1, 128, 256, p["scale"], ws)
        right.logical_and_((p_out == p_ref).all())
        right.logical_and_((d_out == d_ref).all())

    for _ in range(100):
        step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
        step()
    for _ in range(50):
        graph.replay()
    torch.cuda.synchronize()
    assert lib.prefill_status() == 0 and bool(right)


def test_a_small_prefill_beside_more_decode_rows_than_a_grid_has_room_for():
    """70000 decode rows of at most one key: one launch, as for any prefill part; with a scale that is not positive refused, and nothing written."""
    lib, bf, rows = nvk(), torch.bfloat16, 70000
    p = workloads().make_prefill_workload([10], [0], 2, 1, 128, 256, seed=3, paged=True)
    kc, vc, pq, cu, pt = to_dev(p["k_cache"], bf), to_dev(p["v_cache"], bf), to_dev(p["q"], bf), to_dev(p["cu_q"]), to_dev(p["block_tables"])
    dq = torch.ones((rows, 2, 128), dtype=bf, device="cuda")
    ctx = torch.arange(rows, dtype=torch.int32, device="cuda") % 2
    dt = torch.full((rows, 1), int(p["block_tables"][0, 0]), dtype=torch.int32, device="cuda")
    ws = torch.empty(max(16, lib.decode_attention_workspace_bytes(rows, 2, 1, 128, 1, 256)), dtype=torch.uint8, device="cuda")
    p_out, d_out = torch.full_like(pq, 7.0), torch.full_like(dq, 7.0)
    with pytest.raises(ValueError):
        lib.attention_mixed_step(pq, cu, None, None, cu, pt, p_out, dq, ctx, dt, d_out, kc, vc, 1, 128, 256, -p["scale"], ws)
    torch.cuda.synchronize()
    assert bool((p_out == 7.0).all()) and bool((d_out == 7.0).all())
    lib.attention_mixed_step(pq, cu, None, None, cu, pt, p_out, dq, ctx, dt, d_out, kc, vc, 1, 128, 256, p["scale"], ws)
    torch.cuda.synchronize()
    assert lib.prefill_status() == 0
    assert_attention_close(to_np(p_out), oracle.prefill_attention_paged(p["q"], p["k_cache"], p["v_cache"], p["cu_q"], p["cu_k"], p["block_tables"], 1, 128, 256,
                                                                        p["scale"]))
    first = vc[int(p["block_tables"][0, 0]), 0]                            # [1, 128]: a row of one key is that key's value
    assert torch.equal(d_out, (first * ctx[:, None, None].to(bf)).expand_as(d_out))
