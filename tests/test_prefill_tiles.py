"""The persistent tensor-core prefill at the edges of its tiles: every way to share a tile's 128 rows between query rows and heads, lengths
around a tile's query rows and around half and whole key tiles, results that start on a 16-byte boundary only, and whatever lies in the cache
behind a sequence's last key."""
import numpy as np
import pytest

import oracle
from util import assert_attention_close, nvk, to_dev, to_np, workloads

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _run(w, hkv, paged, scale, out=None, dtype=torch.bfloat16, tables=None, kc=None, vc=None):
    lib = nvk()
    q, cu_q, cu_k = to_dev(w["q"], dtype), to_dev(w["cu_q"]), to_dev(w["cu_k"])
    if out is None:
        out = torch.full_like(q, float("nan"))
    if paged:
        lib.launch_prefill_attention_paged(q, cu_q, kc if kc is not None else to_dev(w["k_cache"], dtype), vc if vc is not None else to_dev(w["v_cache"], dtype),
                                           cu_k, to_dev(w["block_tables"]), hkv, 128, 256, scale, out)
        ref = oracle.prefill_attention_paged(w["q"], w["k_cache"], w["v_cache"], w["cu_q"], w["cu_k"], w["block_tables"], hkv, 128, 256, scale)
    else:
        lib.launch_prefill_attention_dense(q, cu_q, to_dev(w["k"], dtype), to_dev(w["v"], dtype), cu_k, hkv, 128, scale, out)
        ref = oracle.prefill_attention_dense(w["q"], w["k"], w["v"], w["cu_q"], w["cu_k"], hkv, 128, scale)
    torch.cuda.synchronize()
    assert lib.prefill_status() == 0
    return out, ref


@pytest.mark.parametrize("hq,hkv", [(2, 1), (4, 1), (6, 1), (8, 1), (16, 1), (24, 2), (4, 2)])
@pytest.mark.parametrize("q_lens,prefix,paged", [
    ([1, 15, 16, 17, 31, 32, 33], [0] * 7, False),
    ([63, 64, 65, 127, 128, 129], [0] * 6, False),
    ([192, 193, 320, 5], [0, 256, 512, 256], True),
    ([40, 64, 65], [256, 768, 256], True),
])
def test_tiles_of_rows_and_heads(hq, hkv, q_lens, prefix, paged):
    w = workloads().make_prefill_workload(q_lens, prefix, hq, hkv, 128, 256, seed=hq + len(q_lens), paged=paged)
    out, ref = _run(w, hkv, paged, w["scale"], dtype=torch.float16 if hq == 8 else torch.bfloat16)
    assert_attention_close(to_np(out), ref)


def test_a_result_on_a_16_byte_boundary():
    w = workloads().make_prefill_workload([70, 130], [0, 0], 8, 2, 128, 256, seed=3, paged=False)
    n = w["q"].size
    room = torch.full((n + 24,), float("nan"), dtype=torch.bfloat16, device="cuda")
    at = (-(room.data_ptr() // 2) % 16) + 8                                # elements: past a 32-byte boundary by 16 bytes
    out, ref = _run(w, 2, False, w["scale"], out=room[at:at + n].view(w["q"].shape))
    assert out.data_ptr() % 32 == 16
    assert_attention_close(to_np(out), ref)
    assert torch.isnan(room[:at].float()).all() and torch.isnan(room[at + n:].float()).all()


@pytest.mark.parametrize("k_len", [40, 64, 100, 128, 190])
def test_rows_behind_a_sequence_do_not_matter(k_len):
    w = workloads().make_prefill_workload([k_len], [0], 8, 2, 128, 256, seed=k_len, paged=True)
    kc, vc = to_dev(w["k_cache"], torch.bfloat16), to_dev(w["v_cache"], torch.bfloat16)
    block = int(w["block_tables"][0, 0])
    kc[block, k_len:] = float("nan")
    vc[block, k_len:] = float("inf")
    vc[block, -1] = float("nan")
    out, ref = _run(w, 2, True, w["scale"], kc=kc, vc=vc)
    assert_attention_close(to_np(out), ref)


def test_rows_that_see_no_key():
    """More query rows than keys: the first rows see none and are zero."""
    bf, lib = torch.bfloat16, nvk()
    gen = torch.Generator(device="cuda").manual_seed(3)
    q = torch.randn((200, 8, 128), generator=gen, device="cuda").to(bf)
    k, v = (torch.randn((140, 2, 128), generator=gen, device="cuda").to(bf) for _ in range(2))
    cu_q, cu_k = (torch.tensor([0, n], dtype=torch.int32, device="cuda") for n in (200, 140))
    out = torch.full_like(q, float("nan"))
    lib.launch_prefill_attention_dense(q, cu_q, k, v, cu_k, 2, 128, 0.088, out)
    torch.cuda.synchronize()
    ref = oracle.prefill_attention_dense(to_np(q), to_np(k), to_np(v), to_np(cu_q), to_np(cu_k), 2, 128, 0.088)
    assert bool((out[:60] == 0).all())
    assert_attention_close(to_np(out), ref)


@pytest.mark.parametrize("scale", [0.0, -0.05])
def test_scales_that_are_not_positive(scale):
    w = workloads().make_prefill_workload([70, 130], [0, 0], 8, 2, 128, 256, seed=11, paged=False)
    out, ref = _run(w, 2, False, scale)
    assert_attention_close(to_np(out), ref)


@pytest.mark.parametrize("scale", [0.0, -0.05])
def test_odd_groups_with_scales_that_are_not_positive(scale):
    """Their tensor-core kernel hides scores before it scales them as well."""
    w = workloads().make_prefill_workload([70, 130], [0, 256], 6, 2, 128, 256, seed=13, paged=True)
    out, ref = _run(w, 2, True, scale)
    assert_attention_close(to_np(out), ref)


def test_a_mixed_step_takes_scales_that_are_not_positive():
    bf, lib, hkv = torch.bfloat16, nvk(), 2
    p = workloads().make_prefill_workload([70, 20], [0, 256], 8, hkv, 128, 256, seed=12, paged=True)
    kc, vc, pt = to_dev(p["k_cache"], bf), to_dev(p["v_cache"], bf), to_dev(p["block_tables"])
    pq, cu_q, cu_k, dq = to_dev(p["q"], bf), to_dev(p["cu_q"]), to_dev(p["cu_k"]), to_dev(p["q"][:2], bf)
    ctx = to_dev(np.array([70, 276], np.int32))
    ws = torch.empty(max(16, lib.decode_attention_workspace_bytes(2, 8, hkv, 128, pt.shape[1], 256)), dtype=torch.uint8, device="cuda")
    want_p, want_d, p_out, d_out = torch.empty_like(pq), torch.empty_like(dq), torch.empty_like(pq), torch.empty_like(dq)
    lib.launch_prefill_attention_paged(pq, cu_q, kc, vc, cu_k, pt, hkv, 128, 256, -0.05, want_p)
    lib.launch_decode_attention_paged(dq, kc, vc, ctx, pt, hkv, 128, 256, -0.05, want_d, ws)
    lib.attention_mixed_step(pq, cu_q, None, None, cu_k, pt, p_out, dq, ctx, pt, d_out, kc, vc, hkv, 128, 256, -0.05, ws)
    torch.cuda.synchronize()
    assert torch.equal(p_out, want_p) and torch.equal(d_out, want_d)


@pytest.mark.parametrize("index", ["i32", "i64"])
@pytest.mark.parametrize("hq,hkv,bs,q_lens,prefix,paged", [
    (8, 1, 256, [8], [256], True), (8, 2, 256, [9, 1], [512, 768], True), (4, 1, 128, [670], [0], True),        # clusters of 8, 8 and 4 (2 rows x 8 heads ...)
    (32, 8, 256, [77], [512], True), (16, 8, 256, [33], [256], True), (32, 8, 256, [100], [0], True),         # of 4, 8 and single blocks
    (32, 8, 256, [1] * 40 + [17, 5], [0] * 42, True), (4, 2, 256, [3, 0, 8, 20] * 9, [0] * 36, False),       # more than 32 sequences, empty ones among them
    (8, 2, 64, [70, 5], [64 * 40, 64 * 37], True), (4, 1, 64, [20], [64 * 70], True),                       # more block ids than lanes
    (16, 8, 256, [200], [0], False), (6, 3, 256, [65, 64, 63], [0, 256, 0], True),
])
def test_small_steps_in_tiles_of_64_rows(index, hq, hkv, bs, q_lens, prefix, paged):
    w = workloads().make_prefill_workload(q_lens, prefix, hq, hkv, 128, bs, seed=hq + len(q_lens), paged=paged)
    lib, bf = nvk(), torch.bfloat16
    it = torch.int32 if index == "i32" else torch.int64
    q, cu_q, cu_k = to_dev(w["q"], bf), to_dev(w["cu_q"]).to(it), to_dev(w["cu_k"]).to(it)
    if paged:
        kc, vc = to_dev(w["k_cache"], bf), to_dev(w["v_cache"], bf)
        for i, (a, b) in enumerate(zip(q_lens, prefix)):              # what lies behind a sequence's last key does not matter
            n = a + b
            if n % bs:
                last = int(w["block_tables"][i, n // bs])
                kc[last, n % bs:], vc[last, n % bs:] = float("nan"), float("inf")
        tables = to_dev(w["block_tables"]).to(it)
        run = lambda out, scale: lib.launch_prefill_attention_paged(q, cu_q, kc, vc, cu_k, tables, hkv, 128, bs, scale, out)
        want = lambda scale: oracle.prefill_attention_paged(w["q"], w["k_cache"], w["v_cache"], w["cu_q"], w["cu_k"], w["block_tables"], hkv, 128, bs, scale)
    else:
        k, v = to_dev(w["k"], bf), to_dev(w["v"], bf)
        run = lambda out, scale: lib.launch_prefill_attention_dense(q, cu_q, k, v, cu_k, hkv, 128, scale, out)
        want = lambda scale: oracle.prefill_attention_dense(w["q"], w["k"], w["v"], w["cu_q"], w["cu_k"], hkv, 128, scale)
    for scale in (w["scale"], -w["scale"]):
        out = torch.full_like(q, float("nan"))
        run(out, scale)
        torch.cuda.synchronize()
        assert lib.prefill_status() == 0
        assert_attention_close(to_np(out), want(scale))


def test_small_steps_keep_infinities_in_their_columns_and_rows_without_keys_at_zero():
    """An infinity in V of the first key: infinite where it is seen, in whatever block's part; rows that see no key give zeros."""
    w = workloads().make_prefill_workload([40], [512], 32, 8, 128, 256, seed=1, paged=True)
    lib, bf = nvk(), torch.bfloat16
    q, kc, vc = to_dev(w["q"], bf), to_dev(w["k_cache"], bf), to_dev(w["v_cache"], bf)
    vc[int(w["block_tables"][0, 0]), 0, :, 7] = float("inf")
    out = torch.full_like(q, float("nan"))
    lib.launch_prefill_attention_paged(q, to_dev(w["cu_q"]), kc, vc, to_dev(w["cu_k"]), to_dev(w["block_tables"]), 8, 128, 256, w["scale"], out)
    ref = oracle.prefill_attention_paged(w["q"], w["k_cache"], w["v_cache"], w["cu_q"], w["cu_k"], w["block_tables"], 8, 128, 256, w["scale"])
    assert bool((out[..., 7] == float("inf")).all())
    keep = [i for i in range(128) if i != 7]
    assert_attention_close(to_np(out[..., keep]), ref[..., keep])
    cu_k = torch.tensor([0, 30], dtype=torch.int32, device="cuda")     # 40 rows, 30 keys: the first ten see none
    lib.launch_prefill_attention_paged(q, to_dev(w["cu_q"]), kc, to_dev(w["v_cache"], bf), cu_k, to_dev(w["block_tables"]), 8, 128, 256, w["scale"], out)
    torch.cuda.synchronize()
    assert bool((out[:10] == 0).all()) and bool((out[10:].float().abs().amax((1, 2)) > 0).all())


@pytest.mark.parametrize("hq,hkv,q_len,bs", [(16, 8, 20, 256), (32, 8, 77, 256), (32, 8, 130, 64)])   # clusters of 8, 4 and 2 over the keys
def test_small_steps_keep_nan(hq, hkv, q_len, bs):
    """A NaN in a query row is in all of that row's results, and NaN keys are in the results of every row that sees them: also where a block's part
    of a row has nothing but NaN scores, and with them no maximum."""
    w = workloads().make_prefill_workload([q_len], [512], hq, hkv, 128, bs, seed=q_len, paged=True)
    lib, bf = nvk(), torch.bfloat16
    cu_q, cu_k, tables = to_dev(w["cu_q"]), to_dev(w["cu_k"]), to_dev(w["block_tables"])
    run = lambda q, kc, out: lib.launch_prefill_attention_paged(q, cu_q, kc, vc, cu_k, tables, hkv, 128, bs, w["scale"], out)
    q, kc, vc = to_dev(w["q"], bf), to_dev(w["k_cache"], bf), to_dev(w["v_cache"], bf)
    ref = oracle.prefill_attention_paged(w["q"], w["k_cache"], w["v_cache"], w["cu_q"], w["cu_k"], w["block_tables"], hkv, 128, bs, w["scale"])
    row, head = q_len // 2, hq - 2
    one = q.clone()
    one[row, head, 3] = float("nan")
    out = torch.zeros_like(q)
    run(one, kc, out)
    assert bool(torch.isnan(out[row, head].float()).all())
    rest = torch.ones((q_len, hq), dtype=torch.bool)
    rest[row, head] = False
    assert_attention_close(to_np(out)[rest.numpy()], ref[rest.numpy()])
    bad = kc.clone()
    for key in range(384):                                           # for one KV head
        bad[int(w["block_tables"][0, key // bs]), key % bs, 1] = float("nan")
    out = torch.zeros_like(q)
    run(q, bad, out)
    torch.cuda.synchronize()
    assert lib.prefill_status() == 0
    group = hq // hkv
    assert bool(torch.isnan(out[:, group:2 * group].float()).all())
    others = np.r_[0:group, 2 * group:hq]
    assert_attention_close(to_np(out)[:, others], ref[:, others])
