"""Tensor-core prefill over many packed sequences: the search for a query tile's sequence at the edges of its 32-sequence windows, with
empty sequences (whole windows of them too) among the others, and outputs of ragged tiles."""
import pytest

import oracle
from util import assert_attention_close, nvk, to_dev, to_np, workloads

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("q_lens,paged", [
    ([1] * 31 + [130], False),
    ([0] * 32 + [129], True),
    ([5] + [0] * 63 + [257], False),
    ([127, 128, 129, 0] * 8 + [0, 1, 300, 0] * 8 + [64], True),
    ([0] * 30 + [256, 3, 0, 131] + [0] * 40, True),
])
def test_every_query_tile_finds_its_sequence(q_lens, paged):
    prefix = [256 * (i % 3) if paged and n else 0 for i, n in enumerate(q_lens)]
    w = workloads().make_prefill_workload(q_lens, prefix, 8, 2, 128, 256, seed=len(q_lens), paged=paged)
    bf = torch.bfloat16
    q, cu_q, cu_k = to_dev(w["q"], bf), to_dev(w["cu_q"]), to_dev(w["cu_k"])
    out = torch.full_like(q, float("nan"))
    if paged:
        nvk().launch_prefill_attention_paged(q, cu_q, to_dev(w["k_cache"], bf), to_dev(w["v_cache"], bf), cu_k, to_dev(w["block_tables"]), 2, 128, 256,
                                             w["scale"], out)
        ref = oracle.prefill_attention_paged(w["q"], w["k_cache"], w["v_cache"], w["cu_q"], w["cu_k"], w["block_tables"], 2, 128, 256, w["scale"])
    else:
        nvk().launch_prefill_attention_dense(q, cu_q, to_dev(w["k"], bf), to_dev(w["v"], bf), cu_k, 2, 128, w["scale"], out)
        ref = oracle.prefill_attention_dense(w["q"], w["k"], w["v"], w["cu_q"], w["cu_k"], 2, 128, w["scale"])
    assert nvk().prefill_status() == 0
    assert_attention_close(to_np(out), ref)


def test_a_replayed_launch_shares_no_ticket_counter_with_eager_ones():
    """A graph with one prefill starts together with an eager one, 64 times: with 64 counters in turn one of them met the graph's."""
    bf, lib = torch.bfloat16, nvk()
    w = workloads().make_prefill_workload([128], [4096], 8, 2, 128, 256, seed=9)
    q, cu_q, cu_k, bt, kc, vc = (to_dev(w["q"], bf), to_dev(w["cu_q"]), to_dev(w["cu_k"]), to_dev(w["block_tables"]), to_dev(w["k_cache"], bf),
                                 to_dev(w["v_cache"], bf))

    def step(out):
        lib.launch_prefill_attention_paged(q, cu_q, kc, vc, cu_k, bt, 2, 128, 256, w["scale"], out)

    want, eager, replayed = torch.empty_like(q), torch.empty_like(q), torch.empty_like(q)
    step(want)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step(replayed)
    sides = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(64):
        eager.fill_(float("nan"))
        replayed.fill_(float("nan"))
        torch.cuda._sleep(400000)                                      # both are in their queues when it ends
        for side in sides:
            side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(sides[0]):
            graph.replay()
        with torch.cuda.stream(sides[1]):
            step(eager)
        torch.cuda.synchronize()
        assert torch.equal(eager, want) and torch.equal(replayed, want)
    assert lib.prefill_status() == 0
