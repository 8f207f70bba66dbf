"""Launches that start under the one before them, where the stream has been forked and joined: eagerly and in a
captured graph.  A layer's step (cache write, decode, prefill) whose queries a second stream makes meanwhile
must give the results of the same step with the device idle between the calls."""

import pytest
import torch

import gpu_util
from gpu_util import DEV
from rotorquant_vllm import cuda as rq
from rotorquant_vllm import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seqs", [3, 130])                  # 130: decode with its plan launch
@pytest.mark.parametrize("captured", [False, True])
def test_a_step_with_a_second_stream(seqs, captured):
    p = {k: v.to(DEV) for k, v in gpu_util.params("iso_fast", 3, 4).items()}
    H, HQ, BS = 4, 28, 16
    lens = torch.tensor([40 + 53 * i % 700 for i in range(seqs)], dtype=torch.int32)
    table, blocks = syn.make_block_table(lens, BS, seqs)
    slots = syn.slot_mapping_for(table, lens, BS).to(DEV)
    table, lens = table.to(DEV), lens.to(DEV)
    key, value = (t.to(DEV) for t in syn.make_kv(int(lens.sum()), H, 128, torch.bfloat16, 1))
    source = syn.make_queries(seqs, HQ, 128, torch.bfloat16, 1).to(DEV)
    cache = torch.zeros(blocks, BS, H * 256, dtype=torch.uint8, device=DEV)
    q = torch.zeros_like(source)
    cu = torch.arange(seqs + 1, dtype=torch.int32, device=DEV)
    outs = [torch.zeros_like(q) for _ in range(3)]
    side = torch.cuda.Stream()

    def step(between):
        main = torch.cuda.current_stream()
        side.wait_stream(main)
        with torch.cuda.stream(side):
            for _ in range(20):                             # long enough to be under way when the write has ended
                torch.mul(source, 1.0, out=q)
        rq.compress_and_store(key, value, cache, slots, p["R"], p["k_boundaries"], p["v_boundaries"])
        between()
        main.wait_stream(side)
        common = (cache, table, lens, p["k_centroids"], p["v_centroids"], p["R"], H, 128, BS)
        rq.fused_paged_rq_decode(q, *common, out=outs[0])
        between()
        rq.fused_paged_rq_int8_prefill(q, *common, out=outs[1], cu_seqlens_q=cu, max_q_len=1, staged=True)
        between()
        rq.fused_paged_rq_decode(q, *common, out=outs[2])

    step(torch.cuda.synchronize)
    torch.cuda.synchronize()
    run = lambda: step(lambda: None)                        # noqa: E731
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            run()
        run = graph.replay
    for factor in (0.5, -1.0, 2.0):
        source *= factor
        key *= factor
        step(torch.cuda.synchronize)
        torch.cuda.synchronize()
        want = [o.clone() for o in outs]
        for t in (cache, q, *outs):
            t.zero_()
        run()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(outs, want))
        assert torch.equal(outs[0], outs[2])
