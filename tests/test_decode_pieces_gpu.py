"""Decode batches whose tiles are fewer than, as many as, or just more than the pieces the launch is
cut into (short sequences under a wide block table), and rows with many parts in the merge."""

import pytest
import torch

import gpu_util
from gpu_util import DEV
from oracle import rq_oracle, tolerance
from rotorquant_vllm import cuda as rq
from rotorquant_vllm import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,HQ,lens,limit", [
    (8, 32, [1], 8192), (8, 32, [333], 8192),
    (8, 32, [128 * 73 + 5], 128 * 80), (8, 32, [128 * 74], 128 * 80), (8, 32, [128 * 74 + 1], 128 * 80),    # 74 pieces
    (1, 8, [128, 129, 0, 4000], 8192), (1, 8, [30000], 30000),                  # a row of 235 parts
    (4, 28, [3] * 130, 1024),                                                   # the plan launch
])
def test_few_tiles_per_piece(H, HQ, lens, limit):
    p = gpu_util.params("iso_fast", 3, 3)
    seq_lens = torch.tensor(lens, dtype=torch.int32)
    bt, nb = syn.make_block_table(seq_lens, 16, 1)
    table = torch.zeros(len(lens), limit // 16, dtype=torch.int32)
    table[:, :bt.shape[1]] = bt
    slots = syn.slot_mapping_for(bt, seq_lens, 16)
    key, value = syn.make_kv(int(seq_lens.sum()), H, 128, torch.bfloat16, 1)
    q = syn.make_queries(len(lens), HQ, 128, torch.bfloat16, 1)
    layer = {k: v.to(DEV) for k, v in p.items()}
    cache = torch.zeros(nb, 16, H * 256, dtype=torch.uint8, device=DEV)
    rq.compress_and_store(key.to(DEV), value.to(DEV), cache, slots.to(DEV), layer["R"], layer["k_boundaries"],
                          layer["v_boundaries"])
    out = rq.fused_paged_rq_decode(q.to(DEV), cache, table.to(DEV), seq_lens.to(DEV), layer["k_centroids"],
                                   layer["v_centroids"], layer["R"], H, 128, 16).cpu()
    args = (q, cache.cpu(), table, seq_lens, p["k_centroids"], p["v_centroids"], p["R"], H, 128, 16)
    worst, over = tolerance.excess(out, rq_oracle.decode(*args, return_rotated_fp32=True), rq_oracle.decode(*args),
                                   torch.bfloat16)
    assert over == 0, worst
