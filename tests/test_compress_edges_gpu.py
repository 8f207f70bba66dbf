"""Cache write at the sizes and values where its dispatch and its fast paths change: remainders of
the rows a warp takes at a time, the change from two to eight rows, rows that are not adjacent in
memory, boundaries that no uniform grid separates, and values that need the division instruction."""

import numpy as np
import pytest
import torch

import gpu_util
from gpu_util import DEV
from oracle import rq_exact
from rotorquant_vllm import cuda as rq

pytestmark = pytest.mark.gpu


def _values(kind, gen, shape):
    x = torch.randn(*shape, generator=gen)
    if kind == "zeros":                       # zero elements and zero rows
        x[torch.rand(*shape, generator=gen) < 0.02] = 0.0
        x[torch.rand(*shape[:2], generator=gen) < 0.1] = 0.0
    elif kind == "scales":                    # norms from 2^-130 to 2^60, elements far below their norm
        x = x * torch.exp2(torch.randint(-130, 60, (*shape[:2], 1), generator=gen).float())
        x = x * torch.exp2(-torch.randint(0, 2, shape, generator=gen).float() * 60)
    return x


@pytest.mark.parametrize("tokens,heads", [(1, 1), (1, 3), (9, 1), (5, 7), (63, 1), (255, 8), (256, 8), (683, 3)])
@pytest.mark.parametrize("kind,bounds", [("plain", "fit"), ("zeros", "fit"), ("scales", "fit"), ("plain", "uneven")])
@pytest.mark.parametrize("bits,dtype", [(3, torch.bfloat16), (4, torch.float32)])
def test_cache_write_edges(tokens, heads, kind, bounds, bits, dtype):
    p = gpu_util.params("iso_full", bits, 3)
    gen = torch.Generator().manual_seed(tokens * 10 + heads)
    k, v = (_values(kind, gen, (tokens, heads, 128)).to(dtype) for _ in range(2))
    kb, vb = p["k_boundaries"].clone(), p["v_boundaries"].clone()
    if bounds == "uneven":                    # repeated and bunched boundaries
        kb = torch.sort(torch.randn(kb.numel(), generator=gen) * 0.05)[0]
        vb[:3] = vb[3]
    slots = torch.randperm(tokens + 2, generator=gen)[:tokens]
    cache = torch.full((tokens + 2, 1, heads * 256), 0xAB, dtype=torch.uint8, device=DEV)
    wide = torch.zeros(tokens, heads + 1, 128, dtype=dtype, device=DEV)     # key rows: adjacent only within a token
    wide[:, :heads] = k.to(DEV)
    rq.compress_and_store(wide[:, :heads], v.to(DEV), cache, slots.to(DEV), p["R"].to(DEV), kb.to(DEV), vb.to(DEV))
    want = rq_exact.build_slots(k.float().numpy(), v.float().numpy(), p["R"].numpy(), kb.numpy(), vb.numpy())
    got = cache.cpu().reshape(tokens + 2, -1)
    assert np.array_equal(got[slots].numpy(), want)
    untouched = torch.ones(tokens + 2, dtype=torch.bool)
    untouched[slots] = False
    assert bool((got[untouched] == 0xAB).all())


@pytest.mark.parametrize("tokens", [3, 300])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_a_boundary_of_minus_zero_is_zero(tokens, dtype):
    """Values of +0 and -0 are not above a boundary of -0; zero rows have nothing else."""
    p = gpu_util.params("iso_fast", 4, 4)
    gen = torch.Generator().manual_seed(tokens)
    x = torch.randn(tokens, 8, 128, generator=gen)
    x[::2] = 0.0
    x[::4, :, ::3] = -0.0
    x = x.to(dtype)
    bounds = p["k_boundaries"].clone()
    bounds[7] = -0.0
    cache = torch.zeros(tokens, 1, 2048, dtype=torch.uint8, device=DEV)
    rq.compress_and_store(x.to(DEV), x.to(DEV), cache, torch.arange(tokens, device=DEV), p["R"].to(DEV), bounds.to(DEV),
                          p["v_boundaries"].to(DEV))
    want = rq_exact.build_slots(x.float().numpy(), x.float().numpy(), p["R"].numpy(), bounds.numpy(),
                                p["v_boundaries"].numpy())
    assert np.array_equal(cache.cpu().reshape(tokens, -1).numpy(), want)


@pytest.mark.parametrize("blocks,bs,lens,width", [(31, 16, [5, 300], 20), (32, 16, [512], 32), (33, 8, [0, 264], 40),
                                                  (1, 1, [1, 1, 1], 1), (1500, 16, [5000, 4000, 1], 700)])
@pytest.mark.parametrize("unused", [0, -1])
def test_referenced_blocks_are_listed_once_in_order(blocks, bs, lens, width, unused):
    """decompress_cache_paged against the plain torch way; sequences share blocks."""
    p = {k: v.to(DEV) for k, v in gpu_util.params("planar", 3, 4).items()}
    gen = torch.Generator().manual_seed(blocks)
    cache = torch.randint(0, 8, (blocks, bs, 512), generator=gen).to(torch.uint8).mul_(0x11)
    cache.view(-1, 512)[:, 128:136] = torch.rand(blocks * bs, 2, generator=gen).view(torch.uint8).view(-1, 8)
    cache.view(-1, 512)[:, 264:272] = torch.rand(blocks * bs, 2, generator=gen).view(torch.uint8).view(-1, 8)
    table = torch.full((len(lens), width), unused, dtype=torch.int32)
    for s, n in enumerate(lens):
        need = -(-n // bs)
        table[s, :need] = torch.randint(0, blocks, (need,), generator=gen).to(torch.int32)
    used = torch.cat([table[s, :-(-n // bs)] for s, n in enumerate(lens)])
    listed = torch.unique(used)
    remap = torch.zeros(blocks, dtype=torch.int32)
    remap[listed.long()] = torch.arange(listed.numel(), dtype=torch.int32)
    for dtype in (torch.bfloat16, torch.float32):
        k, v, got = rq.decompress_cache_paged(cache.to(DEV), table.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV), 2,
                                              p["k_centroids"], p["v_centroids"], dtype)
        assert torch.equal(got.cpu(), remap[table.long()])
        want_k, want_v = rq.decompress_blocks(cache.to(DEV), listed.to(torch.int32).to(DEV), 2, p["k_centroids"],
                                              p["v_centroids"], dtype)
        assert torch.equal(k, want_k) and torch.equal(v, want_v)
        rows = cache[listed.long()].view(-1, 512)
        idx = torch.stack([rows[:, 136:264] >> 4, rows[:, 136:264] & 15], -1).view(-1, 2, 128).long()
        norm = rows[:, 264:272].contiguous().view(torch.float32).view(-1, 2, 1)
        assert torch.equal(v.cpu().view(-1, 2, 128), (p["v_centroids"].cpu()[idx] * norm).to(dtype))


@pytest.mark.parametrize("tables", ["plain", "many"])        # "many" entries: the way through torch
def test_blocks_outside_the_cache(tables):
    """Needed entries outside the cache are an error of the host; entries that no sequence reaches may be anything."""
    p = {k: v.to(DEV) for k, v in gpu_util.params("iso_fast", 3, 3).items()}
    cache = torch.randint(0, 255, (6, 4, 256), dtype=torch.uint8, device=DEV)
    table = torch.full((2, 8 if tables == "plain" else (1 << 19) + 1), 1 << 20, dtype=torch.int32, device=DEV)
    table[0, :3], table[1, :2] = torch.tensor([5, 0, 3]).to(table), torch.tensor([3, 4]).to(table)
    args = (1, p["k_centroids"], p["v_centroids"], torch.bfloat16)
    k, _, remapped = rq.decompress_cache_paged(cache, table, torch.tensor([12, 5], dtype=torch.int32, device=DEV), *args)
    assert k.shape[0] == 4 and remapped[0, :3].tolist() == [3, 0, 1] and remapped[1, :2].tolist() == [1, 2]
    assert int(remapped[:, 3:].abs().max()) == 0
    with pytest.raises(ValueError, match="of a cache of 6 blocks"):
        rq.decompress_cache_paged(cache, table, torch.tensor([12, 9], dtype=torch.int32, device=DEV), *args)
