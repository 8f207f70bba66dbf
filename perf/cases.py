"""The KV-cache work of one attention layer, as a serving program calls it.

A layer's forward pass writes the step's new K/V tokens into the compressed cache and then attends
over the cache: one query token per sequence (``decode``) or a batch with prompt tokens in it
(``prefill``, several sequences, cached prefixes, single-token rows of running requests among them).
``write`` is the cache write of prompt tokens alone; ``rows`` compresses plain rows and expands them
again; ``gather`` expands the cache blocks that a batch references.

Inputs are synthetic: N(0, 1) queries, keys and values with a x10 outlier channel in K and V, and
random block tables, the distributions of the repository's benchmark.  All sizes of a case are in the
case; the seed decides the values, the block tables and the order of the sequence lengths.
"""

from __future__ import annotations

import functools
import math
import os
import sys

import torch

_SRC = os.path.abspath("rotorquant-vllm_b200")
if _SRC not in sys.path:
    sys.path.insert(0, _SRC)

from rotorquant_vllm import cuda as rq  # noqa: E402
from rotorquant_vllm.cuda.decompress import decompress_cache_paged  # noqa: E402
from rotorquant_vllm.quantization import IsoQuantMSE, PlanarQuantMSE  # noqa: E402
from rotorquant_vllm.vllm.rotation import build_rotation_matrix  # noqa: E402

DEV = "cuda"
D = 128                          # the head size of the path
SLOT_BYTES = 136                 # payload of one token and KV head: 2 x (64 index bytes + fp32 norm)
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


def listed() -> list[dict]:
    return [
        # One user of a chat model: a single short sequence under an 8192-token limit, so that the
        # launches and the host path are most of the time.
        _decode("decode_1x333", 1, 333, 333, 32, 8, limit=8192),
        # The headline configuration of the benchmark: 64 sequences of 4096 tokens, 32 / 8 heads.
        _decode("decode_64x4096", 64, 4096, 4096, 32, 8),
        # A busy server with requests of all ages: 256 ragged sequences, planar, 4-bit K, 7 query
        # heads per KV head.
        _decode("decode_256_ragged_planar", 256, 512, 8192, 28, 4, mode="planar", k_bits=4),
        # Long documents: 8 sequences of 131072 tokens, 64 / 8 heads on one GPU, iso-full.
        _decode("decode_8x131072", 8, 131072, 131072, 64, 8, mode="iso_full"),
        # The tensor-parallel shard of such a model: one KV head and 8 query heads per GPU, fp16.
        _decode("decode_16_long_1head_f16", 16, 2048, 32768, 8, 1, mode="iso_full", dtype="f16"),
        # A short prompt of one user.
        _prefill("prefill_1x300", 1, 300, 300, 0, 32, 8, limit=8192),
        # The prefill configuration of the benchmark: 8 prompts of 2048 tokens.
        _prefill("prefill_8x2048", 8, 2048, 2048, 0, 32, 8),
        # A 2048-token chunk of a long prompt whose first 30000 tokens are in the cache already.
        _prefill("prefill_chunk_2048_at_30000", 1, 2048, 2048, 30000, 32, 8, limit=32768),
        # What a scheduler with chunked prefill sends most of the time: running requests with one
        # token each and two prompt chunks in the same batch; fp16, 4-bit, 7 heads per KV head.
        _prefill("prefill_mixed_30_decodes_f16", 32, 250, 1500, 4000, 28, 4, decodes=30, mode="planar", k_bits=4,
                 v_bits=4, dtype="f16"),
        # Cache write of a full prompt batch, the compress metric of the benchmark.
        {"name": "write_16384x8", "kind": "write", "tokens": 16384, "kv_heads": 8, "block": 16, "mode": "iso_fast",
         "k_bits": 3, "v_bits": 3, "dtype": "bf16"},
        # Plain rows to packed rows and back, fp32.
        {"name": "rows_8192x8_f32", "kind": "rows", "tokens": 8192, "kv_heads": 8, "mode": "planar", "k_bits": 3,
         "dtype": "f32"},
        # The blocks of a small batch as plain K and V, for attention kernels that want them.
        {"name": "gather_4x2048", "kind": "gather", "seqs": 4, "ctx_min": 700, "ctx_max": 2048, "kv_heads": 8,
         "block": 16, "limit": 8192, "mode": "iso_fast", "k_bits": 3, "v_bits": 3, "dtype": "bf16"},
    ]


def _decode(name, seqs, ctx_min, ctx_max, q_heads, kv_heads, *, mode="iso_fast", k_bits=3, v_bits=3, dtype="bf16",
            block=16, limit=0) -> dict:
    case = {"kind": "decode", "seqs": seqs, "ctx_min": ctx_min, "ctx_max": ctx_max, "q_heads": q_heads,
            "kv_heads": kv_heads, "mode": mode, "k_bits": k_bits, "v_bits": v_bits, "dtype": dtype, "block": block,
            "limit": max(limit, ctx_max)}
    return {"name": name, **case} if name else case


def _prefill(name, seqs, q_min, q_max, prefix, q_heads, kv_heads, *, decodes=0, mode="iso_fast", k_bits=3, v_bits=3,
             dtype="bf16", block=16, limit=0) -> dict:
    """``seqs - decodes`` prompt chunks of ``q_min .. q_max`` tokens and ``decodes`` single-token rows; the
    prompts have up to ``prefix`` cached tokens, the single-token rows 1 .. ``prefix``."""
    case = {"kind": "prefill", "seqs": seqs, "decodes": decodes, "q_min": q_min, "q_max": q_max, "prefix": prefix,
            "q_heads": q_heads, "kv_heads": kv_heads, "mode": mode, "k_bits": k_bits, "v_bits": v_bits,
            "dtype": dtype, "block": block, "limit": max(limit, q_max + prefix)}
    return {"name": name, **case} if name else case


# ---- drawn cases ------------------------------------------------------------------------------------

# query heads / KV heads on one GPU: whole models of the configurations and their tensor-parallel shards
HEADS = [(32, 8), (28, 4), (64, 8), (16, 4), (16, 2), (8, 1), (8, 8), (32, 2)]


def _log_int(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng) -> dict:
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "prefill", "write", "rows", "gather"])
    q_heads, kv_heads = rng.choice(HEADS)
    opts = {"mode": rng.choice(["iso_fast", "iso_full", "planar"]), "k_bits": rng.choice([3, 3, 4]),
            "v_bits": rng.choice([3, 3, 4]), "dtype": rng.choice(["bf16", "bf16", "f16"]),
            "block": rng.choice([16, 16, 32, 64])}
    if kind == "decode":
        seqs = _log_int(rng, 1, 256)
        # no more cached tokens and heads than 8 sequences of 131072 tokens with 8 KV heads
        most = max(32, min(131072, 8 * 131072 * 8 // (seqs * kv_heads)))
        ctx_max = _log_int(rng, 16, most)
        ctx_min = ctx_max if rng.random() < 0.3 else _log_int(rng, 1, ctx_max)
        return _decode(None, seqs, ctx_min, ctx_max, q_heads, kv_heads, limit=_limit(rng, ctx_max), **opts)
    if kind == "prefill":
        q_max = _log_int(rng, 8, 4096)
        q_min = q_max if rng.random() < 0.3 else _log_int(rng, 1, q_max)
        seqs = _log_int(rng, 1, max(1, 16384 // q_max))
        decodes = rng.choice([0, 0, 0, 12, 30, 60])
        prefix = rng.choice([0, 0, _log_int(rng, 16, 30000)]) if not decodes else _log_int(rng, 16, 6000)
        seqs = min(seqs, 64)
        # no more query-key pairs than 2048 tokens after 30000 with 32 query heads
        while seqs * q_max * (prefix + q_max / 2) * q_heads > 2048 * 30000 * 32:
            seqs, prefix = (seqs // 2, prefix) if seqs > 1 else (1, prefix // 2)
        return _prefill(None, seqs + decodes, q_min, q_max, prefix, q_heads, kv_heads, decodes=decodes,
                        limit=_limit(rng, q_max + prefix), **opts)
    if kind == "write":
        return {"kind": "write", "tokens": _log_int(rng, 1, 16384), "kv_heads": kv_heads,
                **dict(opts, dtype=rng.choice(["bf16", "f16", "f32"]))}
    if kind == "rows":
        opts.pop("v_bits"), opts.pop("block")
        return {"kind": "rows", "tokens": _log_int(rng, 1, 16384), "kv_heads": kv_heads,
                **dict(opts, dtype=rng.choice(["bf16", "f16", "f32"]))}
    ctx_max = _log_int(rng, 16, 8192)
    return {"kind": "gather", "seqs": _log_int(rng, 1, 16), "ctx_min": _log_int(rng, 1, ctx_max), "ctx_max": ctx_max,
            "kv_heads": kv_heads, "limit": _limit(rng, ctx_max), **opts}


def _limit(rng, tokens: int) -> int:
    """The longest sequence the server admits, which is the width of the block table."""
    return max(tokens, rng.choice([tokens, 8192]))


# ---- sizes --------------------------------------------------------------------------------------------

def _spread(lo: int, hi: int, n: int) -> list[int]:
    """``n`` whole numbers from ``lo`` to ``hi``, evenly spread."""
    return [hi] if n == 1 else [lo + (hi - lo) * i // (n - 1) for i in range(n)]


def _lengths(case: dict) -> tuple[list[int], list[int]]:
    """(query tokens, cached tokens with the new ones) of every sequence, in a fixed order."""
    if case["kind"] in ("decode", "gather"):
        ctx = _spread(case["ctx_min"], case["ctx_max"], case["seqs"])
        return [1] * len(ctx), ctx
    n = case["seqs"] - case["decodes"]
    q = _spread(case["q_min"], case["q_max"], n)
    kv = [a + b for a, b in zip(q, _spread(case["prefix"] // 2, case["prefix"], n))]
    return q + [1] * case["decodes"], kv + _spread(1, max(1, case["prefix"]), case["decodes"]) if case["decodes"] else kv


def work(case: dict) -> dict:
    es = DTYPES[case["dtype"]].itemsize
    h = case["kv_heads"]
    if case["kind"] == "write":           # K and V in, payload out
        return {"bytes": case["tokens"] * (h * (2 * D * es + SLOT_BYTES) + 8), "flops": case["tokens"] * h * 2 * 12 * D}
    if case["kind"] == "rows":            # in, packed rows and norms, out
        return {"bytes": case["tokens"] * h * (2 * D * es + 2 * (D // 2 + 4)), "flops": case["tokens"] * h * 13 * D}
    q, kv = _lengths(case)
    table = sum(4 * -(-n // case["block"]) for n in kv)
    if case["kind"] == "gather":
        cells = sum(-(-n // case["block"]) for n in kv) * case["block"] * h
        return {"bytes": cells * (SLOT_BYTES + 2 * D * es) + 2 * 4 * case["seqs"] * -(-case["limit"] // case["block"]),
                "flops": cells * 2 * D}
    hq = case["q_heads"]
    pairs = sum(a * (b - a) + a * (a + 1) // 2 for a, b in zip(q, kv))      # causal: query tokens x visible keys
    new = sum(q)
    return {"bytes": sum(kv) * h * SLOT_BYTES + table + new * (2 * hq * D * es + 2 * h * D * es + h * SLOT_BYTES + 8),
            "flops": 4 * D * hq * pairs}


def tolerance(case: dict):
    """Compressed bytes and their expansion are the reference's bit for bit; attention outputs carry the
    rounding of their type (twice: before and after the output rotation) and of the probabilities."""
    if case["kind"] in ("write", "rows", "gather"):
        return "exact"
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 4e-3, "differ": 0.0}


# ---- inputs -------------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _layer(mode: str, k_bits: int, v_bits: int) -> dict:
    """Codebooks and rotation of a layer, built once when the layer is."""
    def make(bits):
        if mode == "planar":
            return PlanarQuantMSE(D, bits, seed=42)
        return IsoQuantMSE(D, bits, seed=42, mode="full" if mode == "iso_full" else "fast")

    k, v = make(k_bits), make(v_bits)
    rot = build_rotation_matrix(k, D, "cpu")
    return {"rot": rot.to(DEV), "rot_T_even": rot.T[:, 0::2].contiguous().to(DEV),
            "rot_T_odd": rot.T[:, 1::2].contiguous().to(DEV),
            "ck": k.centroids.to(DEV), "cv": v.centroids.to(DEV), "bk": k.boundaries.to(DEV), "bv": v.boundaries.to(DEV)}


def _kv(gen, tokens: int, heads: int, dtype) -> tuple[torch.Tensor, torch.Tensor]:
    x = torch.randn(2, tokens, heads, D, generator=gen, device=DEV)
    x[..., int(torch.randint(D, (1,), generator=gen, device=DEV))] *= 10.0
    return x[0].to(dtype), x[1].to(dtype)


def _paged(gen, kv: list[int], case: dict):
    """A random deal of the physical blocks: (block table as wide as the longest admitted sequence, number of
    blocks)."""
    bs = case["block"]
    need = [-(-n // bs) for n in kv]
    num_blocks = sum(need) + 2
    perm = torch.randperm(num_blocks, generator=gen, device=DEV).to(torch.int32)
    table = torch.zeros(len(kv), -(-case["limit"] // bs), dtype=torch.int32, device=DEV)
    at = 0
    for s, nb in enumerate(need):
        table[s, :nb] = perm[at:at + nb]
        at += nb
    return table, num_blocks


def _slots(table, lo: int, hi: int, s: int, bs: int) -> torch.Tensor:
    pos = torch.arange(lo, hi, device=DEV)
    return table[s].long()[pos // bs] * bs + pos % bs


def prepare(case: dict, seed: int) -> dict:
    gen = torch.Generator(device=DEV).manual_seed(seed)
    h, dtype = case["kv_heads"], DTYPES[case["dtype"]]
    layer = _layer(case["mode"], case["k_bits"], case.get("v_bits", case["k_bits"]))
    if case["kind"] == "rows":
        return {"kind": "rows", "planar": case["mode"] == "planar", "x": _kv(gen, case["tokens"], h, dtype)[0], **layer}
    if case["kind"] == "write":
        bs = case["block"]
        blocks = -(-case["tokens"] // bs) + 2
        key, value = _kv(gen, case["tokens"], h, dtype)
        slots = torch.randperm(blocks, generator=gen, device=DEV)[:, None] * bs + torch.arange(bs, device=DEV)
        return {"kind": "write", "key": key, "value": value, "slots": slots.reshape(-1)[:case["tokens"]].contiguous(),
                "cache": torch.zeros(blocks, bs, h * 256, dtype=torch.uint8, device=DEV), **layer}

    q_lens, kv_lens = _lengths(case)
    order = torch.randperm(len(q_lens), generator=torch.Generator().manual_seed(seed)).tolist()
    if case["kind"] == "prefill":          # running requests first, as a scheduler lays a batch out
        order.sort(key=lambda i: q_lens[i] > 1)
    q_lens, kv_lens = [q_lens[i] for i in order], [kv_lens[i] for i in order]
    table, num_blocks = _paged(gen, kv_lens, case)
    bs = case["block"]
    cache = torch.zeros(num_blocks, bs, h * 256, dtype=torch.uint8, device=DEV)
    # every cached token of the batch, written a few tens of thousands at a time
    all_slots = torch.cat([_slots(table, 0, n, s, bs) for s, n in enumerate(kv_lens)])
    for part in all_slots.split(1 << 17):
        rq.compress_and_store(*_kv(gen, part.numel(), h, dtype), cache, part.contiguous(), layer["rot"], layer["bk"],
                              layer["bv"])
    state = {"kind": case["kind"], "cache": cache, "table": table, "heads": h, "block": bs, "dtype": dtype,
             "seq_lens": torch.tensor(kv_lens, dtype=torch.int32, device=DEV), **layer}
    if case["kind"] == "gather":
        return state
    n = sum(q_lens)
    key, value = _kv(gen, n, h, dtype)
    q = torch.randn(n, case["q_heads"], D, generator=gen, device=DEV).to(dtype)
    slots = torch.cat([_slots(table, kv - ql, kv, s, bs) for s, (ql, kv) in enumerate(zip(q_lens, kv_lens))])
    state.update(key=key, value=value, q=q, slots=slots, out=torch.empty_like(q), scale=D ** -0.5)
    if case["kind"] == "prefill":
        # what the scheduler knows on the host
        state["bounds"] = {"max_q_len": max(q_lens), "max_seq_len": max(kv_lens)}
        if len(q_lens) > 1:
            cu = torch.tensor([0] + q_lens, device=DEV).cumsum(0).to(torch.int32)
            state["bounds"]["cu_seqlens_q"] = cu
    return state


# ---- one pass -----------------------------------------------------------------------------------------

def run(s: dict):
    kind = s["kind"]
    if kind == "rows":
        pack, unpack = ((rq.planar_compress, rq.planar_decompress) if s["planar"]
                        else (rq.iso_compress, rq.iso_decompress))
        packed, norms = pack(s["x"], s["rot_T_even"], s["rot_T_odd"], s["bk"])
        return packed, norms, unpack(packed, norms, s["ck"], s["x"].dtype)
    if kind == "gather":
        return decompress_cache_paged(s["cache"], s["table"], s["seq_lens"], s["heads"], s["ck"], s["cv"], s["dtype"])
    rq.compress_and_store(s["key"], s["value"], s["cache"], s["slots"], s["rot"], s["bk"], s["bv"])
    if kind == "write":
        return s["cache"]
    common = (s["q"], s["cache"], s["table"], s["seq_lens"], s["ck"], s["cv"], s["rot"], s["heads"], D, s["block"])
    if kind == "decode":
        rq.fused_paged_rq_decode(*common, sm_scale=s["scale"], out=s["out"])
    else:
        rq.fused_paged_rq_int8_prefill(*common, sm_scale=s["scale"], out=s["out"], **s["bounds"])
    return s["out"], s["cache"]
