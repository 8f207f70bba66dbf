"""The launchers' native side (``_host-*.so``) takes ordinary calls; everything else goes through the
Python path.  Both must give the same bytes, and the native side must not take what it may not."""

import pytest
import torch

import gpu_util
from gpu_util import DEV
from rotorquant_vllm import _lib
from rotorquant_vllm import cuda as rq

pytestmark = pytest.mark.gpu


def _layer():
    return {k: v.to(DEV) for k, v in gpu_util.params("iso_fast", 3, 3).items()}


@pytest.mark.parametrize("tokens,heads", [(1, 8), (37, 3), (2049, 8)])
@pytest.mark.parametrize("variant", ["plain", "column_rows", "f64_boundaries", "wider_rows"])
def test_both_paths_write_the_same_bytes(tokens, heads, variant):
    p = _layer()
    gen = torch.Generator(device=DEV).manual_seed(tokens)
    k = torch.randn(tokens, heads, 128, generator=gen, device=DEV).to(torch.bfloat16)
    slots = torch.randperm(tokens, generator=gen, device=DEV)
    want, got = (torch.zeros(tokens, 1, heads * 256, dtype=torch.uint8, device=DEV) for _ in range(2))
    assert _lib.host().compress_store(k, k, want, slots, p["R"], p["k_boundaries"], p["v_boundaries"], True) is None, \
        "a rotation that was never validated must not be taken"
    rq.compress_and_store(k, k, want, slots, p["R"], p["k_boundaries"], p["v_boundaries"])
    src, bounds = k, p["k_boundaries"]
    if variant == "column_rows":            # elements of a row are not adjacent: copied by the Python path
        src = k.transpose(1, 2).contiguous().transpose(1, 2)
    elif variant == "f64_boundaries":
        bounds = bounds.double()
    elif variant == "wider_rows":            # a strided view of a wider tensor: taken as it is
        src = torch.empty(tokens, heads + 1, 128, dtype=k.dtype, device=DEV)[:, :heads].copy_(k)
    taken = _lib.host().compress_store(src, k, got, slots, p["R"], bounds, p["v_boundaries"], True)
    assert (taken is None) == (variant in ("column_rows", "f64_boundaries"))
    rq.compress_and_store(src, k, got, slots, p["R"], bounds, p["v_boundaries"])
    assert torch.equal(got, want)


def test_a_rotation_changed_in_place_is_checked_again():
    p = _layer()
    x = torch.randn(5, 8, 128, device=DEV)
    cache = torch.zeros(5, 1, 2048, dtype=torch.uint8, device=DEV)
    args = (x, x, cache, torch.arange(5, device=DEV), p["R"], p["k_boundaries"], p["v_boundaries"])
    rq.compress_and_store(*args)
    p["R"][0, 100] = 0.5
    with pytest.raises(ValueError, match="diagonal"):
        rq.compress_and_store(*args)


@pytest.mark.parametrize("other", [lambda r: r[:64, :64].contiguous(), lambda r: r.double(), lambda r: r[:, ::2]])
def test_a_validated_rotation_that_was_given_other_data_is_refused(other):
    """Such an assignment does not change the version of the tensor."""
    p = _layer()
    x = torch.randn(5, 8, 128, device=DEV)
    cache = torch.zeros(5, 1, 2048, dtype=torch.uint8, device=DEV)
    args = (x, x, cache, torch.arange(5, device=DEV), p["R"], p["k_boundaries"], p["v_boundaries"])
    rq.compress_and_store(*args)
    p["R"].data = other(p["R"].clone())
    with pytest.raises(ValueError, match="rotation must be"):
        rq.compress_and_store(*args)


def test_errors_of_the_library_keep_their_types():
    p = _layer()
    q = torch.randn(1, 8, 128, device=DEV)                      # fp32 queries are not supported
    cache = torch.zeros(4, 16, 256, dtype=torch.uint8, device=DEV)
    table, lens = torch.zeros(1, 4, dtype=torch.int32, device=DEV), torch.ones(1, dtype=torch.int32, device=DEV)
    for _ in range(2):                                          # before and after the scratch is in place
        with pytest.raises(ValueError, match="dtype"):
            rq.fused_paged_rq_decode(q, cache, table, lens, p["k_centroids"], p["v_centroids"], p["R"], 1, 128, 16)
        rq.fused_paged_rq_decode(q.half(), cache, table, lens, p["k_centroids"], p["v_centroids"], p["R"], 1, 128, 16)


def test_scratch_must_be_on_the_device_of_the_call():
    p = _layer()
    q = torch.randn(1, 8, 128, device=DEV).half()
    cache = torch.zeros(4, 16, 256, dtype=torch.uint8, device=DEV)
    table, lens = torch.zeros(1, 4, dtype=torch.int32, device=DEV), torch.ones(1, dtype=torch.int32, device=DEV)
    args = (q, cache, table, lens, p["k_centroids"], p["v_centroids"], p["R"], 1, 128, 16)
    for call in (rq.fused_paged_rq_decode, rq.fused_paged_rq_int8_prefill):
        with pytest.raises(RuntimeError, match="CUDA tensors only"):
            call(*args, workspace=torch.empty(1 << 22, dtype=torch.uint8))
