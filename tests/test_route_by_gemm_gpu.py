"""Decode-sized calls whose GEMMs sort the (token, choice) slots themselves, against the same call on the
aligned path (a token block of 64 keeps it there) and against the oracle's routing order.

Both paths multiply the same 16-bit or FP8 rows with the same weights; what differs is the order in which an
output's at most topk fp32 terms are added and, for int4, the rounding of the expanded weights (fp16, 2^-11 of each),
so 16-bit and FP8 agree to a few units of the 16-bit output and int4 to 2e-3 in the 2-norm."""
import pytest
import torch

import flaggems_sglang_b200 as F
from flaggems_sglang_b200 import _lib
from flaggems_sglang_b200.quant import quantize_awq, quantize_fp8_block, repack_awq_for_kernel
from flaggems_sglang_b200.testing import make_tokens, make_weights
from oracle import moe as OM
from parity import assert_parity

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm()).item()


def _routing(tw, ids, e):
    order = torch.argsort(ids.flatten().long(), stable=True)
    return torch.bincount(ids.flatten().long(), minlength=e).int(), order.int(), tw.flatten()[order]


def _problem(kind, h, i, e, k, m, dev, variant):
    dtype = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp8": torch.bfloat16, "int4": torch.float16}[kind]
    w13, w2 = make_weights(h, i, e, dtype=dtype, device=dev, seed=3)
    x, tw, ids = make_tokens(m, h, e, k, dtype=dtype, device=dev, seed=4, skew=variant == "skew")
    kw = {}
    if variant == "twice":                       # a token that names an expert twice
        ids[:, 1] = ids[:, 0]
    elif variant == "map":                       # experts that live elsewhere
        emap = torch.arange(e, device=dev, dtype=torch.int32).flip(0)
        emap[::3] = -1
        kw["expert_map"] = emap
    elif variant == "nowhere":                   # slots without an expert
        ids[::2] = -1
    if kind == "fp8":
        (w13, s13), (w2, s2) = quantize_fp8_block(w13), quantize_fp8_block(w2)
        kw.update(use_fp8_w8a8=True, w13_scale=s13, w2_scale=s2)
    elif kind == "int4":
        w13, z13 = repack_awq_for_kernel(*quantize_awq(w13.transpose(1, 2).contiguous()))
        w2, z2 = repack_awq_for_kernel(*quantize_awq(w2.transpose(1, 2).contiguous()))
        kw.update(use_int4_w4a16=True, w13_sz=z13, w2_sz=z2)
    return x, w13, w2, tw, ids, kw


# tokens: one slot more and one less than a scan of 256, whole and odd blocks of 16 and 32, several blocks of an expert
@pytest.mark.parametrize("kind,h,i,e,k,m,variant", [
    ("bf16", 1024, 512, 128, 8, 31, "plain"), ("bf16", 1024, 512, 128, 8, 33, "skew"), ("bf16", 520, 264, 64, 4, 70, "twice"),
    ("bf16", 512, 256, 32, 4, 97, "map"), ("fp16", 512, 256, 16, 3, 85, "plain"), ("bf16", 512, 256, 8, 2, 100, "nowhere"),
    ("bf16", 256, 128, 1024, 8, 512, "plain"),
    ("fp8", 1024, 512, 64, 8, 32, "skew"), ("fp8", 512, 256, 64, 4, 64, "twice"), ("fp8", 512, 256, 64, 4, 61, "map"),
    ("fp8", 512, 256, 256, 12, 85, "plain"), ("fp8", 512, 256, 64, 4, 30, "nowhere"),
    ("int4", 1024, 512, 8, 2, 51, "plain"), ("int4", 640, 384, 16, 4, 33, "twice"), ("int4", 512, 256, 16, 4, 60, "map"),
    ("int4", 512, 256, 8, 2, 100, "nowhere"),
])
def test_sorted_by_the_gemms(cuda_device, kind, h, i, e, k, m, variant):
    x, w13, w2, tw, ids, kw = _problem(kind, h, i, e, k, m, cuda_device, variant)
    out = F.fused_experts(x, w13, w2, tw, ids, **kw)
    names = _lib.launch_stats()[1]
    assert "align_block_kernel" not in names, names
    wide = F.fused_experts(x, w13, w2, tw, ids.long(), **kw)
    aligned = F.fused_experts(x, w13, w2, tw, ids, block_tokens=64, **kw)
    assert "align_block_kernel" in _lib.launch_stats()[1]
    F.check_status()
    bound = 2e-3 if kind == "int4" else 1e-3
    assert _rel(out, aligned) <= bound
    assert _rel(wide, out) <= 1e-3
    if variant in ("plain", "skew", "twice"):
        triple = F.fused_experts(x, w13, w2, routing=(*_routing(tw, ids, e), k), **kw)
        assert _rel(triple, out) <= 1e-3
    if kind in ("bf16", "int4"):
        weighted = dict(kw, apply_router_weight_on_input=True)
        assert _rel(F.fused_experts(x, w13, w2, tw, ids, **weighted),
                    F.fused_experts(x, w13, w2, tw, ids, block_tokens=64, **weighted)) <= 4e-3


def test_largest_number_of_slots(cuda_device):
    """4096 slots sort in the GEMMs, 4104 on the aligned path; a graph replays the former with other routing."""
    h, i, e, k = 256, 128, 512, 8
    w13, w2 = make_weights(h, i, e, device=cuda_device, seed=1)
    for m, aligned in ((512, False), (513, True)):
        x, tw, ids = make_tokens(m, h, e, k, device=cuda_device, seed=2)
        out = F.fused_experts(x, w13, w2, tw, ids)
        assert ("align_block_kernel" in _lib.launch_stats()[1]) == aligned
        assert _rel(out, F.fused_experts(x, w13, w2, tw, ids, block_tokens=64)) <= 1e-3
    x, tw, ids = make_tokens(512, h, e, k, device=cuda_device, seed=5)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = F.fused_experts(x, w13, w2, tw, ids)
    for seed in (6, 7):
        x2, tw2, ids2 = make_tokens(512, h, e, k, device=cuda_device, seed=seed)
        x.copy_(x2), tw.copy_(tw2), ids.copy_(ids2)
        graph.replay()
        assert _rel(out, F.fused_experts(x2, w13, w2, tw2, ids2, block_tokens=64)) <= 1e-3
    F.check_status()


# the last call whose GEMMs sort the slots and the first one that is aligned; half of all slots name one expert, so that its
# blocks start behind several vectors of 256 slots
@pytest.mark.parametrize("kind,h,i,e,k,m,most", [
    ("bf16", 512, 256, 128, 8, 208, 208), ("bf16", 512, 256, 128, 8, 209, 208),
    ("fp8", 512, 256, 256, 8, 128, 128), ("fp8", 512, 256, 256, 8, 129, 128),
    ("int4", 512, 256, 64, 8, 40, 40), ("int4", 512, 256, 64, 8, 41, 40),
])
@pytest.mark.parametrize("variant", ["plain", "hot"])
def test_slots_of_a_call(cuda_device, kind, h, i, e, k, m, most, variant):
    x, w13, w2, tw, ids, kw = _problem(kind, h, i, e, k, m, cuda_device, variant)
    if variant == "hot":
        ids[:, :k // 2] = 3
    if kind == "fp8":
        kw["block_tokens"] = 16
    out = F.fused_experts(x, w13, w2, tw, ids, **kw)
    assert ("align_block_kernel" in _lib.launch_stats()[1]) == (m > most)
    kw["block_tokens"] = 64
    aligned = F.fused_experts(x, w13, w2, tw, ids, **kw)
    F.check_status()
    assert _rel(out, aligned) <= (2e-3 if kind == "int4" else 1e-3)
    if m == most and kind != "int4":                 # (int4 decode: tests/test_int4_gpu.py)
        c = [t.cpu() for t in (x, w13, w2, tw, ids)]
        ref = OM.fused_experts(*c) if kind == "bf16" else \
            OM.fused_experts_fp8(*c[:3], kw["w13_scale"].cpu(), kw["w2_scale"].cpu(), *c[3:])
        assert_parity(out, ref, what=f"sorted by the GEMMs {kind} {variant}")
