"""FP8 blocks of 128 in one launch with blocks of at most 16 rows (moe_gemm_fp8_mixed_kernel), against blocks of 16
alone on the same quantised inputs.

Every product and every per-slice scaling is the same in both; the down projection adds an output's fp32 terms in another
order or, with pair rows, rounds each to the 16-bit type first (2^-9 of it), so outputs agree to 4e-3 in the 2-norm."""
import importlib

import pytest
import torch

import flaggems_sglang_b200 as F
from flaggems_sglang_b200 import _lib
from flaggems_sglang_b200.quant import quantize_fp8_block
from flaggems_sglang_b200.testing import make_tokens, make_weights, route, zipf_bias
from oracle import moe as OM
from parity import assert_parity

pytestmark = pytest.mark.gpu

EDGES = [1, 15, 16, 17, 127, 128, 129, 0, 300, 2, 255, 257]


def _ids(counts, m, k, seed):
    """[m, k] expert ids with these numbers of slots (the rest is -1), in any order: an expert may stand twice in a token."""
    slots = torch.cat([torch.full((c,), e) for e, c in enumerate(counts)])
    flat = torch.full((m * k,), -1)
    flat[: slots.numel()] = slots
    g = torch.Generator().manual_seed(seed)
    return flat[torch.randperm(m * k, generator=g)].view(m, k).to(torch.int32)


@pytest.mark.parametrize("h,i,counts,kw", [
    (512, 256, EDGES, {}),
    (512, 256, EDGES, dict(no_combine=True)),
    (512, 384, EDGES, dict(apply_router_weight_on_input=True)),
    (384, 256, EDGES, dict(bias=True, activation="swiglu_oai", swiglu_alpha=1.7, swiglu_limit=7.0)),
    (512, 256, [9] * 96, {}),                       # nothing but cold blocks
    (512, 256, [64] * 24, {}),                      # nothing but hot ones
    (512, 256, [700] + [1] * 250, {}),
    (512, 256, [20] * 40 + [3] * 4, {}),            # too few cold blocks for CTAs of their own; one more
    (512, 256, [20] * 40 + [3] * 10, {}),
    (2560, 256, [20] * 200 + [16, 1] * 30, {}),      # pair rows, 35 x 10 tiles; enough cold blocks for CTAs of their own
    # the down projection stores pair rows (29 full blocks' worth of slots x 11 tiles of columns, from 296 on)
    (2816, 256, EDGES * 3, {}),
    (2816, 256, EDGES * 3, dict(bias=True)),
    (2688, 256, EDGES * 3, dict(dtype=torch.float16)),      # half of a tile's columns past the end
])
def test_hot_and_cold_blocks(cuda_device, h, i, counts, kw):
    d, e, k = cuda_device, len(counts), 4
    kw = dict(kw)
    dtype, bias = kw.pop("dtype", torch.bfloat16), kw.pop("bias", False)
    m = (sum(counts) + k - 1) // k + 3
    if m * k <= 4 * e:                               # enough slots for blocks of 128
        m = e + 1
    ids = _ids(counts, m, k, seed=1).to(d)
    g = torch.Generator(device=d).manual_seed(2)
    x = torch.randn(m, h, generator=g, device=d).to(dtype)
    tw = torch.rand(m, k, generator=g, device=d)
    w13, w2 = make_weights(h, i, e, device=d, seed=3)
    (w13, s13), (w2, s2) = quantize_fp8_block(w13), quantize_fp8_block(w2)
    kw.update(use_fp8_w8a8=True, w13_scale=s13, w2_scale=s2)
    if bias:
        kw.update(b13=torch.randn(e, 2 * i, generator=g, device=d) * 0.1, b2=torch.randn(e, h, generator=g, device=d) * 0.1)
    out = F.fused_experts(x, w13, w2, tw, ids, **kw)
    names = _lib.launch_stats()[1]
    assert "moe_gemm_fp8_mixed_kernel<gate/up>" in names and "group_quant_slots_kernel" in names, names
    assert ("finalize_pairs_kernel" in names) == (h > 512), names
    ref = F.fused_experts(x, w13, w2, tw, ids, block_tokens=16, **kw)
    F.check_status()
    err = ((out.float() - ref.float()).norm() / ref.float().norm()).item()
    assert torch.isfinite(out).all() and err <= 4e-3, err
    rows = (out.float() - ref.float()).flatten(0, -2).norm(dim=-1) / ref.float().flatten(0, -2).norm(dim=-1).clamp_min(1e-3)
    assert rows.max().item() <= 2e-2, rows.max().item()


@pytest.mark.parametrize("h,i,e,k,m", [(2048, 256, 16, 8, 640), (4096, 128, 16, 2, 1500)])
def test_routing_triple_of_many_pairs(cuda_device, h, i, e, k, m):
    """A call from a routing triple quantises its tokens into the activations' room (the second layer's activations have
    fewer bytes than its tokens) and gathers them: the same rows as the call from ids, and with pair rows the same bits."""
    d = cuda_device
    x, tw, ids = make_tokens(m, h, e, k, device=d, seed=6, skew=True)
    w13, w2 = make_weights(h, i, e, device=d, seed=7)
    (w13, s13), (w2, s2) = quantize_fp8_block(w13), quantize_fp8_block(w2)
    kw = dict(use_fp8_w8a8=True, w13_scale=s13, w2_scale=s2)
    ref = F.fused_experts(x, w13, w2, tw, ids, **kw)
    assert "finalize_pairs_kernel" in _lib.launch_stats()[1]
    order = torch.argsort(ids.flatten().long(), stable=True)
    triple = (torch.bincount(ids.flatten().long(), minlength=e).int(), order.int(), tw.flatten()[order], k)
    out = F.fused_experts(x, w13, w2, routing=triple, **kw)
    assert "gather_rows_kernel" in _lib.launch_stats()[1]
    F.check_status()
    assert torch.equal(out, ref)


@pytest.mark.parametrize("entry", ["ids", "int64 ids", "logits", "map", "logits and map"])
@pytest.mark.parametrize("h,i,e,k,m", [(512, 256, 32, 4, 250), (2048, 256, 64, 8, 700)])      # fp32 sums; pair rows
def test_hot_and_cold_blocks_against_the_oracle(cuda_device, h, i, e, k, m, entry):
    """The same launch against the fp32 evaluation on the CPU, from every form of the routing that it takes (the router's ids
    are replaced in place by the rows of the slots)."""
    d = cuda_device
    x, _, _ = make_tokens(m, h, e, k, seed=8)
    logits = torch.randn(m, e, generator=torch.Generator().manual_seed(9)) + zipf_bias(e, 1.1, seed=10)
    tw, ids = route(logits, k)
    w13, w2 = make_weights(h, i, e, seed=11)
    (w13, s13), (w2, s2) = quantize_fp8_block(w13), quantize_fp8_block(w2)
    counts = torch.bincount(ids.flatten().long(), minlength=e)
    assert (counts > 128).any() and ((counts > 0) & (counts <= 16)).any(), counts
    kw = dict(use_fp8_w8a8=True, w13_scale=s13.to(d), w2_scale=s2.to(d))
    ref_tw = tw
    if "map" in entry:
        emap = torch.arange(e, dtype=torch.int32)
        emap[1::3] = -1
        kw["expert_map"] = emap.to(d)
        ref_tw = torch.where(emap[ids.long()] >= 0, tw, torch.zeros_like(tw))
    if "logits" in entry:
        out = F.fused_moe(x.to(d), w13.to(d), w2.to(d), logits.to(d), k, **kw)
    else:
        ids_in = ids.long() if entry == "int64 ids" else ids
        out = F.fused_experts(x.to(d), w13.to(d), w2.to(d), tw.to(d), ids_in.to(d), **kw)
    names = _lib.launch_stats()[1]
    assert "moe_gemm_fp8_mixed_kernel<gate/up>" in names and ("finalize_pairs_kernel" in names) == (h == 2048), names
    F.check_status()
    assert_parity(out, OM.fused_experts_fp8(x, w13, w2, s13, s2, ref_tw, ids), what=f"fp8 mixed {(h, i, e, k, m)} {entry}")


@pytest.mark.parametrize("sms", [1, 2, 3])
@pytest.mark.parametrize("counts,h", [(EDGES, 512), ([130, 3, 140, 1, 5, 2, 9, 4], 512), ([9] * 8, 512)])
def test_few_sms(cuda_device, monkeypatch, sms, counts, h):
    """A call that is given a few SMs only (the configuration's num_sms): with one, no CTAs can be kept for cold blocks."""
    fused_moe = importlib.import_module("flaggems_sglang_b200.ops.fused_moe")
    d, i, e, k = cuda_device, 256, len(counts), 4
    m = max(4 * e // k + 1, (sum(counts) + k - 1) // k + 3)
    ids = _ids(counts, m, k, seed=1).to(d)
    g = torch.Generator(device=d).manual_seed(2)
    x = torch.randn(m, h, generator=g, device=d).to(torch.bfloat16)
    tw = torch.rand(m, k, generator=g, device=d)
    w13, w2 = make_weights(h, i, e, device=d, seed=3)
    (w13, s13), (w2, s2) = quantize_fp8_block(w13), quantize_fp8_block(w2)
    kw = dict(use_fp8_w8a8=True, w13_scale=s13, w2_scale=s2, block_tokens=128)
    ref = F.fused_experts(x, w13, w2, tw, ids, **kw)
    make_cfg = fused_moe._make_cfg

    def few(*args, **kwargs):
        cfg = make_cfg(*args, **kwargs)
        cfg.num_sms = sms
        return cfg

    monkeypatch.setattr(fused_moe, "_plans", {})
    monkeypatch.setattr(fused_moe, "_make_cfg", few)
    out = F.fused_experts(x, w13, w2, tw, ids, **kw)
    assert "moe_gemm_fp8_mixed_kernel<gate/up>" in _lib.launch_stats()[1]
    F.check_status()
    err = ((out.float() - ref.float()).norm() / ref.float().norm()).item()
    assert torch.isfinite(out).all() and err <= 4e-3, err
