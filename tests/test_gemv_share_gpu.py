"""Down projection of a handful of pairs from a share of the weights in shared memory (moe_gemv_down_share_kernel), at the
edges of the rule that picks it, against the grouped path on the same inputs.

Both keep the activations in 16 bits and add at most topk fp32 terms per output in some order, so they agree to a few
units of the 16-bit output: 4e-3 in the 2-norm."""
import pytest
import torch

import flaggems_sglang_b200 as F
from flaggems_sglang_b200 import _lib
from flaggems_sglang_b200.testing import make_tokens, make_weights
from oracle import moe as OM
from parity import assert_parity

pytestmark = pytest.mark.gpu
SHARE, PLAIN, EARLY = "moe_gemv_down_share_kernel<down>", "moe_gemv_down_kernel<down>", "plain, all loads early"


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm()).item()


# 148 CTAs: 16 rows each at 2368 and below; 190 KiB for the rows of every pair and their activations
@pytest.mark.parametrize("h,i,e,k,m,dtype,kernel", [
    (2048, 768, 64, 8, 1, torch.bfloat16, SHARE), (2368, 256, 64, 8, 1, torch.bfloat16, SHARE),
    (2376, 256, 64, 8, 1, torch.bfloat16, PLAIN), (2048, 856, 64, 8, 1, torch.float16, PLAIN),
    (2048, 808, 64, 8, 1, torch.float16, SHARE), (264, 136, 16, 2, 1, torch.bfloat16, SHARE),
    (1000, 520, 64, 8, 2, torch.bfloat16, SHARE), (40, 8, 64, 16, 1, torch.float16, SHARE),
    (2400, 520, 64, 4, 3, torch.bfloat16, PLAIN),
    # six slots of 256 elements for a warp of the other kernel, which then has them all in flight; seven and five
    (2048, 768, 64, 4, 1, torch.bfloat16, EARLY), (768, 2048, 64, 3, 1, torch.float16, EARLY),
    (2048, 512, 64, 7, 1, torch.bfloat16, SHARE), (2048, 768, 64, 3, 1, torch.bfloat16, SHARE),
    # the routing triple's counts, 128 experts at a time
    (264, 136, 129, 16, 1, torch.bfloat16, SHARE), (264, 136, 300, 8, 2, torch.float16, SHARE),
    # up kernel with six CTAs an SM, or not: 3671 to 5683 columns and at most two tokens take it (rows of six chunks: from 4737)
    (1000, 464, 64, 8, 1, torch.float16, SHARE), (768, 704, 64, 8, 1, torch.bfloat16, EARLY),
    (768, 712, 64, 8, 1, torch.bfloat16, EARLY), (1536, 600, 64, 8, 1, torch.bfloat16, SHARE),
    (1024, 512, 64, 8, 1, torch.bfloat16, SHARE), (1000, 456, 64, 8, 1, torch.float16, SHARE),
    (776, 296, 64, 8, 2, torch.bfloat16, SHARE), (2048, 736, 64, 8, 1, torch.bfloat16, SHARE),
])
@pytest.mark.parametrize("variant", ["plain", "triple", "no_combine", "bias", "nowhere", "on_input"])
def test_share_of_the_down_weights(cuda_device, h, i, e, k, m, dtype, kernel, variant):
    d = cuda_device
    w13, w2 = make_weights(h, i, e, dtype=dtype, device=d, seed=3)
    x, tw, ids = make_tokens(m, h, e, k, dtype=dtype, device=d, seed=4)
    kw = {}
    if variant == "no_combine":
        kw.update(no_combine=True)
    elif variant == "bias":
        g = torch.Generator(device=d).manual_seed(5)
        kw.update(b13=torch.randn(e, 2 * i, generator=g, device=d) * 0.1, b2=torch.randn(e, h, generator=g, device=d) * 0.1,
                  activation="swiglu_oai", swiglu_alpha=1.7, swiglu_limit=7.0)
    elif variant == "nowhere":
        ids[:, 0] = -1
    elif variant == "on_input":
        kw.update(apply_router_weight_on_input=True, routed_scaling_factor=2.5)
    if variant == "triple":
        order = torch.argsort(ids.flatten().long(), stable=True)
        kw.update(routing=(torch.bincount(ids.flatten().long(), minlength=e).int(), order.int(), tw.flatten()[order], k))
        out = F.fused_experts(x, w13, w2, **kw)
    else:
        out = F.fused_experts(x, w13, w2, tw, ids, **kw)
    if kernel == EARLY:                              # (for results by pair the other kernel has nothing in flight early)
        kernel = SHARE if variant == "no_combine" else PLAIN
    assert kernel in _lib.launch_stats()[1], _lib.launch_stats()[1]
    kw.pop("routing", None)
    ref = F.fused_experts(x, w13, w2, tw, ids, block_tokens=16, **kw)
    F.check_status()
    assert torch.isfinite(out).all() and _rel(out, ref) <= 4e-3


@pytest.mark.parametrize("h,i,e,k,m,dtype", [(2048, 768, 64, 8, 1, torch.bfloat16), (1000, 456, 64, 8, 2, torch.float16),
                                             (264, 136, 129, 16, 1, torch.bfloat16)])
def test_share_of_the_down_weights_against_the_oracle(cuda_device, h, i, e, k, m, dtype):
    w13, w2 = make_weights(h, i, e, dtype=dtype, seed=5)
    x, tw, ids = make_tokens(m, h, e, k, dtype=dtype, seed=6)
    out = F.fused_experts(*(t.to(cuda_device) for t in (x, w13, w2, tw, ids)))
    assert SHARE in _lib.launch_stats()[1]
    F.check_status()
    assert_parity(out, OM.fused_experts(x, w13, w2, tw, ids), what=f"share kernel {(h, i, e, k, m)}")
