"""FP8 layers of fewer than eight slots per expert: a token's terms are added in fp32, whatever block of tokens the call
takes.

All experts are one expert up to the sign of their down projection, and a token's weights nearly cancel: y of the single
expert (up to 1) comes from the oracle, the output is y * sum(+-weights), about 0.03 y.  Terms of 0.125 y rounded to bf16
one by one would be off by 2^-9 / sqrt(3) * 0.125 * sqrt(8) / 0.03 = 1.3e-2 in the 2-norm; fp32 sums leave the roundings of
the output and of the oracle's y, 1.1e-3 each, and e4m3 roundings of the activations that fall the other way."""
import pytest
import torch

import flaggems_sglang_b200 as F
from flaggems_sglang_b200 import _lib, ep
from flaggems_sglang_b200.quant import quantize_fp8_block
from flaggems_sglang_b200.testing import make_weights
from oracle import moe as OM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [176, 200, 255])      # of 256 experts, top-8: from 1408 slots on the down projection has many tiles
@pytest.mark.parametrize("entry", ["experts", "block 128", "expert parallel"])
def test_terms_are_added_in_fp32(cuda_device, m, entry):
    h, i, e, k, d = 7168, 2048, 256, 8, cuda_device
    w13, w2 = make_weights(h, i, 1, seed=1)
    (q13, s13), (q2, s2) = quantize_fp8_block(w13), quantize_fp8_block(w2)
    g = torch.Generator().manual_seed(2)
    x = torch.randn(m, h, generator=g).to(torch.bfloat16)
    # four even and four odd experts; half of the tokens share the first two, so that there are hot blocks too
    ids = torch.stack([torch.randperm(e // 2, generator=g)[:k] for _ in range(m)])
    ids[::2, 0], ids[::2, 1] = 0, 0
    ids = ids * 2 + torch.arange(k) % 2
    ids[::2, 2:][ids[::2, 2:] < 2] += 2
    sign = 1.0 - 2.0 * (torch.arange(k) % 2)
    tw = 0.125 + sign * (0.002 + 0.004 * torch.rand(m, k, generator=g))
    y = OM.fused_experts_fp8(x, q13, q2, s13, s2, torch.ones(m, 1), torch.zeros(m, 1, dtype=torch.int32)).float()
    ref = y * (tw * sign).sum(1, keepdim=True)

    q13, q2 = (t.to(d).expand(e, -1, -1).contiguous() for t in (q13, q2))
    q2.view(torch.uint8)[1::2] ^= 0x80               # the sign bit of e4m3
    s13, s2 = (t.to(d).expand(e, -1, -1).contiguous() for t in (s13, s2))
    x, tw, ids = x.to(d), tw.to(d), ids.to(torch.int32).to(d)
    if entry == "expert parallel":
        ctxs = ep.EpContext.emulate(1, m, h, i, k, e, e, d)
        try:
            out = torch.empty(m, h, dtype=x.dtype, device=d)
            for phase in (1, 2, 4):
                ctxs[0].forward(x, q13, q2, s13, s2, tw, ids, ep.plan_placement(e, 1), phases=phase, out=out)
            torch.cuda.synchronize()
            ctxs[0].check_status()
        finally:
            ep.EpContext.close_emulated(ctxs)
    else:
        out = F.fused_experts(x, q13, q2, tw, ids, use_fp8_w8a8=True, w13_scale=s13, w2_scale=s2,
                              block_tokens=128 if entry == "block 128" else 0)
        assert "finalize_kernel" in _lib.launch_stats()[1]
        F.check_status()
    err = ((out.float().cpu() - ref).norm() / ref.norm()).item()
    assert err <= 4e-3, err
