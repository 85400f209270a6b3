"""GPU: the int4 GEMMs where their tiles can go wrong -- odd numbers of quantisation groups (decode blocks take two at a
time), experts with no, one and ragged numbers of rows, the widest token tile, a reduction split over CTAs -- and the
16-bit pair kernel on the same ragged rows.  All against the oracle."""
import pytest
import torch

from oracle import moe as OM
from parity import assert_parity

pytestmark = pytest.mark.gpu


def _skewed(m, e, k, seed):
    """Routing that leaves the last expert empty and sends most tokens to the first."""
    g = torch.Generator().manual_seed(seed)
    logits = torch.randn(m, e, generator=g)
    logits[:, 0] += 2.0
    logits[:, e - 1] = -1e9
    w, ids = torch.topk(torch.softmax(logits, -1), k, -1)
    return w / w.sum(-1, keepdim=True), ids.to(torch.int32)


@pytest.mark.parametrize("h,i,e,k,m,bt", [
    (384, 640, 5, 2, 17, 16),      # three and five groups: a half-empty last unit
    (128, 128, 3, 1, 40, 32),      # a single group
    (640, 384, 5, 2, 37, 32),
    (256, 384, 4, 2, 193, 0),      # rows just above one 192-token tile
    (256, 1920, 3, 2, 400, 256),   # several tiles per expert, fifteen groups
    (384, 256, 6, 2, 64, 64),
])
def test_int4_ragged_tiles(cuda_device, h, i, e, k, m, bt):
    import flaggems_sglang_b200 as F
    from flaggems_sglang_b200.quant import quantize_awq, repack_awq_for_kernel
    g = torch.Generator().manual_seed(h + m)
    q1 = quantize_awq(torch.randn(e, h, 2 * i, generator=g) * 0.05)
    q2 = quantize_awq(torch.randn(e, i, h, generator=g) * 0.05)
    x = torch.randn(m, h, generator=g).to(torch.float16)
    tw, ids = _skewed(m, e, k, m)
    d = cuda_device
    p1, z1 = repack_awq_for_kernel(*[t.to(d) for t in q1])
    p2, z2 = repack_awq_for_kernel(*[t.to(d) for t in q2])
    args = (x.to(d), p1, p2, tw.to(d), ids.to(d))
    out = F.fused_experts(*args, use_int4_w4a16=True, w13_sz=z1, w2_sz=z2, block_tokens=bt)
    weighted = F.fused_experts(*args, use_int4_w4a16=True, w13_sz=z1, w2_sz=z2, block_tokens=bt,
                               apply_router_weight_on_input=True)
    F.check_status()
    assert_parity(out, OM.fused_experts_awq(x, *q1, *q2, tw, ids), rtol=2e-2, atol=2e-2, what=f"int4 {(h, i, e, k, m, bt)}")
    assert_parity(weighted, OM.fused_experts_awq(x, *q1, *q2, tw, ids, apply_router_weight_on_input=True), rtol=2e-2,
                  atol=2e-2, what=f"int4 weight on input {(h, i, e, k, m, bt)}")


@pytest.mark.parametrize("m,bt", [(40, 16), (40, 32), (40, 64), (1, 0)])
def test_int4_many_experts(cuda_device, m, bt):
    """More experts than any router here serves: the prefixes over them still fit beside the rings."""
    import flaggems_sglang_b200 as F
    from flaggems_sglang_b200.quant import quantize_awq, repack_awq_for_kernel
    from oracle import routing as R
    h, i, e, k = 256, 128, 5000, 2
    d = cuda_device
    g = torch.Generator(device=d).manual_seed(m + bt)
    q1 = quantize_awq(torch.randn(e, h, 2 * i, generator=g, device=d) * 0.05)
    q2 = quantize_awq(torch.randn(e, i, h, generator=g, device=d) * 0.05)
    p1, z1 = repack_awq_for_kernel(*q1)
    p2, z2 = repack_awq_for_kernel(*q2)
    x = torch.randn(m, h, generator=g, device=d).to(torch.float16)
    ids = torch.stack([torch.randperm(e, generator=g, device=d)[:k] for _ in range(m)]).sort(dim=1).values.cpu()
    ids[:, 0] = ids[:, 0] % 3                  # a few experts with many rows, the first ones
    ids[0, 1] = e - 1
    tw = torch.rand(m, k, generator=g, device=d).cpu()
    r = R.topk_to_routing(tw.numpy(), ids.numpy(), e)
    routing = tuple(torch.from_numpy(r[n]).to(d) for n in ("hist", "topk_indx", "gate_scal"))
    out = F.fused_experts(x, p1, p2, routing=(*routing, k), use_int4_w4a16=True, w13_sz=z1, w2_sz=z2, block_tokens=bt)
    F.check_status()
    ref = OM.fused_experts_awq(x.cpu(), *[t.cpu() for t in q1], *[t.cpu() for t in q2], tw, ids)
    assert_parity(out, ref, rtol=2e-2, atol=2e-2, what=f"int4 E=5000 M={m} BT={bt}")


@pytest.mark.parametrize("h,i,e,k,m,bt", [(264, 136, 5, 2, 33, 128), (512, 200, 3, 1, 257, 256), (128, 320, 6, 2, 900, 160)])
def test_pair_kernel_ragged_tiles(cuda_device, h, i, e, k, m, bt):
    import flaggems_sglang_b200 as F
    from flaggems_sglang_b200.testing import make_weights
    w13, w2 = make_weights(h, i, e, seed=m, scale=0.05)
    g = torch.Generator().manual_seed(m)
    x = torch.randn(m, h, generator=g).to(torch.bfloat16)
    tw, ids = _skewed(m, e, k, m + 1)
    d = cuda_device
    out = F.fused_experts(x.to(d), w13.to(d), w2.to(d), tw.to(d), ids.to(d), block_tokens=bt)
    F.check_status()
    assert_parity(out, OM.fused_experts(x, w13, w2, tw, ids), what=f"pairs {(h, i, e, k, m, bt)}")
