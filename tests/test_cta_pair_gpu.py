"""GPU: the 16-bit prefill GEMMs on CTA pairs (tcgen05.mma.cta_group::2, token blocks of 128 and more) against the
oracle and against the one-CTA-per-tile kernels, which blocks of 64 tokens run on.  Shapes with ragged numbers of rows
per expert, several n-tiles, ragged K, and the pair-row and fp32-atomic epilogues."""
import pytest
import torch

from oracle import moe as OM
from parity import assert_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,i,e,k,m,dtype", [(512, 384, 8, 2, 300, torch.bfloat16), (1024, 512, 4, 2, 1100, torch.bfloat16),
                                              (2048, 1024, 8, 2, 4800, torch.bfloat16), (520, 264, 3, 1, 700, torch.float16)])
def test_cta_pairs_match_oracle_and_single_cta(cuda_device, h, i, e, k, m, dtype):
    import flaggems_sglang_b200 as F
    from flaggems_sglang_b200 import _lib
    from flaggems_sglang_b200.testing import make_tokens, make_weights
    w13, w2 = make_weights(h, i, e, dtype=dtype, seed=h + m, scale=0.05)
    x, tw, ids = make_tokens(m, h, e, k, dtype=dtype, seed=h + m)
    d = cuda_device
    args = (x.to(d), w13.to(d), w2.to(d), tw.to(d), ids.to(d))
    single = F.fused_experts(*args, block_tokens=64)
    F.check_status()
    assert any("moe_gemm_tc_kernel" in n for n in _lib.launch_stats()[1]), _lib.launch_stats()[1]
    pair = F.fused_experts(*args, block_tokens=128)
    again = F.fused_experts(*args, block_tokens=128)
    torch.cuda.synchronize()
    F.check_status()
    assert any("tc2" in n for n in _lib.launch_stats()[1]), _lib.launch_stats()[1]
    ref = OM.fused_experts(x, w13, w2, tw, ids)
    assert_parity(pair, ref, what=f"cta pairs {(h, i, e, k, m)}")
    # the same products summed in the same order: wherever no atomics add, the bits agree
    if "finalize_pairs_kernel" in _lib.launch_stats()[1]:
        assert torch.equal(pair, single) and torch.equal(pair, again)
    else:       # fp32 atomics in another order, then one rounding to the 16-bit type: a unit in its last place
        ulp = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -10
        torch.testing.assert_close(pair.float(), single.float(), rtol=ulp, atol=1e-4)
