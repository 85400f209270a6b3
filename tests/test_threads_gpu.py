"""Host threads, each with a stream of its own, serve two layers whose kernels are the same and whose shared memory is not.

The shared memory a kernel may be given is one setting per kernel and device: a call that lowers it to its own size
between another thread's setting and launch makes that launch fail."""
import sys
import threading

import pytest
import torch

import flaggems_sglang_b200 as F
from flaggems_sglang_b200 import _lib
from flaggems_sglang_b200.quant import quantize_fp8_block
from flaggems_sglang_b200.testing import make_tokens, make_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,kernel,layers", [       # h, i, e, k, m of the two layers
    ("bf16", "moe_gemv_down_share_kernel<down>", [(2048, 768, 16, 8, 1), (512, 256, 16, 8, 1)]),
    ("bf16", "moe_gemv_down_kernel<down>", [(4096, 2048, 8, 8, 1), (4096, 256, 8, 2, 1)]),
    ("bf16", "moe_gemm_tc_kernel<down>", [(512, 256, 8, 2, 40), (512, 256, 200, 2, 150)]),
    ("fp8", "moe_gemm_fp8_kernel<down>", [(512, 256, 8, 2, 8), (512, 256, 200, 2, 150)]),
    ("fp8", "moe_gemm_fp8_mixed_kernel<down>", [(512, 256, 8, 2, 300), (512, 256, 300, 8, 300)]),
])
def test_threads_share_kernels(cuda_device, kind, kernel, layers):
    d, errors, worst = cuda_device, [], []
    calls = []
    for n, (h, i, e, k, m) in enumerate(layers):
        x, tw, ids = make_tokens(m, h, e, k, device=d, seed=n)
        w13, w2 = make_weights(h, i, e, device=d, seed=2 + n)
        kw = {}
        if kind == "fp8":
            (w13, s13), (w2, s2) = quantize_fp8_block(w13), quantize_fp8_block(w2)
            kw = dict(use_fp8_w8a8=True, w13_scale=s13, w2_scale=s2)
        calls.append(lambda x=x, w13=w13, w2=w2, tw=tw, ids=ids, kw=kw: F.fused_experts(x, w13, w2, tw, ids, **kw))
        ref = calls[-1]()
        assert kernel in _lib.launch_stats()[1], _lib.launch_stats()[1]
        calls[-1] = (calls[-1], ref)
    torch.cuda.synchronize()
    F.release_workspaces()                    # four streams to come, all with room of their own
    calls *= 2
    start = threading.Barrier(len(calls))

    def serve(call, ref):
        try:
            with torch.cuda.device(d), torch.cuda.stream(torch.cuda.Stream(d)):
                start.wait()
                for _ in range(12000):
                    out = call()
                torch.cuda.current_stream().synchronize()
                worst.append(((out.float() - ref.float()).norm() / ref.float().norm()).item())
        except Exception as exc:      # noqa: BLE001  (reported by the test's own thread)
            errors.append(exc)

    threads = [threading.Thread(target=serve, args=c) for c in calls]
    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-5)
    try:
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(interval)
    assert not errors, errors
    assert max(worst) <= 2e-3, worst          # fp32 sums in another order, rounded to 16 bits
    F.check_status()
