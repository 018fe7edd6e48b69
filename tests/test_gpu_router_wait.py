"""GPU: a wait of router_tc_k (tcgen05) that runs out ends in logits all the same, summed in a plain loop: the copies of one step are left out (harness hook), at a block per tile and at a cluster's
split, for bf16 rows, bf16 rows on the fine sums and fp16 rows; the next launch is clean. Bound: 3e-6 of the largest logit as in test_gpu_routing.py."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,n,h,e", ((torch.bfloat16, 2500, 512, 200), (torch.bfloat16, 300, 2048, 256), (torch.bfloat16, 1024, 2048, 48), (torch.bfloat16, 3000, 512, 17),
                                         (torch.float16, 2500, 768, 100), (torch.float16, 300, 2048, 256)))
@pytest.mark.parametrize("step", (0, 5))
def test_logits_after_a_wait_that_runs_out(dtype, n, h, e, step):
    from tqllm_b200 import capi, moe
    g = torch.Generator("cuda").manual_seed(n + h)
    w, v = torch.randn(e, h, generator=g, device="cuda") * 0.02, torch.randn(h, generator=g, device="cuda") * 0.02
    x = torch.randn(n, h, generator=g, device="cuda").to(dtype)
    clean = moe.router(w, x, v)
    want = x.double() @ torch.cat([w, v[None]]).double().T
    capi.lib.b2moe_harness_wait_probe(step, 0)
    try:
        got = moe.router(w, x, v)
        torch.cuda.synchronize()
    finally:
        capi.lib.b2moe_harness_wait_probe(-1, 0)
    assert not torch.equal(got, clean)                    # the sums are the plain loop's
    assert float((got - want).abs().max()) < 3e-6 * max(1.0, float(want.abs().max()))
    assert torch.equal(moe.router(w, x, v), clean)
