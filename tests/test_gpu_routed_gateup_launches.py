"""GPU: which launches a layer of a few tokens makes, and that a wait that runs out in the gate/up launch that routes for itself (up to eight tokens) is reported in the plan's status word, the next call clean. The copy that is left out (harness hook,
a short limit) is the second of a warp: the down product of these shapes has one copy a warp, so the report can only be the gate/up launch's. One token more takes the routing launch: the same there."""
import pytest
import torch

from tqllm_b200 import synth
from make_golden import layer_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,launches", ((1, 4), (8, 4), (9, 5)))
@pytest.mark.parametrize("fmt", (synth.Q4_K, synth.IQ3_S))
def test_a_wait_that_runs_out_is_reported(fmt, n, launches):
    from tqllm_b200 import capi, moe
    shape = synth.LayerShape("routed-wait", 1024, 8, 1, 256, types=(fmt,) * 3)
    layer, x = layer_inputs(shape, 8, n, 77)
    dev = moe.MoeLayer.from_synth(layer, experts=8)
    xd = x.cuda()
    with capi.family("decode_kernels"):
        want = dev.forward(xd).clone()
        before = capi.lib.b2moe_harness_launches()
        assert torch.equal(dev.forward(xd), want)
        assert capi.lib.b2moe_harness_launches() - before == launches
        for _ in range(3):
            capi.lib.b2moe_harness_wait_probe(1, 2000)
            try:
                dev.forward(xd)
                torch.cuda.synchronize()
                assert dev.artefacts()["status"] == 3
            finally:
                capi.lib.b2moe_harness_wait_probe(-1, 0)
            assert torch.equal(dev.forward(xd), want)
            assert dev.artefacts()["status"] == 0


@pytest.mark.parametrize("experts,topk,n,launches", ((512, 10, 8, 4), (300, 13, 8, 4), (520, 2, 2, 5), (512, 10, 9, 5), (512, 33, 1, 5)))
def test_launches_of_a_layer(experts, topk, n, launches):
    """the self-routing launch up to eight tokens, 512 experts, 32 selections and 128 assignments; past them a routing launch more"""
    import dataclasses

    from tqllm_b200 import capi, moe
    shape = synth.LayerShape("routed", 512, experts, topk, 256, types=(synth.Q4_K,) * 3)
    layer = synth.make_layer(shape, 4, "cpu", experts=8)
    layer = dataclasses.replace(layer, router_w=torch.randn(experts, 512) * 0.05, raw=tuple(r.reshape(8, -1).repeat(-(-experts // 8), 1)[:experts].reshape(-1) for r in layer.raw))
    dev = moe.MoeLayer.from_synth(layer, experts=experts)
    x = torch.randn(n, 512, device="cuda").to({"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[shape.act_dtype])
    dev.forward(x)
    before = capi.lib.b2moe_harness_launches()
    dev.forward(x)
    assert capi.lib.b2moe_harness_launches() - before == launches
