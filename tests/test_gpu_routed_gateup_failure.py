"""GPU: a wait that runs out in the gate/up launch that routes for itself (up to eight tokens) is reported in the plan's status word, and the next call is clean. The copy that is left out (harness hook,
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
