"""GPU: the decode kernels' down product that asks for its weights, and reads the plan, before the launches before it are done. Forward passes launched back to back over other tokens, through one arena, give the
bits of the separate entry points with a synchronisation after each of them: rows staged inside the kernel (few jobs; K = 256, a first segment of fewer copies than a ring holds, and 1024), rows staged by a
launch (many jobs: a short first segment, a long one, one active expert more than a probe round), a shared expert. The number of launches says which way the rows went (5: inside, 6: by a launch); Q4_K's large
launches wait first, and have to agree all the same."""
import dataclasses

import pytest
import torch

from tqllm_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", (synth.Q4_K, synth.IQ3_S))
@pytest.mark.parametrize("hidden,ff,experts,topk,tokens,shared,launches", ((256, 256, 64, 4, 12, False, 5), (512, 1024, 64, 2, 9, True, 5), (512, 256, 128, 8, 70, False, 6), (2048, 1024, 128, 8, 70, True, 6),
                                                                           (768, 512, 33, 4, 64, False, 6)))
def test_back_to_back_layers_equal_separate_steps(fmt, hidden, ff, experts, topk, tokens, shared, launches):
    from tqllm_b200 import capi, moe
    shape = synth.LayerShape("early", hidden, experts, topk, ff, shared=shared, types=(fmt,) * 3, act_dtype="bf16")
    layer = synth.make_layer(shape, 3, "cpu", experts=8)
    rep, g = -(-experts // 8), torch.Generator().manual_seed(1)
    layer = dataclasses.replace(layer, router_w=torch.randn(experts, hidden, generator=g) * 0.05, raw=tuple(r.reshape(8, -1).repeat(rep, 1)[:experts].reshape(-1) for r in layer.raw))
    dev = moe.MoeLayer.from_synth(layer, experts=experts)
    g = torch.Generator("cuda").manual_seed(7)
    xs = [torch.randn(tokens, hidden, generator=g, device="cuda").bfloat16() for _ in range(4)]
    outs = [torch.empty(tokens, hidden, device="cuda") for _ in xs]
    dev.reserve(tokens)
    before = capi.lib.b2moe_harness_launches()
    for _ in range(3):
        for x, out in zip(xs, outs):
            dev.forward(x, out=out)
    torch.cuda.synchronize()
    assert capi.lib.b2moe_harness_launches() - before == 12 * launches
    for x, out in zip(xs, outs):
        logits = moe.router(dev.router_w, x)
        ids, w, _ = moe.topk_softmax(logits, experts, topk, shape.scale)
        plan = moe.dispatch(ids, experts, tokens if shared else 0)
        torch.cuda.synchronize()
        act = moe.expert_gateup_swiglu(dev.gate, dev.up, x, plan, *(dev.sh[:2] if shared else ()))
        torch.cuda.synchronize()
        y = moe.expert_down(dev.down, act, plan, dev.sh[2] if shared else None)
        torch.cuda.synchronize()
        assert torch.equal(out, moe.combine(y, w, tokens, topk, hidden, tokens if shared else 0))
