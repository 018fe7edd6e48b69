"""GPU: the down product of a layer call asks for its weights before the launches before it are done, the grouped GEMM's products read the plan before their rows are converted. Forward
passes launched back to back over other tokens, through one arena, give the bits of the separate entry points with a synchronisation after each of them, down to a first segment of fewer
copies than a ring holds (K = 256), blocks without work. (The decode kernels' early form: test_gpu_early_decode.py; here they meet up to three tokens, whose gate/up launch makes the plan, so that down waits.)"""
import dataclasses

import pytest
import torch

from tqllm_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", (synth.Q4_K, synth.IQ3_S, synth.NVFP4G, synth.IQ4_XS))
@pytest.mark.parametrize("hidden,ff,experts,topk,tokens", ((256, 256, 4, 1, 1), (512, 256, 9, 2, 70), (256, 1024, 200, 4, 3), (1024, 512, 8, 4, 300)))
def test_back_to_back_layers_equal_separate_steps(fmt, hidden, ff, experts, topk, tokens):
    from tqllm_b200 import moe
    shape = synth.LayerShape("early", hidden, experts, topk, ff, types=(fmt,) * 3, act_dtype="bf16")
    layer = synth.make_layer(shape, 3, "cpu", experts=min(experts, 8))
    if experts > 8:                                       # a bank of more experts repeats eight
        rep = -(-experts // 8)
        g = torch.Generator().manual_seed(1)
        layer = dataclasses.replace(layer, router_w=torch.randn(experts, hidden, generator=g) * 0.05,
                                    raw=tuple(r.reshape(8, -1).repeat(rep, 1)[:experts].reshape(-1) for r in layer.raw))
    dev = moe.MoeLayer.from_synth(layer, experts=experts)
    g = torch.Generator("cuda").manual_seed(7)
    xs = [torch.randn(tokens, hidden, generator=g, device="cuda").bfloat16() for _ in range(4)]
    outs = [torch.empty(tokens, hidden, device="cuda") for _ in xs]
    dev.reserve(tokens)
    for _ in range(3):
        for x, out in zip(xs, outs):
            dev.forward(x, out=out)
    torch.cuda.synchronize()
    for x, out in zip(xs, outs):
        logits = moe.router(dev.router_w, x)
        ids, w, _ = moe.topk_softmax(logits, experts, topk, shape.scale)
        plan = moe.dispatch(ids, experts)
        torch.cuda.synchronize()
        act = moe.expert_gateup_swiglu(dev.gate, dev.up, x, plan)
        torch.cuda.synchronize()
        y = moe.expert_down(dev.down, act, plan)
        torch.cuda.synchronize()
        assert torch.equal(out, moe.combine(y, w, tokens, topk, hidden))
