"""GPU: the gate/up launch of up to eight tokens that routes for itself gives what the separate launches give: ids, weights, every part of the plan, the output's bits. At the ends of the
number of experts a lane keeps (128, 256, 512) and past them, one and many selections, ties (equal logits: the lowest indices of every token, one expert with all of them), a shared expert with and without
its gate, sigmoid routing with a bias, rows of all types; and one token more, which takes the routing launch."""
import dataclasses

import pytest
import torch

from tqllm_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", (synth.Q4_K, synth.IQ3_S))
@pytest.mark.parametrize("experts,topk,n,gating,shared,gated,dtype,ties", (
    (8, 2, 1, 1, False, False, "f32", False), (32, 4, 7, 1, False, False, "f32", False), (128, 8, 8, 2, True, False, "bf16", False), (129, 3, 5, 1, True, True, "f16", False),
    (256, 8, 3, 2, False, False, "bf16", True), (300, 16, 8, 1, True, True, "bf16", True), (512, 10, 1, 1, True, False, "bf16", False), (512, 10, 8, 1, True, True, "bf16", False),
    (520, 2, 2, 1, False, False, "bf16", False), (512, 10, 9, 1, True, False, "bf16", False)))
def test_equals_the_separate_launches(fmt, experts, topk, n, gating, shared, gated, dtype, ties):
    from tqllm_b200 import moe
    hidden, ff = 512, 256
    shape = synth.LayerShape("routed", hidden, experts, topk, ff, gating=gating, shared=shared, types=(fmt,) * 3, act_dtype=dtype, sel_bias=gating == 2)
    layer = synth.make_layer(shape, 4, "cpu", experts=8)
    g = torch.Generator().manual_seed(experts + n)
    layer = dataclasses.replace(layer, router_w=torch.zeros(experts, hidden) if ties else torch.randn(experts, hidden, generator=g) * 0.05,
                                sel_bias=torch.randn(experts, generator=g) * 0.01 if gating == 2 and not ties else torch.zeros(experts) if gating == 2 else None,
                                raw=tuple(r.reshape(8, -1).repeat(-(-experts // 8), 1)[:experts].reshape(-1) for r in layer.raw))
    vec = torch.randn(hidden, generator=g) * 0.05 if gated else None
    dev = moe.MoeLayer.from_synth(layer, experts=experts, shared_gate_vec=vec)
    x = torch.randn(n, hidden, generator=g).to({"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[dtype]).cuda()
    for _ in range(2):
        out = dev.forward(x)
    torch.cuda.synchronize()
    art = dev.artefacts()
    logits = moe.router(dev.router_w, x, vec.cuda() if gated else None)
    sw = None
    if gating == 1:
        ids, w, sw = moe.topk_softmax(logits, experts, topk, shape.scale, shared=gated)
    else:
        ids, w = moe.route_sigmoid(logits, experts, topk, dev.sel_bias, shape.norm, shape.scale)[:2]
    plan = moe.dispatch(ids, experts, n if shared else 0)
    torch.cuda.synchronize()
    na = plan.n_active
    assert art["n_active"] == na and art["status"] == 0
    assert torch.equal(art["ids"], ids) and torch.equal(art["weights"], w)
    for name in ("counts", "offsets", "perm"):
        assert torch.equal(art[name][:getattr(plan, name).numel()], getattr(plan, name)), name
    assert torch.equal(art["active"][:na], plan.active[:na]) and torch.equal(art["passes"][:na + 1], plan.passes[:na + 1])
    if gated:
        assert torch.equal(art["shared_weights"], sw)
    act = moe.expert_gateup_swiglu(dev.gate, dev.up, x, plan, *(dev.sh[:2] if shared else ()))
    y = moe.expert_down(dev.down, act, plan, dev.sh[2] if shared else None)
    assert torch.equal(out, moe.combine(y, w, n, topk, hidden, n if shared else 0, shared_weights=sw))
