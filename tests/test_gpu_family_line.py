"""GPU: the line between the decode family and the grouped GEMM. Below it (fewer than 32 assignments per expert, or a bank of fewer than
128 experts) a call has the decode family's bits (the decode kernels', or at these densities for 4-bit codes those of the exact grouped
product) and at least their precision, from it on the GEMM's: the library's own choice is
compared, bit for bit, with either family forced. The decode kernels round the activations to 15 bits of a row's largest magnitude (about
four standard deviations of a normal row: 1e-4 of the values' RMS) and the weights not at all; the GEMM's 11 bits of both give at least 2.9e-4."""
import pytest
import torch

from tqllm_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("types,layout", (((12, 12, 12), "codes"), ((21, 21, 21), "codes"), ((21, 21, 21), "gguf")), ids=("q4k", "iq3s", "iq3s-gguf"))
@pytest.mark.parametrize("experts,per,family", ((128, 16, "decode"), (128, 31, "decode"), (128, 32, "gemm"), (127, 40, "decode"), (12, 300, "decode")))
def test_family_of_a_density(types, layout, experts, per, family):
    from tqllm_b200 import capi, moe
    topk = 4
    shape = synth.LayerShape("line", 512, experts, topk, 256, types=types)
    dev = moe.MoeLayer.from_synth(synth.make_layer(shape, 3, "cuda"), iq3s_layout=layout)
    x = synth.make_tokens(shape, -(-per * experts // topk), 4, "cuda")
    ids = torch.arange(x.shape[0] * topk, device="cuda", dtype=torch.int32).remainder(experts).reshape(-1, topk)
    plan = moe.dispatch(ids, experts)
    got = {}
    for name in ("auto", "decode", "gemm"):
        with capi.family(name):
            act = moe.expert_gateup_swiglu(dev.gate, dev.up, x, plan)
            got[name] = act, moe.expert_down(dev.down, act, plan)
    assert not torch.equal(got["decode"][0], got["gemm"][0])
    assert torch.equal(got["auto"][0], got[family][0]) and torch.equal(got["auto"][1], got[family][1])
    if family == "decode":
        w = [b.dequant().double().reshape(experts, b.rows, b.cols)[0] for b in (dev.gate, dev.up)]
        rows = (ids.reshape(-1) == 0).nonzero().flatten()
        g, u = (x[rows // topk].double() @ m.T for m in w)
        want = g * torch.sigmoid(g) * u
        assert float((got["auto"][0][rows].double() - want).norm() / want.norm()) < 1e-4
