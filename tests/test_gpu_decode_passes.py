"""GPU: the 4-bit decode kernels where the form of a pass changes: experts that hold 1 .. 9 and 12 tokens in one launch (up to four
tokens share one product for both activation bytes, more take two; nine and twelve make a second pass), against the exact fp32
kernels. Bound: the activations' fixed point, 2^-15 of a row's largest value, through two products: 2e-3 of the RMS as in the
layer tests."""
import pytest
import torch

from tqllm_b200 import synth
from util import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("types,hidden,ff", (((12, 12, 12), 512, 256), ((21, 21, 21), 768, 512)), ids=("q4k", "iq3s"))
def test_passes_of_every_size(types, hidden, ff):
    from tqllm_b200 import capi, moe
    held = (4, 1, 9, 3, 5, 12, 2, 8, 6, 7)                     # tokens of each expert
    n, experts = sum(held), len(held)
    shape = synth.LayerShape("passes", hidden, experts, 1, ff, shared=True, types=types)
    dev = moe.MoeLayer.from_synth(synth.make_layer(shape, 3, "cuda"))
    x = synth.make_tokens(shape, n, 4, "cuda")
    ids = torch.repeat_interleave(torch.arange(experts), torch.tensor(held))[torch.randperm(n, generator=torch.Generator().manual_seed(1))]
    plan = moe.dispatch(ids.to(torch.int32).reshape(n, 1).cuda(), experts, n)
    out = {}
    for path in ("generic", "decode"):
        with capi.family(path):
            act = moe.expert_gateup_swiglu(dev.gate, dev.up, x, plan, dev.sh[0], dev.sh[1])
            y = moe.expert_down(dev.down, act, plan, dev.sh[2])
        assert int(plan.buf[3]) == 0, "a bounded wait ran out"
        out[path] = act.cpu().numpy(), y.cpu().numpy()
    for got, want in zip(out["decode"], out["generic"]):
        assert rel_err(got, want) <= 2e-3
