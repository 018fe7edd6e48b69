"""GPU: the routing launch of a layer call stages the input rows for the 4-bit decode kernels only where gate/up runs on them. From nine
assignments per expert on it does not: the bytes of the expert scratch beyond what the down product's rows take stay as they were."""
import ctypes as C

import pytest
import torch

from tqllm_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("types", ((12, 12, 12), (21, 21, 21)), ids=("q4k", "iq3s"))
@pytest.mark.parametrize("n,staged", ((32, True), (12, True), (36, False), (40, False), (90, False)))
def test_staged_rows(types, n, staged):
    from tqllm_b200 import capi, moe
    hidden, ff, experts, topk = 2048, 256, 8, 2
    dev = moe.MoeLayer.from_synth(synth.make_layer(synth.LayerShape("staging", hidden, experts, topk, ff, types=types), 3, "cuda"))
    x = synth.make_tokens(dev.shape, n, 4, "cuda")
    dev.reserve(n)
    dev.ws.fill_(0x5A)
    out = dev.forward(x)
    assert dev.artefacts()["status"] == 0
    down_rows = n * topk * (ff * 4 + ff // 8 + 4) + 512
    rest = dev.ws[dev.ws_view.expert_scratch + down_rows:dev.ws_view.expert_scratch + n * hidden * 2]
    assert rest.numel() > n * hidden // 2 and bool((rest != 0x5A).any()) == staged
    with capi.family("generic"):
        want = dev.forward(x)
    assert float((out - want).abs().max() / want.std()) <= 2e-3
