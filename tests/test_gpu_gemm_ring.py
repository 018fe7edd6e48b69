"""GPU: the raw ring of the grouped GEMM with an odd number of slots (IQ4 banks at 256 tokens per item: three), whose chunks the two groups
of decode warps take in turn: the same bits every time. A ring whose barriers the groups shared let a group read a slot before
its chunk had arrived, once in about ten calls."""
import ctypes as C

import pytest
import torch

from tqllm_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("types,hidden,ff,tokens", (((20, 20, 20), 1344, 1088, 900), ((23, 23, 20), 4096, 1408, 900), ((20, 20, 20), 1344, 1088, 200)))
def test_same_bits_every_time(types, hidden, ff, tokens):
    from tqllm_b200 import capi, moe
    shape = synth.LayerShape("ring", hidden, 16, 4, ff, shared=True, types=types)
    dev = moe.MoeLayer.from_synth(synth.make_layer(shape, 5, "cuda"))
    x = synth.make_tokens(shape, tokens, 6, "cuda")
    with capi.family("generic"):
        exact = dev.forward(x)
    with capi.family("gemm"):
        first = dev.forward(x)
        assert float((first - exact).abs().max() / exact.std()) < 2e-2
        for _ in range(60):
            assert torch.equal(dev.forward(x), first)
    assert dev.artefacts()["status"] == 0
