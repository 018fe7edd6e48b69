"""GPU: the shares of small decode launches: passes on blocks of their own (the row tiles of a pass divided by its blocks leave a remainder), equal
shares again where a pass has more row tiles than one round, more passes than blocks and than 32 active experts. Against the exact fp32
kernels; bound as in test_gpu_layer.py (activations of 15 bits: 2e-3 of the output's RMS as the largest error)."""
import pytest
import torch

from tqllm_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("types", ((12, 12, 12), (21, 21, 21)), ids=("q4k", "iq3s"))
@pytest.mark.parametrize("hidden,ff,experts,topk,n", ((2048, 512, 64, 10, 1), (1024, 512, 32, 4, 3), (768, 1280, 70, 9, 5), (3072, 1536, 40, 8, 2), (2048, 256, 200, 6, 25)))
def test_shares(types, hidden, ff, experts, topk, n):
    from tqllm_b200 import capi, moe
    dev = moe.MoeLayer.from_synth(synth.make_layer(synth.LayerShape("few", hidden, experts, topk, ff, shared=n % 2 == 1, types=types), 3, "cuda"))
    x = synth.make_tokens(dev.shape, n, 4, "cuda")
    out = dev.forward(x)
    art = {k: v.clone() if torch.is_tensor(v) else v for k, v in dev.artefacts().items()}
    assert art["status"] == 0
    with capi.family("generic"):
        want = dev.forward(x)
    ref = dev.artefacts()
    for name in ("act", "y"):
        assert float((art[name] - ref[name]).abs().max() / ref[name].std()) <= 2e-3
    assert float((out - want).abs().max() / want.std()) <= 2e-3
    assert torch.equal(dev.forward(x), out)
