"""GPU: router_tile_k at more than two blocks per SM of router_mma_k, where it still serves: fp32 rows, and fp16 rows below 768 columns. A tile's columns split over a cluster (fewer than 100 tiles) give
the bits of whole ones; both are held to fp64 (3e-6 of the largest logit, as in test_gpu_routing.py). Two partial sums of 256 columns, a ragged second one, one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", (torch.float16, torch.float32), ids=("f16", "f32"))
@pytest.mark.parametrize("h", (512, 320, 256))
def test_split_tiles_give_the_bits_of_whole_ones(dtype, h):
    from tqllm_b200 import moe
    g = torch.Generator("cuda").manual_seed(h)
    w, gate = torch.randn(511, h, generator=g, device="cuda") * 0.02, torch.randn(h, generator=g, device="cuda") * 0.02
    x = torch.randn(2048, h, generator=g, device="cuda").to(dtype)
    full, want = moe.router(w, x, gate), x.double() @ torch.cat([w, gate[None]]).double().T      # 128 tiles: one block each
    assert float((full - want).abs().max()) < 3e-6 * max(1.0, float(want.abs().max()))
    assert torch.equal(moe.router(w, x[:1300].contiguous(), gate), full[:1300])                  # 88 tiles: split
