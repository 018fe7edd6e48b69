"""GPU: the forms of the tensor-core routers and the rules between them. A token's logits have the same bits in every form of a kernel:
in router_mma_k whatever the number of tokens a block takes (8, 16, 32, 64), in router_tile_k (fp32; short fp16 rows: test_gpu_router_tiles.py) and
router_tc_k (16-bit rows) whether a tile's columns are split over a cluster (few tiles) or not. All are held to fp64, to 3e-6 of the largest logit as in test_gpu_routing.py, at the sizes where
they begin and end: one partial sum of 256 columns, several per block (more than 2048 columns), a ragged last one, ragged rows and tokens."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DTYPES = pytest.mark.parametrize("dtype", (torch.bfloat16, torch.float16, torch.float32), ids=("bf16", "f16", "f32"))


def inputs(n, h, e, dtype):
    g = torch.Generator("cuda").manual_seed(n * 3 + h + e)
    w, gate = torch.randn(e, h, generator=g, device="cuda") * 0.02, torch.randn(h, generator=g, device="cuda") * 0.02
    return w, gate, torch.randn(n, h, generator=g, device="cuda").to(dtype)


def held(w, gate, x):
    from tqllm_b200 import moe
    got = moe.router(w, x, gate)
    want = x.double() @ torch.cat([w, gate[None]]).double().T
    assert float((got - want).abs().max()) < 3e-6 * max(1.0, float(want.abs().max()))
    return got


@DTYPES
@pytest.mark.parametrize("h", (1024, 272))
def test_tokens_a_block(dtype, h):
    from tqllm_b200 import moe
    w, gate, x = inputs(64, h, 512, dtype)               # 33 tiles of rows, in clusters of four (h = 1024): one size a range of n
    full = held(w, gate, x)
    for n in (1, 8, 9, 16, 17, 32, 33):
        assert torch.equal(moe.router(w, x[:n].contiguous(), gate), full[:n])
    few = moe.router(w[:20].contiguous(), x, gate)        # two tiles of rows: eight tokens a block for all 64
    assert torch.equal(few[:, :20], full[:, :20]) and torch.equal(few[:, 20], full[:, 512])


@DTYPES
def test_small_routers_of_many_tokens(dtype):
    from tqllm_b200 import moe
    w, gate, x = inputs(700, 1024, 40, dtype)
    full = held(w, gate, x)
    if dtype != torch.bfloat16:                          # fp16 and fp32 rows leave router_mma_k only above two blocks per SM here
        assert torch.equal(moe.router(w, x[:9].contiguous(), gate), full[:9])


@DTYPES
@pytest.mark.parametrize("n,h,e", ((1950, 4000, 70), (300, 3072, 511), (300, 256, 32), (5000, 256, 129), (1300, 96, 512)))
def test_tiles_against_fp64(dtype, n, h, e):
    held(*inputs(n, h, e, dtype))


@DTYPES
@pytest.mark.parametrize("h", (3072, 992))
def test_split_tiles_give_the_bits_of_whole_ones(dtype, h):
    from tqllm_b200 import moe
    w, gate, x = inputs(2048, h, 511, dtype)              # 128 tiles: one block each
    full = held(w, gate, x)
    assert torch.equal(moe.router(w, x[:600].contiguous(), gate), full[:600])        # 40 tiles: split


@pytest.mark.parametrize("dtype", (torch.float16, torch.float32), ids=("f16", "f32"))
@pytest.mark.parametrize("n,h", ((65535 * 128 + 3, 32), (65535 * 64 + 3, 16)))
def test_more_tokens_than_a_grid_has_blocks(dtype, n, h):
    from tqllm_b200 import moe
    w, gate, x = inputs(1000, h, 3, dtype)
    many = x.repeat(-(-n // 1000), 1)[:n]
    got, want = moe.router(w, many, gate), x.double() @ torch.cat([w, gate[None]]).double().T
    assert float((got[-1003:-3] - want.roll(-((n - 1003) % 1000), 0)).abs().max()) < 3e-6
    assert float((got[:1000] - want).abs().max()) < 3e-6
