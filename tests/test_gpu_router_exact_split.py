"""GPU: fp16 and bf16 rows of router_tc_k (tcgen05) with router weights of very different magnitudes: the terms of a weight hold all of its bits, however small it is beside its neighbours. The large weights meet
activations of zero, so that the logits are those of the small ones alone: 1e-6, 1e-9, 1e-25 of one weight of 1 in every 32 columns, and magnitudes spread from 1 down to 1e-12. Bounds as
for the plain case (test_gpu_router_tc.py): every product is exact, what is left is that the sums are cut off. bf16 with spread magnitudes: a few columns make up the sum, which then has
its full size for the rest of a part and not 2/3 of it on average: 3/2 of the plain case's 4.8e-7, bound 9e-7."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,bound", ((torch.bfloat16, 6e-7), (torch.float16, 1e-7)), ids=("bf16", "f16"))
@pytest.mark.parametrize("small", (1e-6, 1e-9, 1e-25, None))
@pytest.mark.parametrize("n,h,e", ((640, 1024, 256), (4096, 1056, 512)))        # a tile's columns split over a cluster; a block per tile, a last half step
def test_small_weights_beside_large_ones(dtype, bound, small, n, h, e):
    from tqllm_b200 import moe
    g = torch.Generator("cuda").manual_seed(n + h)
    w, x = torch.randn(e, h, generator=g, device="cuda"), torch.randn(n, h, generator=g, device="cuda").to(dtype)
    if small is None:
        w *= 10.0 ** (-12.0 * torch.rand(1, h, generator=g, device="cuda"))
        x[:, w.abs().amax(0) > 1e-7] = 0.
    else:
        w *= small
        w[:, ::32] = 1.
        x[:, ::32] = 0.
    if small is None and dtype == torch.bfloat16:
        bound = 9e-7
    want = x.double() @ w.double().T
    got = moe.router(w, x)[:, :e].double()
    assert float((got - want).norm() / want.norm()) < bound
