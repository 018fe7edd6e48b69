"""GPU: router logits of fp16 and fp32 rows are as precise as a scalar fp32 loop. Bound on the relative error (2-norm over all logits) against
fp64: sums that round to nearest err by 2^-24 / sqrt(3) of the running sum per addition, and a running sum of m random terms has
on average half of the final variance: 2^-24 sqrt(m / 6). The longest chain, 8 additions per 256 columns and h / 256 of those sums, is m = 24 at
h = 4096; with the tensor core's own rounding of 16 products (at most 2^-23) and the result's: 2^-24 (sqrt(24 / 6) + 0.1) = 1.25e-7. A
chain of truncated sums, which this is to tell apart, has 1.6e-7 from h = 768 on."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", (torch.float16, torch.float32), ids=("f16", "f32"))
@pytest.mark.parametrize("n,h,e", ((7, 768, 100), (12, 2048, 100), (24, 3072, 60), (77, 4096, 70), (127, 2560, 60), (300, 2048, 512), (600, 4096, 512),
                                   (2048, 3072, 512), (300, 4000, 512)))
def test_error_against_fp64(dtype, n, h, e):
    from tqllm_b200 import moe
    g = torch.Generator("cuda").manual_seed(n + h)
    w = torch.randn(e, h, generator=g, device="cuda") * 0.02
    x = torch.randn(n, h, generator=g, device="cuda").to(dtype)
    want = x.double() @ w.double().T
    assert float((moe.router(w, x)[:, :e].double() - want).norm() / want.norm()) < 1.25e-7
