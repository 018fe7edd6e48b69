"""GPU: infinities and NaN in fp16 and fp32 router inputs give what a plain fp32 loop gives, in every form of the kernels: one infinite
activation makes logits infinite with the signs of its weights, two that disagree or a NaN make NaN, and other tokens do not notice.
Also the largest fp32 values, which round to infinity as bf16."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", (torch.float16, torch.float32), ids=("f16", "f32"))
@pytest.mark.parametrize("n,h,e", ((7, 256, 20), (40, 1024, 300), (600, 2304, 511), (2048, 768, 511), (9, 40, 20)))
def test_like_a_plain_loop(dtype, n, h, e):
    from tqllm_b200 import moe
    g = torch.Generator("cuda").manual_seed(n + h)
    w, gate = torch.randn(e, h, generator=g, device="cuda") * 0.02, torch.randn(h, generator=g, device="cuda") * 0.02
    w[::3] = w[::3].bfloat16().float()                     # exact as one bf16 term: the others are zero
    x = torch.randn(n, h, generator=g, device="cuda").to(dtype)
    clean = moe.router(w, x, gate)
    inf = float("inf")
    x[1, 5], x[2, h - 1], x[3, 0], x[3, 1], x[4, 17] = inf, -inf, inf, -inf, float("nan")
    if dtype == torch.float32:
        x[5] = 0.
        x[5, 3] = torch.finfo(torch.float32).max
    got, rows = moe.router(w, x, gate), torch.cat([w, gate[None]])
    assert torch.equal(got[1], rows[:, 5].sign() * inf) and torch.equal(got[2], rows[:, h - 1].sign() * -inf)
    both = rows[:, 0].sign() == rows[:, 1].sign()         # inf w0 - inf w1: NaN where the signs agree
    assert torch.equal(got[3].isnan(), both) and bool(got[4].isnan().all())
    same = [0] + list(range(6 if dtype == torch.float32 else 5, n))
    assert torch.equal(got[same], clean[same])
    if dtype == torch.float32:
        assert torch.equal(got[5], rows[:, 3] * x[5, 3])
