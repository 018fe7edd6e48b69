"""GPU: bf16 logits of a few tokens on banks of more than 592 experts, where router_mma_k has more than a block per SM even for one token: its small instances cost less than the 64-token tiles of
router_tc_k there. A logit of router_mma_k has the same bits in any batch and beside any other rows, and banks of up to 512 experts are its own up to 64 tokens: so a large bank's logits are those of its parts.
Error against 64 bits: 3e-7 (one truncation of at most 2^-23 of a growing sum for each of up to 2 x 5120 / 64 products in a chain), 1e-7 where the fine form of router_tc_k is the cheaper one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def logits(n, h, e):
    from tqllm_b200 import moe
    g = torch.Generator("cuda").manual_seed(n + h + e)
    w, x = torch.randn(e, h, generator=g, device="cuda") * 0.02, torch.randn(n, h, generator=g, device="cuda").bfloat16()
    got = moe.router(w, x)[:, :e]
    parts = torch.cat([moe.router(w[i:i + 512].contiguous(), x)[:, :min(512, e - i)] for i in range(0, e, 512)], 1)
    want = x.double() @ w.double().T
    return got, parts, float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("e", (600, 1024, 1500))
@pytest.mark.parametrize("n,h", ((1, 1024), (1, 2048), (1, 5120), (7, 2048), (8, 3072), (9, 2048), (16, 4096)))
def test_few_tokens_take_the_small_instances(n, h, e):
    got, parts, error = logits(n, h, e)
    assert torch.equal(got, parts)
    assert error < 3e-7


@pytest.mark.parametrize("n,h,e", ((1, 2048, 4000), (17, 2048, 4000), (33, 2048, 2048), (64, 3072, 1024)))
def test_fine_form_where_it_is_cheaper(n, h, e):
    got, parts, error = logits(n, h, e)
    assert not torch.equal(got, parts) and error < 1e-7
