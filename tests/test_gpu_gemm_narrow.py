"""GPU: the grouped GEMM in launches of narrow items (up to 24 assignments per expert on average: two issuing warps, K split by chunks over the
halves and quarters of an accumulator) and in those with an odd number of 256-column chunks (one issuer). Experts with the token counts at which an
item changes its form, rows of K that end inside a chunk or a unit, against 64-bit sums. NVFP4 weights and bf16 rows are exact in fp16, so what is left is one
truncation of at most 2^-23 of a partial sum for each of K / 16 products, and the row scales' and the store's roundings: (K / 16 + 4) 2^-23 of the norm."""
import pytest
import torch

from tqllm_b200 import synth

pytestmark = pytest.mark.gpu
COUNTS = (1, 15, 16, 17, 32, 33, 64, 65, 0, 0, 2, 3)                # tokens of an expert: 20 on average


@pytest.mark.parametrize("rows", (16, 208))
@pytest.mark.parametrize("k", (256, 384, 512, 640, 768, 896, 1024))   # 1, 2, 2, 3, 3, 4, 4 chunks
def test_token_counts(k, rows):
    from tqllm_b200 import capi, moe
    g = torch.Generator(device="cuda")
    g.manual_seed(k + rows)
    e = len(COUNTS)
    bank = moe.DeviceBank(synth.NVFP4G, synth.quantize(synth.NVFP4G, torch.randn(e * rows, k, generator=g, device="cuda") * 0.02).reshape(-1), e, rows, k)
    ids = torch.repeat_interleave(torch.arange(e, device="cuda"), torch.tensor(COUNTS, device="cuda"))
    ids = ids[torch.randperm(ids.numel(), generator=g, device="cuda")].int().reshape(-1, 1)
    act = torch.randn(ids.numel(), k, generator=g, device="cuda").bfloat16().float()
    plan = moe.dispatch(ids, e)
    with capi.family("gemm"):
        y = moe.expert_down(bank, act, plan)
    assert int(plan.buf[3]) == 0, "a bounded wait ran out"
    w = bank.dequant().double().reshape(e, -1, k)[:, :rows]
    want = torch.einsum("ark,ak->ar", w[ids.flatten().long()], act.double())
    err = (y[:ids.numel()].double() - want).norm(dim=1) / want.norm(dim=1)
    assert float(err.max()) <= (k / 16 + 4) * 2.0 ** -23
