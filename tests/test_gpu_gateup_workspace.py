"""GPU: the gate/up product through the grouped GEMM with the smallest workspace (token rows gathered) and with the larger one (rows
in slot order, below and above the size from which they are converted once per token), with skipped assignments. Both read the same
fp16 rows in the same order, so the results are the same bits; the larger one is also held to the exact fp32 kernels (1e-2 of the RMS,
the bound of the GEMM tests)."""
import ctypes as C

import pytest
import torch

from tqllm_b200 import synth
from util import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", (33, 1500))
def test_both_forms(n):
    from tqllm_b200 import capi, moe
    experts, topk = 8, 3
    shape = synth.LayerShape("ws", 512, experts, topk, 256, shared=True, types=(12, 12, 12))
    dev = moe.MoeLayer.from_synth(synth.make_layer(shape, 3, "cuda"))
    x = synth.make_tokens(shape, n, 4, "cuda")
    g = torch.Generator().manual_seed(n)
    ids = torch.rand(n, experts, generator=g).argsort(1)[:, :topk].to(torch.int32)
    ids[torch.rand(n, topk, generator=g) < 0.2] = -1
    plan = moe.dispatch(ids.cuda(), experts, n)
    total = n * topk + n

    def gateup(nbytes):
        act = torch.zeros(total, shape.ff, device="cuda")
        ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        ref = lambda b: C.byref(b.c)
        capi.check(capi.lib.b2moe_expert_gateup_swiglu(ref(dev.gate), ref(dev.up), ref(dev.sh[0]), ref(dev.sh[1]), x.data_ptr(), capi.BF16,
                                                       plan.buf.data_ptr(), n, topk, n, act.data_ptr(), ws.data_ptr(), nbytes,
                                                       torch.cuda.current_stream().cuda_stream), "gateup")
        assert int(plan.buf[3]) == 0, "a bounded wait ran out"
        return act.cpu()

    size = lambda rows: capi.lib.b2moe_expert_workspace_bytes(12, rows, 512, capi.BF16)
    gemm_bytes = lambda rows: -(-rows * 512 * 2 // 256) * 256 + -(-rows * 4 // 256) * 256
    with capi.family("gemm"):
        small, large = gateup(size(n)), gateup(size(total) + 4 * total)
    assert size(n) < gemm_bytes(total) + 4 * total, "the smaller workspace has to be below the line"
    assert torch.equal(small, large)
    with capi.family("generic"):
        exact = moe.expert_gateup_swiglu(dev.gate, dev.up, x, plan, dev.sh[0], dev.sh[1])
    assert rel_err(large.numpy(), exact.cpu().numpy()) <= 1e-2
