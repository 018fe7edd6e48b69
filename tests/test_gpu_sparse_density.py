"""GPU: a caller that says how many of its assignments are live (an expert-parallel rank, which sees every token and owns a part of the
experts) gets the grouped GEMM's items for that density. The same 320 live assignments, padded with 14 skipped slots a token or not:
the same bits. 20 per expert make items of up to 64 tokens, so the 100 tokens of one expert are two items whose K is split; at the 160
per expert that the padded call seems to have they are one item, summed in another order."""
import ctypes as C

import pytest
import torch

from tqllm_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("types", ((323, 323, 323), (23, 23, 20)), ids=("nvfp4", "iq4"))
def test_padded_slots_change_no_bit(types):
    from tqllm_b200 import capi, moe
    n, experts, hidden, ff = 160, 16, 1024, 512
    shape = synth.LayerShape("sparse", hidden, experts, 2, ff, types=types)
    dev = moe.MoeLayer.from_synth(synth.make_layer(shape, 3, "cuda"))
    x = synth.make_tokens(shape, n, 4, "cuda")
    ids = torch.arange(n, device="cuda", dtype=torch.int32)[:, None] % 5 + torch.tensor([[1, 7]], device="cuda", dtype=torch.int32)
    ids[:100, 0] = 0                                       # one expert with 100 tokens
    ref, lib, got = lambda b: C.byref(b.c), capi.lib, []
    for topk in (2, 16):
        padded = torch.full((n, topk), -1, dtype=torch.int32, device="cuda")
        padded[:, :2] = ids
        plan = moe.dispatch(padded, experts)
        act, y = torch.zeros(n * topk, ff, device="cuda"), torch.zeros(n * topk, hidden, device="cuda")
        need = max(lib.b2moe_expert_workspace_bytes(types[0], n, hidden, capi.BF16), lib.b2moe_expert_workspace_bytes(types[2], n * topk, ff, capi.F32))
        ws = torch.empty(need + n * topk * (2 * hidden + 8) + 512, dtype=torch.uint8, device="cuda")
        tail, s = (ws.data_ptr(), ws.numel()), torch.cuda.current_stream().cuda_stream
        capi.check(lib.b2moe_expert_gateup_swiglu_sparse(ref(dev.gate), ref(dev.up), None, None, x.data_ptr(), capi.BF16, plan.buf.data_ptr(), n, topk, 0,
                                                         2 * n, act.data_ptr(), *tail, s), "gateup")
        capi.check(lib.b2moe_expert_down_sparse(ref(dev.down), None, act.data_ptr(), plan.buf.data_ptr(), n, topk, 0, 2 * n, y.data_ptr(), *tail, s), "down")
        assert int(plan.buf[3]) == 0
        got.append([t.reshape(n, topk, -1)[:, :2].clone() for t in (act, y)])
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
