"""GPU: gate/up with the smallest workspace, where the grouped GEMM gathers token rows, against the same call with room for the rows in slot
order: the same fp16 rows in the same order, so the same bits. Every bank type, items of 64, 128 and 256 tokens, an odd number of
units and a last unit of one step, counts of rows that do not divide by the loaders' four, skipped assignments, a shared expert, an
expert with most of the tokens."""
import ctypes as C

import pytest
import torch

from tqllm_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout,types,hidden", (("codes", (12, 12, 12), 1280), ("codes", (21, 21, 21), 768), ("gguf", (21, 21, 21), 768),
                                                 ("codes", (23, 23, 20), 1280), ("codes", (20, 20, 20), 1344), ("codes", (323, 323, 323), 640)),
                         ids=("q4k", "iq3s", "iq3s-gguf", "iq4xs", "iq4nl", "nvfp4"))
@pytest.mark.parametrize("n,skip,skew,shared", ((3, 0., False, True), (77, .1, True, True), (331, .3, True, False), (1203, .05, False, True)))
def test_gathered_rows_change_no_bit(layout, types, hidden, n, skip, skew, shared):
    from tqllm_b200 import capi, moe
    experts, topk, ff = 16, 4, 512
    shape = synth.LayerShape("gather", hidden, experts, topk, ff, shared=shared, types=types)
    dev = moe.MoeLayer.from_synth(synth.make_layer(shape, 3, "cuda"), iq3s_layout=layout)
    x = synth.make_tokens(shape, n, 4, "cuda")
    g = torch.Generator().manual_seed(n)
    order = torch.rand(n, experts, generator=g)
    if skew:
        order[:, 11] -= 0.9                                # nearly every token's first expert
    ids = order.argsort(1)[:, :topk].to(torch.int32).contiguous()
    ids[torch.rand(n, topk, generator=g) < skip] = -1
    st = n if shared else 0
    plan = moe.dispatch(ids.cuda(), experts, st)
    slots = n * topk + st
    rows_bytes = lambda rows: -(-rows * hidden * 2 // 256) * 256 + -(-rows * 4 // 256) * 256          # the GEMM's own: fp16 rows and their scales
    small, large = capi.lib.b2moe_expert_workspace_bytes(dev.gate.type, n, hidden, capi.BF16), rows_bytes(slots) + 4 * slots
    assert small < large, "the smaller workspace has to be below the line"
    sh = [C.byref(b.c) for b in dev.sh[:2]] if shared else (None, None)
    out = []
    with capi.family("gemm"):
        for nbytes in (small, large):
            act, ws = torch.zeros(slots, ff, device="cuda"), torch.empty(nbytes, dtype=torch.uint8, device="cuda")
            capi.check(capi.lib.b2moe_expert_gateup_swiglu(C.byref(dev.gate.c), C.byref(dev.up.c), *sh, x.data_ptr(), capi.BF16, plan.buf.data_ptr(), n, topk,
                                                           st, act.data_ptr(), ws.data_ptr(), nbytes, torch.cuda.current_stream().cuda_stream), "gateup")
            assert int(plan.buf[3]) == 0, "a bounded wait ran out"
            out.append(act)
    assert torch.equal(out[0], out[1])
