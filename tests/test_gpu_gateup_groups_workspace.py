"""GPU: the fused per-matrix gate/up call (groups in, typed rows out) with a workspace that has no room for the activation rows in slot order,
as its size was before those rows were part of it: accepted, and the same bits as with the full size, through the GEMM and
through the decode kernels; one byte less is refused."""
import ctypes as C

import pytest
import torch

from tqllm_b200 import synth

pytestmark = pytest.mark.gpu
up256 = lambda b: -(-b // 256) * 256


@pytest.mark.parametrize("types", ((12, 12, 12), (323, 323, 323)), ids=("q4k", "nvfp4"))
@pytest.mark.parametrize("family", ("auto", "gemm"))
@pytest.mark.parametrize("n", (5, 300))
def test_smaller_workspace(types, family, n):
    from tqllm_b200 import capi, moe
    lib, experts, topk, hidden, ff = capi.lib, 16, 4, 1024, 256
    shape = synth.LayerShape("groups", hidden, experts, topk, ff, types=types)
    dev = moe.MoeLayer.from_synth(synth.make_layer(shape, 3, "cuda"))
    x = synth.make_tokens(shape, n, 4, "cuda").half()
    ids = torch.rand(n, experts, generator=torch.Generator().manual_seed(n)).argsort(1)[:, :topk].to(torch.int32).contiguous().cuda()
    counts, groups = moe.plan_to_groups(moe.dispatch(ids, experts))
    a, s = n * topk, torch.cuda.current_stream().cuda_stream
    full = lib.b2moe_expert_gemm_gateup_workspace_bytes(C.byref(dev.gate.c), n, topk, capi.F16)
    small = full - (up256(up256(a * hidden * 2) + up256(a * 4) + a * 4) - up256(a * ff * 4))
    out = []
    with capi.family(family):
        for nbytes in (full, small):
            act, ws = torch.zeros(a, ff, dtype=torch.float16, device="cuda"), torch.empty(nbytes, dtype=torch.uint8, device="cuda")
            call = lambda room: lib.b2moe_expert_gemm_gateup(C.byref(dev.gate.c), C.byref(dev.up.c), x.data_ptr(), capi.F16, act.data_ptr(), capi.F16,
                                                             counts.data_ptr(), groups.data_ptr(), n, topk, ws.data_ptr(), room, s)
            capi.check(call(nbytes), "gateup")
            out.append(act)
        assert call(small - 256) == capi.ERR_WORKSPACE
    assert float(out[0].abs().sum()) > 0 and torch.equal(out[0], out[1])
