"""GPU: the grouped GEMM where its unit of two 64-column steps does not divide the rows: odd numbers of units, a last unit of one
step, several items per block, at the three item widths (64, 128, 256 tokens), rows in slot order and gathered. Against the
exact fp32 kernels of the library; bound as in test_gpu_gemm.py (weights and activations rounded to fp16: 1e-2 of the RMS)."""
import ctypes as C

import pytest
import torch

from tqllm_b200 import synth
from util import rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-2


@pytest.mark.parametrize("tokens", (20, 200, 900))      # 5, 50 and 225 tokens per expert
@pytest.mark.parametrize("types,hidden,ff", (((323, 323, 323), 2944, 384),      # 23 and 3 units
                                             ((23, 23, 20), 1280, 448),         # 10 units; 7 steps: a last unit of one step
                                             ((20, 20, 20), 1376 - 32, 1088)),  # 21 and 17 steps
                         ids=("nvfp4", "iq4xs-nl", "iq4nl"))
def test_ragged_units(types, hidden, ff, tokens):
    from tqllm_b200 import capi, moe
    shape = synth.LayerShape("units", hidden, 16, 4, ff, shared=True, types=types)
    dev = moe.MoeLayer.from_synth(synth.make_layer(shape, 5, "cuda"))
    x = synth.make_tokens(shape, tokens, 6, "cuda")
    out = {}
    for path in ("generic", "gemm"):
        with capi.family(path):
            out[path] = dev.forward(x).cpu().numpy()
        art = dev.artefacts()
        assert art["status"] == 0, "a bounded wait ran out"
    assert rel_err(out["gemm"], out["generic"]) <= TOL
    # the product alone with the smallest workspace has no room for the rows in slot order and gathers them
    plan = moe.dispatch(art["ids"].clone(), 16, tokens)
    slots, t = tokens * 4 + tokens, types[0]
    small = capi.lib.b2moe_expert_workspace_bytes(t, tokens, hidden, capi.BF16)
    assert small < slots * (2 * hidden + 8)
    act, ws = torch.zeros(slots, ff, device="cuda"), torch.empty(small, dtype=torch.uint8, device="cuda")
    ref = lambda b: C.byref(b.c)
    with capi.family("gemm"):
        capi.check(capi.lib.b2moe_expert_gateup_swiglu(ref(dev.gate), ref(dev.up), ref(dev.sh[0]), ref(dev.sh[1]), x.data_ptr(), capi.BF16, plan.buf.data_ptr(),
                                                       tokens, 4, tokens, act.data_ptr(), ws.data_ptr(), small, torch.cuda.current_stream().cuda_stream), "gateup")
    assert int(plan.buf[3]) == 0
    assert torch.equal(act, art["act"])
