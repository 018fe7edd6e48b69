"""GPU: one arena for the largest batch: a layer call gives the same bits in it as in a workspace of its own batch's size, below and above the
densities where the products change over (nine and 32 assignments per expert), and where the arena ends just above such a line."""
import ctypes as C

import pytest
import torch

from tqllm_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("types,hidden,ff,experts,topk,sizes,largest", (((12, 12, 12), 256, 512, 128, 4, (280, 300, 900, 1000, 1023), 1024),
                                                                        ((21, 21, 21), 512, 512, 128, 8, (100, 150, 500), 513),
                                                                        ((12, 12, 20), 4096, 64, 48, 32, (13, 16, 40), 48)))
@pytest.mark.parametrize("dtype", (torch.bfloat16, torch.float32), ids=("bf16", "f32"))
def test_same_bits_in_a_larger_arena(types, hidden, ff, experts, topk, sizes, largest, dtype):
    from tqllm_b200 import capi, moe
    dev = moe.MoeLayer.from_synth(synth.make_layer(synth.LayerShape("arena", hidden, experts, topk, ff, types=types), 3, "cuda"))
    size = lambda n: (v := capi.LayerWs(), capi.check(capi.lib.b2moe_layer_workspace(C.byref(dev.c), n, C.byref(v)), "workspace"))[0].total
    code = capi.F32 if dtype == torch.float32 else capi.BF16
    for n in sizes:
        x = torch.randn(n, hidden, device="cuda", generator=torch.Generator("cuda").manual_seed(n)).to(dtype)
        outs = []
        for nbytes in (size(n), size(largest)):
            ws, out = torch.zeros(nbytes, dtype=torch.uint8, device="cuda"), torch.empty(n, hidden, device="cuda")
            capi.check(capi.lib.b2moe_layer_forward(C.byref(dev.c), x.data_ptr(), code, n, out.data_ptr(), capi.F32, ws.data_ptr(), nbytes,
                                                    torch.cuda.current_stream().cuda_stream), "forward")
            outs.append(out)
        assert float(outs[0].abs().sum()) > 0 and torch.equal(outs[0], outs[1]), n
