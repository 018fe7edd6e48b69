"""GPU: bf16 rows of 65 to 255 tokens where router_mma_k would have more than a block per SM: router_tc_k's fine form takes what costs fewer cycles there (bound 1e-7 of the 2-norm, derived in
test_gpu_router_tc.py), router_mma_k the rest (bound 3e-7: one truncation of at most 2^-23 of a growing sum for each of up to 2 x 5120 / 64 products in a chain, which errors of either sign of the
partial sums leave at 2.3e-7). Few and many rows, the gate as the last row, ragged tokens, one token more than a tile of 64. And rows of columns that a warp's sixteen do not divide evenly: the columns that a lane holds."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,e,gate,bound", ((65, 2048, 512, True, 1e-7), (77, 2048, 512, False, 1e-7), (128, 2048, 512, True, 1e-7), (129, 3072, 256, False, 1e-7), (255, 3072, 256, True, 1e-7),
                                              (200, 5120, 128, False, 3e-7), (255, 4096, 60, True, 3e-7), (193, 1056, 300, True, 3e-7), (255, 512, 512, False, 3e-7), (66, 256, 4000, False, 3e-7),
                                              (64, 2048, 512, True, 3e-7), (9, 48, 17, True, 3e-7), (33, 816, 40, False, 3e-7)))
def test_error_against_fp64(n, h, e, gate, bound):
    from tqllm_b200 import moe
    g = torch.Generator("cuda").manual_seed(n + h)
    w, v = torch.randn(e, h, generator=g, device="cuda") * 0.02, torch.randn(h, generator=g, device="cuda") * 0.02
    x = torch.randn(n, h, generator=g, device="cuda").bfloat16()
    rows = torch.cat([w, v[None]]) if gate else w
    want = x.double() @ rows.double().T
    got = moe.router(w, x, v if gate else None)[:, :rows.shape[0]].double()
    assert float((got - want).norm() / want.norm()) < bound
    again = moe.router(w, x, v if gate else None)[:, :rows.shape[0]].double()
    assert torch.equal(got, again)
