"""GPU: bf16 rows between one and two blocks per SM of router_mma_k with 17 to 48 router rows: router_tc_k sums half steps with compensation and is as exact as for fp16 rows (bound 1e-7 of the 2-norm,
derived in test_gpu_router_tc.py; router_mma_k has up to 2.7e-7 there, the chains of a part 4.7e-7). One part of 512 columns, less than one and a ragged last one, a last half step, one block per tile and clusters of one
and two parts a block, the gate as the last row, ragged tokens."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,e,gate", ((8192, 96, 24, False), (8192, 256, 24, False), (3000, 512, 17, False), (2047, 512, 47, True), (2600, 1056, 17, False), (1024, 2048, 48, False), (2047, 2048, 31, True),
                                        (1500, 3072, 33, False), (1499, 4096, 48, False), (1500, 5120, 20, True)))
def test_error_against_fp64(n, h, e, gate):
    from tqllm_b200 import moe
    g = torch.Generator("cuda").manual_seed(n + h)
    w, v = torch.randn(e, h, generator=g, device="cuda") * 0.02, torch.randn(h, generator=g, device="cuda") * 0.02
    w[1] *= 1e-4 + torch.rand(h, generator=g, device="cuda") ** 8
    x = torch.randn(n, h, generator=g, device="cuda").bfloat16()
    rows = torch.cat([w, v[None]]) if gate else w
    want = x.double() @ rows.double().T
    got = moe.router(w, x, v if gate else None)[:, :rows.shape[0]].double()
    assert float((got - want).norm() / want.norm()) < 1e-7
    assert float((got[:, 1] - want[:, 1]).norm() / want[:, 1].norm()) < 2e-7



def test_a_nan_stays_in_its_token():
    from tqllm_b200 import moe
    g = torch.Generator("cuda").manual_seed(5)
    w, x = torch.randn(48, 2048, generator=g, device="cuda") * 0.02, torch.randn(1024, 2048, generator=g, device="cuda").bfloat16()
    clean = moe.router(w, x)
    x[77, 1000] = float("nan")
    got = moe.router(w, x)
    assert bool(got[77, :48].isnan().all())
    keep = torch.arange(1024, device="cuda") != 77
    assert torch.equal(got[keep], clean[keep])
