"""GPU: router_tc_k (many 16-bit rows, tcgen05) against fp64 where it begins and ends: rows around a tile of 128 with the gate in a tile of its own, ragged tokens, a last step of half a
step, one part of 512 columns and a ragged last one, more parts than a cluster splits, splits of one and two parts a block. Bounds (2-norm of the error over that of the logits):
a product that meets a sum of full size cuts off up to 2^-23 of it, half of that on average, and always towards zero. bf16: 32 such products a part,
whose sum grows as the square root, 2/3 of its end on average: 32 x 2^-24 x 2/3 = 1.3e-6 at most; half an ulp is 3/8 of a binade's mean, so 4.8e-7 is expected: bound 6e-7. fp16: two such
products a half step, and one rounding to nearest a step: 2 x 2^-24 x 3/4 = 8.9e-8, bound 1e-7 (one chain for a part has 4.7e-7)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,bound", ((torch.bfloat16, 6e-7), (torch.float16, 1e-7)), ids=("bf16", "f16"))
@pytest.mark.parametrize("n,h,e,gate", ((640, 768, 256, True), (700, 800, 255, True), (1025, 1056, 130, False), (321, 2048, 512, True), (2047, 512, 256, False), (2500, 3072, 127, True),
                                        (300, 4096, 300, False), (1200, 8736, 60, True), (9000, 1024, 49, True)))
def test_error_against_fp64(dtype, bound, n, h, e, gate):
    from tqllm_b200 import moe
    g = torch.Generator("cuda").manual_seed(n + h)
    w, v = torch.randn(e, h, generator=g, device="cuda") * 0.02, torch.randn(h, generator=g, device="cuda") * 0.02
    w[1] *= 1e-4 + torch.rand(h, generator=g, device="cuda") ** 8            # a row of very different magnitudes
    w[2] = 0.
    x = torch.randn(n, h, generator=g, device="cuda").to(dtype)
    rows = torch.cat([w, v[None]]) if gate else w
    want = x.double() @ rows.double().T
    got = moe.router(w, x, v if gate else None)[:, :rows.shape[0]].double()
    assert bool((got[:, 2] == 0).all())
    assert float((got - want).norm() / want.norm()) < bound
    assert float((got[:, 1] - want[:, 1]).norm() / want[:, 1].norm()) < 2 * bound


def test_a_bf16_nan_stays_in_its_token():
    from tqllm_b200 import moe
    g = torch.Generator("cuda").manual_seed(5)
    w, x = torch.randn(256, 1024, generator=g, device="cuda") * 0.02, torch.randn(600, 1024, generator=g, device="cuda").bfloat16()
    clean = moe.router(w, x)
    x[77, 1000] = float("nan")
    got = moe.router(w, x)
    assert bool(got[77, :256].isnan().all())
    keep = torch.arange(600, device="cuda") != 77
    assert torch.equal(got[keep], clean[keep])
