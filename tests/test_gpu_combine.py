"""GPU: the weighted sum over a token's slots where the groups of five slots that the kernel reads together begin and end, with
skipped slots (their rows hold NaN and must not be read into the sum) and the shared expert's row, against fp64. Bound: k + 1 terms
added in fp32, a rounding of at most 2^-24 each for the sum and the product: (k + 3) 2^-24 of the sum of the terms' magnitudes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", (1, 4, 5, 6, 10, 11))
@pytest.mark.parametrize("skip", (False, True))
def test_slot_groups(k, skip):
    from tqllm_b200 import moe
    n, h = 7, 516
    g = torch.Generator().manual_seed(k)
    y = torch.randn(n * k + n, h, generator=g)
    w, sw = torch.rand(n, k, generator=g), torch.rand(n, generator=g)
    ids = torch.randint(0, 9, (n, k), generator=g, dtype=torch.int32)
    if skip:
        ids[torch.rand(n, k, generator=g) < 0.4] = -1
        ids[2] = -1
        y[:n * k][ids.reshape(-1) < 0] = float("nan")
    got = moe.combine(y.cuda(), w.cuda(), n, k, h, n, sw.cuda(), ids.cuda()).cpu().double()
    rows = torch.where((ids >= 0)[..., None], y[:n * k].reshape(n, k, h), 0.).double() * w[..., None].double()
    shared = y[n * k:].double() * sw[:, None].double()
    bound = (k + 3) * 2.0 ** -24 * (rows.abs().sum(1) + shared.abs())
    assert bool(((got - rows.sum(1) - shared).abs() <= bound).all())
