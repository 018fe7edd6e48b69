"""GPU: the selection of the register-resident top-k. A line that at least k keys reach, the keys above it ranked, and round by round where more than 32 keys reach the line: equal keys inside a
lane, across lanes and at the border of the selection, all keys equal, more experts selected than lanes have keys, logits whose probabilities underflow, infinities and NaN. Logits are multiples of 1 / 4 here, so
equal keys are equal logits and the order is known: larger logit first, lower index among equal ones. And the softmax's quotient against CUDA's division, to the bit."""
import ctypes
import os
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
LIB = os.path.join(HERE, "_build", "quotient_kernel.so")


def want_ids(logits, k):
    return torch.sort(-logits.double(), dim=1, stable=True).indices[:, :k].int()


@pytest.mark.parametrize("e", (1, 8, 31, 33, 100, 128, 129, 256, 300, 512))
@pytest.mark.parametrize("levels", (1, 3, 12, 60))                   # distinct logits: 1 = all equal
def test_order_with_equal_keys(e, levels):
    from tqllm_b200 import moe
    g = torch.Generator("cuda").manual_seed(e * 100 + levels)
    logits = torch.randint(0, levels, (40, e + 1), generator=g, device="cuda") * 0.25
    logits[7, : e // 2 + 1] = 20.0                                    # more than 32 equal keys at the top, or a few
    for k in sorted({1, min(e, 7), min(e, 10), min(e, 32)}):
        want = want_ids(logits[:, :e], k)
        ids, w, _ = moe.topk_softmax(logits, e, k)
        assert torch.equal(ids, want)
        p = torch.softmax(logits[:, :e].double(), 1).gather(1, want.long())
        assert float((w.double() - p / p.sum(1, keepdim=True)).abs().max()) <= 3e-6
        ids, w = moe.route_sigmoid(logits, e, k, norm=True)
        assert torch.equal(ids, want)
        p = torch.sigmoid(logits[:, :e].double()).gather(1, want.long())
        assert float((w.double() - p / p.sum(1, keepdim=True)).abs().max()) <= 3e-6


def test_bias_selects_and_does_not_weigh():
    from tqllm_b200 import moe
    g = torch.Generator("cuda").manual_seed(3)
    logits, bias = torch.randn(33, 257, generator=g, device="cuda"), torch.randn(256, generator=g, device="cuda")
    ids, w = moe.route_sigmoid(logits, 256, 8, bias=bias, norm=False)
    s = 1.0 / (1.0 + torch.exp(-logits[:, :256]))
    keys = torch.gather(s + bias, 1, ids.long())
    assert bool((keys[:, :-1] >= keys[:, 1:] - 1e-6).all()) and float((keys[:, -1:] - torch.sort(s + bias, dim=1, descending=True).values[:, 7:8]).abs().max()) <= 1e-6
    assert float((w - torch.gather(s, 1, ids.long())).abs().max()) <= 3e-7


def test_tiny_probabilities_infinities_and_nan():
    from tqllm_b200 import moe
    g = torch.Generator("cuda").manual_seed(4)
    logits = torch.randint(-8, 8, (8, 513), generator=g, device="cuda") * 0.25
    logits[0, :512] -= 100.0 * (torch.arange(512, device="cuda") > 3)         # all but four underflow in part
    logits[1, 5:512] = float("-inf")                                          # fewer than k keys above zero: the rest in the order of their indices
    logits[2, 100] = float("nan")
    logits[3, 200] = float("inf")
    ids, w, _ = moe.topk_softmax(logits, 512, 10)
    clean = [0, 1, 4, 5, 6, 7]
    assert torch.equal(ids[clean], want_ids(logits[:, :512], 10)[clean])
    assert bool(w[clean].isfinite().all()) and float((w[clean].sum(1) - 1).abs().max()) <= 1e-5
    assert bool(w[2].isnan().any()) and bool(w[3].isnan().any())
    for row in ids.tolist():
        assert len(set(row)) == 10 and min(row) >= 0 and max(row) < 512


def test_quotient_is_the_division():
    if not os.path.isfile(LIB):
        os.makedirs(os.path.dirname(LIB), exist_ok=True)
        subprocess.run(["nvcc", "-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                        os.path.join(HERE, "quotient_kernel.cu"), "-o", LIB], check=True)
    lib = ctypes.CDLL(LIB)
    lib.count_different.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
    g = torch.Generator("cuda").manual_seed(5)
    n = 1 << 25
    differ = torch.zeros(1, dtype=torch.int32, device="cuda")
    for low in (-100.0, -24.0, -1.0):
        a = torch.exp2(torch.rand(n, generator=g, device="cuda") * low).clamp(2.0 ** -100, 1.0)
        b = torch.exp2(torch.rand(n, generator=g, device="cuda") * 19.99)
        b = torch.where((b.view(torch.int32) & 0x7FFFFF) == 0x7FFFFF, torch.ones_like(b), b)
        assert lib.count_different(a.data_ptr(), b.data_ptr(), n, differ.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    assert int(differ) == 0
