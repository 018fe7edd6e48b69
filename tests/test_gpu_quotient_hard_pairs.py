"""GPU: the quotient of the routing's softmax against CUDA's division, to the bit, where it could go wrong if anywhere: quotients as near to the middle between two floats as 24-bit mantissas allow, and
divisors next to 2, whose reciprocals make the first quotient 1.5 ulp off."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def differ():
    import __graft_entry__ as entry
    lib = ctypes.CDLL(entry.kernel_path("quotient_kernel") if entry.kernel_is_current("quotient_kernel") else entry.build_test_kernel("quotient_kernel"))
    lib.count_different.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]

    def count(a, b):
        """pairs of mantissas (24-bit integers) whose quotients differ, the divisor times 2^0 and 2^18, the dividend below 1 and at 2^-100"""
        total = torch.zeros(1, dtype=torch.int32, device="cuda")
        for down, up in ((0, 0), (75, 18)):
            fa, fb = torch.ldexp(a.float(), torch.tensor(-24 - down, device="cuda")).contiguous(), torch.ldexp(b.float(), torch.tensor(-23 + up, device="cuda")).contiguous()
            assert lib.count_different(fa.data_ptr(), fb.data_ptr(), fa.numel(), total.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        return int(total)
    return count


def inverse_of_power(b, n):
    """2^-n modulo the odd b"""
    half, r = (b + 1) // 2, torch.ones_like(b)
    for _ in range(n):
        r = r * half % b
    return r


@pytest.mark.parametrize("below", (True, False), ids=("a<b", "a>=b"))
def test_next_to_the_middle(differ, below):
    """a 2^n = b (2 m + 1) + c, c = +- 1, 3, .. 9: a / b lies c / 2 b ulp from the middle"""
    b = torch.arange(2 ** 23 + 1, 2 ** 24 - 1, 2, dtype=torch.int64, device="cuda")
    inv = inverse_of_power(b, 25 if below else 24)
    pairs = 0
    for c in (-9, -7, -5, -3, -1, 1, 3, 5, 7, 9):
        a = c * inv % b
        if not below:
            a = a + b
        keep = (a >= 2 ** 23) & (a < 2 ** 24)
        pairs += int(keep.sum())
        assert differ(a[keep], b[keep]) == 0
    assert pairs > 5_000_000


def test_divisors_next_to_two(differ):
    a = torch.arange(2 ** 23, 2 ** 24, dtype=torch.int64, device="cuda")
    for b in (2 ** 24 - 2, 2 ** 24 - 3, 2 ** 24 - 5, 2 ** 24 - 7, 2 ** 24 - 9, 2 ** 24 - 11, 2 ** 24 - 101, 2 ** 24 - 4095, 2 ** 23 + 1, 2 ** 23 + 3, 11863283, 11863285):
        assert differ(a, torch.full_like(a, b)) == 0
