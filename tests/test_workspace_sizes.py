"""Host arithmetic: workspace sizes grow with the batch, so that scratch sized once for the largest batch is accepted for every smaller
one; looked at where the kernels change over and where the dispatch blocks of 1,024 ids are all taken (148 of them: 151,552 ids)."""
import ctypes as C

import pytest

from tqllm_b200 import capi
from tqllm_b200.capi import lib

EDGES = sorted({max(1, e + d) for e in (1, 1024, 8192, 37888, 65536, 151552, 303104, 1 << 20, 5 << 20) for d in (-1025, -1, 0, 1, 33, 1025)})


@pytest.mark.parametrize("experts", (1, 8, 128, 512, 900, 1000, 4096))
def test_dispatch_scratch(experts):
    sizes = [lib.b2moe_dispatch_workspace_bytes(experts, a) for a in EDGES]
    assert all(s % 16 == 0 and s >= 16 for s in sizes)
    assert sizes == sorted(sizes)


@pytest.mark.parametrize("type_id,experts,rows,cols", ((12, 256, 1536, 3072), (323, 512, 512, 2048), (20, 8, 64, 64), (0x1015, 512, 256, 256)))
@pytest.mark.parametrize("topk", (1, 8))
def test_product_scratch(type_id, experts, rows, cols, topk):
    bank = capi.Bank(16, None, type_id, experts, rows, cols)
    for size in (lambda n: lib.b2moe_expert_matvec_workspace_bytes(C.byref(bank), n, topk),
                 lambda n: lib.b2moe_expert_gemm_gateup_workspace_bytes(C.byref(bank), n, topk, capi.F16),
                 lambda n: lib.b2moe_expert_workspace_bytes(type_id, n, cols, capi.BF16)):
        sizes = [size(a // topk + 1) for a in EDGES]
        assert sizes == sorted(sizes) and sizes[0] > 0
