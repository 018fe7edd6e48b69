"""Host arithmetic: workspace sizes grow with the batch, so that scratch sized once for the largest batch is accepted for every smaller
one; looked at where the kernels change over and where the dispatch blocks of 1,024 ids are all taken (148 of them: 151,552 ids)."""
import ctypes as C

import pytest

from tqllm_b200 import capi
from tqllm_b200.capi import lib

EDGES = sorted({max(1, e + d) for e in (1, 1024, 4096, 8192, 37888, 65536, 151552, 303104, 1 << 20, 5 << 20) for d in (-1025, -1, 0, 1, 33, 1025)})


@pytest.mark.parametrize("experts", (1, 8, 128, 512, 640, 900, 1000, 4096))
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
                 lambda n: lib.b2moe_expert_workspace_bytes(type_id, n, cols, capi.BF16),
                 lambda n: lib.b2moe_expert_slot_workspace_bytes(C.byref(bank), n, capi.F32)):
        sizes = [size(a // topk + 1) for a in EDGES]
        assert sizes == sorted(sizes) and sizes[0] > 0


def test_product_scratch_with_a_row_per_assignment():
    """never below the size that the products accept; for banks of 4-bit codes fp32 rows as two fp16 terms with their sub-block sums and a scale fit"""
    for type_id in (12, 20, 21, 23, 323, 0x1015):
        bank = capi.Bank(16, None, type_id, 60, 512, 1024)
        for dt in (capi.F32, capi.F16, capi.BF16):
            for rows in (1, 7, 600, 5000):
                size = lib.b2moe_expert_slot_workspace_bytes(C.byref(bank), rows, dt)
                assert size >= lib.b2moe_expert_workspace_bytes(type_id, rows, 1024, dt)
                if type_id in (12, 0x1015):
                    assert size >= rows * (1024 * (4 if dt == capi.F32 else 2) + 128 + 4)
    assert lib.b2moe_expert_slot_workspace_bytes(None, 4, 0) == 0 and lib.b2moe_expert_slot_workspace_bytes(C.byref(bank), 0, 0) == 0
    assert lib.b2moe_expert_slot_workspace_bytes(C.byref(bank), 4, 7) == 0


@pytest.mark.parametrize("gate,down,experts,topk,hidden,ff,shared", ((12, 12, 256, 8, 3072, 1536, 0), (0x1015, 0x1015, 512, 10, 2048, 512, 1), (12, 20, 128, 4, 1024, 512, 0),
                                                                     (12, 12, 60, 6, 2560, 768, 0), (12, 20, 48, 32, 4096, 64, 1), (323, 323, 512, 10, 2048, 512, 1)))
def test_layer_workspace(gate, down, experts, topk, hidden, ff, shared):
    """every batch up to past the lines of nine and 32 assignments per expert; where the exact form serves the down product its rows of two fp16 terms are in it"""
    L = capi.Layer(hidden=hidden, experts=experts, topk=topk, ff=ff, has_shared=shared)
    L.gate = L.up = capi.Bank(16, None, gate, experts, ff, hidden)
    L.down = capi.Bank(16, None, down, experts, hidden, ff)
    before = 0
    for n in range(1, 40 * experts // topk):
        v = capi.LayerWs()
        capi.check(lib.b2moe_layer_workspace(C.byref(L), n, C.byref(v)), "b2moe_layer_workspace")
        assert v.total >= before, n
        before = v.total
        if down in (12, 0x1015) and 9 * experts <= n * topk < (32 * experts if experts >= 128 else 1 << 30):
            assert v.total - v.expert_scratch >= n * (topk + shared) * (4 * ff + ff // 8 + 4)
