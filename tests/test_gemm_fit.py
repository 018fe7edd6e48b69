"""Host arithmetic: the raw chunks that a block of the grouped GEMM holds, and the item sizes it keeps, over the number of experts. A line of the table is the last number of experts at which that many chunks still
fit beside the B stages, the decoders' tables, one unit's constants a decode warp (8 KB for Q4_K and IQ3_S codes) and 16 bytes an expert."""
import pytest

from tqllm_b200.capi import lib

Q4_K, IQ3_CODES = 12, 0x1015


@pytest.mark.parametrize("type_id,item,want", (
    (Q4_K, 256, ((805, 256, 4), (1957, 256, 3), (2597, 64, 6))), (Q4_K, 128, ((805, 128, 4), (1957, 128, 3), (2597, 64, 6))), (Q4_K, 64, ((2597, 64, 6), (3749, 64, 5))),
    (Q4_K, 32, ((2085, 32, 6), (3237, 32, 5), (4096, 32, 4))),
    (IQ3_CODES, 256, ((53, 256, 5), (1125, 256, 4), (2197, 256, 3), (3077, 64, 6))), (IQ3_CODES, 128, ((53, 128, 5), (1125, 128, 4), (2197, 128, 3))), (IQ3_CODES, 32, ((2565, 32, 6), (3637, 32, 5)))))
def test_raw_chunks(type_id, item, want):
    first = 1
    for last, tokens, chunks in want:
        for experts in (first, last):
            got = lib.b2moe_harness_gemm_fit(type_id, experts, item)
            assert (got >> 4, got & 15) == (tokens, chunks), experts
        first = last + 1
