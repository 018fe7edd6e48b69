"""GPU: precision of the grouped GEMM in launches of narrow items, whose K is split over the two issuers' chunks. Reference: the same experts in a launch of wide items (more than 24
assignments per expert), which splits their K over even and odd products, at the same numbers of products. Weights and activations are exact in fp16 (NVFP4, IQ4_NL with scales that are powers of two, bf16 rows), so
an error against 64 bits is what truncated sums and a few fp32 roundings leave. It grows with the longest chain of products and is measured over some 80,000 values, where two runs of the
same split differ by half a percent. 33 to 64 tokens, last chunk not full: quarters, whose chains are shorter than the reference's halves (K = 384: 8 products and 12): below it; halves of whole chunks (16) lie 1 to 3 %
above. Last chunk full: halves of the same length: within 2 %. Up to 32 tokens: quarters. And against an item of 100 tokens, which has one chain: halves have half its length, quarters a fourth; what is
compared may be half as far off again, and twice."""
import ctypes as C

import pytest
import torch

from tqllm_b200 import synth

pytestmark = pytest.mark.gpu
EXPERTS, ROWS = 32, 208


def exact_bank(t, k, scale, g):
    """weights that fp16 holds exactly"""
    from tqllm_b200 import moe
    raw = synth.quantize(t, torch.randn(EXPERTS * ROWS, k, generator=g, device="cuda") * scale).reshape(-1)
    if t == synth.IQ4_NL:
        raw = raw.reshape(-1, 18).clone()
        raw[:, :2] = torch.tensor([scale / 64], dtype=torch.float16).view(torch.uint8).cuda()      # values of up to 127 times it
        raw = raw.reshape(-1)
    return moe.DeviceBank(t, raw, EXPERTS, ROWS, k)


def weights_of(bank, k):
    return bank.dequant().double().reshape(EXPERTS, -1, k)[:, :ROWS]


def error(t, k, tokens, others, gate_up):
    """relative error of eight experts of `tokens` tokens each beside 24 of `others`"""
    from tqllm_b200 import capi, moe
    g = torch.Generator("cuda").manual_seed(k + tokens)
    first = exact_bank(t, k, 2.0 if gate_up else 2.0 ** -5, g)               # a gate this large makes SwiGLU the product of two sums, or nothing
    second = exact_bank(t, k, 2.0 ** -5, g) if gate_up else None
    x = torch.randn(8 * tokens, k, generator=g, device="cuda").bfloat16()
    x = torch.cat([x, torch.randn(24 * others, k, generator=g, device="cuda").bfloat16()])
    counts = torch.tensor([tokens] * 8 + [others] * 24, device="cuda")
    ids = torch.repeat_interleave(torch.arange(EXPERTS, device="cuda"), counts).int().reshape(-1, 1)
    plan = moe.dispatch(ids, EXPERTS)
    with capi.family("gemm"):
        y = moe.expert_gateup_swiglu(first, second, x, plan) if gate_up else moe.expert_down(first, x.float(), plan)
    assert int(plan.buf[3]) == 0, "a bounded wait ran out"
    n = 8 * tokens
    product = lambda bank: torch.einsum("ark,atk->atr", weights_of(bank, k)[:8], x[:n].double().reshape(8, tokens, k)).reshape(n, ROWS)
    want = product(first)
    if gate_up:
        want = want * torch.sigmoid(want) * product(second)
    return float((y[:n].double() - want).norm() / want.norm())


@pytest.mark.parametrize("gate_up", (False, True), ids=("down", "gate/up"))
@pytest.mark.parametrize("t,k", ((synth.IQ4_NL, 320), (synth.NVFP4G, 384), (synth.NVFP4G, 896), (synth.IQ4_NL, 960), (synth.NVFP4G, 1408)))
@pytest.mark.parametrize("tokens", (33, 50, 64))
def test_last_chunk_not_full(t, k, tokens, gate_up):
    assert error(t, k, tokens, 0, gate_up) <= error(t, k, tokens, 100, gate_up)


@pytest.mark.parametrize("gate_up", (False, True), ids=("down", "gate/up"))
@pytest.mark.parametrize("tokens", (16, 32, 50, 64))
def test_full_chunks(tokens, gate_up):
    for t in (synth.IQ4_NL, synth.NVFP4G):
        narrow = error(t, 2048, tokens, 0, gate_up)
        assert narrow <= (0.8 if tokens <= 32 else 1.02) * error(t, 2048, tokens, 100, gate_up)
        assert narrow <= (0.5 if tokens <= 32 else 0.75) * error(t, 2048, 100, 100, gate_up)


@pytest.mark.parametrize("k", (384, 1344, 1408))
@pytest.mark.parametrize("tokens", (33, 48, 64))
def test_gathered_rows_have_the_same_bits(k, tokens):
    """the always-on expert holds every token; the smallest workspace has no room for rows in slot order"""
    from tqllm_b200 import capi, moe
    t = synth.IQ4_NL if k % 128 else synth.NVFP4G
    shape = synth.LayerShape("ragged", k, 32, 4, 256, shared=True, types=(t, t, t))
    dev = moe.MoeLayer.from_synth(synth.make_layer(shape, 5, "cuda"))
    x = synth.make_tokens(shape, tokens, 6, "cuda")
    with capi.family("gemm"):
        dev.forward(x)
    art = dev.artefacts()
    assert art["status"] == 0
    plan = moe.dispatch(art["ids"].clone(), 32, tokens)
    small = capi.lib.b2moe_expert_workspace_bytes(t, tokens, k, capi.BF16)
    act, ws = torch.zeros(tokens * 5, 256, device="cuda"), torch.empty(small, dtype=torch.uint8, device="cuda")
    ref = lambda b: C.byref(b.c)
    with capi.family("gemm"):
        capi.check(capi.lib.b2moe_expert_gateup_swiglu(ref(dev.gate), ref(dev.up), ref(dev.sh[0]), ref(dev.sh[1]), x.data_ptr(), capi.BF16, plan.buf.data_ptr(),
                                                       tokens, 4, tokens, act.data_ptr(), ws.data_ptr(), small, torch.cuda.current_stream().cuda_stream), "gateup")
    assert int(plan.buf[3]) == 0
    assert torch.equal(act, art["act"])
