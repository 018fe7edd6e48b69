"""GPU: the exact form of the grouped GEMM (banks of 4-bit codes from nine assignments per expert on): integer operands, activations in one
fp16 term (16-bit rows: no rounding above 2^-29 of the row's largest value) or two (fp32 rows: 2^-22), sums scaled and added in fp32. Against products in 64 bits. Bound: the
tensor core's truncated fp32 sums of up to 256 columns and their fp32 total, about sqrt(256) 2^-24 = 1e-6 of a row's result in the
2-norm, twice through both products; the decode kernels, which a wrong choice of the family would give, lie above 1.6e-5."""
import ctypes as C

import pytest
import torch

from tqllm_b200 import synth

pytestmark = pytest.mark.gpu
TOL = 4e-6
Q4_K, IQ3_S = 12, 21


def products(dev, x, ids, shared):
    """act and y of every assignment (and the shared expert's rows) in 64 bits"""
    n, k = ids.shape
    w = [b.dequant().double().view(b.experts, b.rows, b.cols) for b in (dev.gate, dev.up, dev.down)]
    xd, rows = x.double(), n * k + (n if shared else 0)
    act, y = xd.new_zeros(rows, w[0].shape[1]), xd.new_zeros(rows, w[2].shape[1])
    def put(at, t, m):
        g, u = xd[t] @ m[0].T, xd[t] @ m[1].T
        act[at] = g * torch.sigmoid(g) * u
        y[at] = act[at] @ m[2].T
    for e in range(dev.experts):
        t, s = (ids == e).nonzero(as_tuple=True)
        put(t * k + s, t, [m[e] for m in w])
    if shared:
        put(torch.arange(n * k, rows, device="cuda"), torch.arange(n, device="cuda"), [b.dequant().double() for b in dev.sh])
    return act, y


def err(got, want):
    return float((got.double() - want).norm() / want.norm())


# an odd and an even number of 256-column chunks, items of one class of rows and of both, several items of an expert, a shared expert
@pytest.mark.parametrize("dtype", (torch.bfloat16, torch.float16, torch.float32), ids=("bf16", "f16", "f32"))
@pytest.mark.parametrize("types,hidden,ff,experts,topk,n,shared", (((Q4_K,) * 3, 256, 256, 7, 1, 63, False), ((Q4_K,) * 3, 1280, 768, 12, 3, 36, True),
                                                                   ((Q4_K,) * 3, 3072, 512, 16, 4, 300, False), ((IQ3_S,) * 3, 768, 1792, 9, 3, 65, True),
                                                                   ((IQ3_S,) * 3, 2048, 512, 24, 2, 500, True)))
def test_layer(types, hidden, ff, experts, topk, n, shared, dtype):
    from tqllm_b200 import moe
    dev = moe.MoeLayer.from_synth(synth.make_layer(synth.LayerShape("exact", hidden, experts, topk, ff, shared=shared, types=types), 3, "cuda"))
    x = torch.randn(n, hidden, device="cuda", generator=torch.Generator("cuda").manual_seed(n)).to(dtype)
    x[1] = 0
    x[2] *= 1e-6
    out = dev.forward(x)
    art = dev.artefacts()
    assert art["status"] == 0
    act, y = products(dev, x, art["ids"].long(), shared)
    assert err(art["act"], act) < TOL and err(art["y"], y) < TOL
    for _ in range(3):
        assert torch.equal(dev.forward(x), out)
    # a row that is not finite touches no other
    x[5, 3] = float("inf")
    bad = dev.forward(x)
    keep = torch.arange(n, device="cuda") != 5
    assert torch.equal(bad[keep], out[keep]) and not torch.isfinite(bad[5]).all()


# the experts' tokens at the edges of the boxes and items: 1, 16, 17, 31, 32, 33, 64, 65 and none; rows that end inside an item (five row tiles of 16)
@pytest.mark.parametrize("types", ((Q4_K,) * 3, (IQ3_S,) * 3), ids=("q4k", "iq3s"))
def test_edges(types):
    from tqllm_b200 import capi, moe
    lib, hidden, ff = capi.lib, 512, 256
    sizes = [1, 16, 17, 31, 32, 33, 64, 65, 0]
    dev = moe.MoeLayer.from_synth(synth.make_layer(synth.LayerShape("edges", hidden, len(sizes), 1, ff, types=types), 4, "cuda"))
    ids = torch.cat([torch.full((s,), e, dtype=torch.int32) for e, s in enumerate(sizes)]).cuda()[:, None].contiguous()
    ids = ids[torch.randperm(ids.shape[0], generator=torch.Generator().manual_seed(1)).cuda()].contiguous()
    n = ids.shape[0]
    x = torch.randn(n, hidden, device="cuda", generator=torch.Generator("cuda").manual_seed(2)).half()
    plan = moe.dispatch(ids, len(sizes))
    act = moe.expert_gateup_swiglu(dev.gate, dev.up, x, plan)
    want = products(dev, x, ids.long(), False)[0]
    assert int(plan.buf[3]) == 0 and err(act, want) < TOL
    # one matrix with rows of the caller's types: 80 rows of the gate bank's 256, as a bank of its own
    raw = torch.cat([dev_raw for dev_raw in (synth.quantize(types[0], torch.randn(80, hidden, device="cuda") * 0.02) for _ in sizes)]).reshape(-1)
    bank = moe.DeviceBank(capi.IQ3_S_X4 if types[0] == IQ3_S else types[0], raw, len(sizes), 80, hidden)
    counts, groups = moe.plan_to_groups(plan)
    ws = torch.empty(lib.b2moe_expert_matvec_workspace_bytes(C.byref(bank.c), n, 1), dtype=torch.uint8, device="cuda")
    y = torch.zeros(n, 80, device="cuda")
    capi.check(lib.b2moe_expert_gemm(C.byref(bank.c), x.data_ptr(), capi.F16, y.data_ptr(), capi.F32, counts.data_ptr(), groups.data_ptr(), n, 1, 0,
                                     ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream), "gemm")
    w = bank.dequant().double().view(len(sizes), 80, hidden)
    assert err(y, torch.einsum("nk,nrk->nr", x.double(), w[ids[:, 0].long()])) < TOL


def test_where_it_begins_and_small_workspaces():
    """below nine assignments per expert the decode kernels, from there on this form (their errors tell them apart); a layer call with the
    workspace that holds no rows of two terms takes the decode kernels for the down product"""
    from tqllm_b200 import capi, moe
    dev = moe.MoeLayer.from_synth(synth.make_layer(synth.LayerShape("line", 1024, 16, 2, 512, types=(Q4_K,) * 3), 5, "cuda"))
    for n, exact in ((71, False), (72, True)):
        x = synth.make_tokens(dev.shape, n, 6, "cuda")
        dev.forward(x)
        art = dev.artefacts()
        act, y = products(dev, x, art["ids"].long(), False)
        assert (err(art["act"], act) < TOL) == exact and (err(art["y"], y) < TOL) == exact
        if exact:
            dev.ws = dev.ws[:dev.ws_view.expert_scratch + capi.lib.b2moe_expert_workspace_bytes(Q4_K, 2 * n, 512, capi.F32)]
            dev.forward(x)
            art = dev.artefacts()
            assert err(art["act"], act) < TOL and 1e-5 < err(art["y"], y) < 1e-3


@pytest.mark.parametrize("dtype", (torch.bfloat16, torch.float32), ids=("bf16", "f32"))
@pytest.mark.parametrize("types", ((Q4_K,) * 3, (IQ3_S,) * 3), ids=("q4k", "iq3s"))
def test_plan_driven_products(types, dtype):
    """the products over a ready plan, with skipped ids and a shared expert, in scratch of the size with a row per assignment: this form for both"""
    from tqllm_b200 import moe
    n, experts, topk = 130, 12, 3
    dev = moe.MoeLayer.from_synth(synth.make_layer(synth.LayerShape("plan", 768, experts, topk, 512, shared=True, types=types), 6, "cuda"))
    g = torch.Generator().manual_seed(3)
    ids = torch.rand(n, experts, generator=g).argsort(1)[:, :topk].to(torch.int32)
    ids[torch.rand(n, topk, generator=g) < 0.3] = -1
    ids = ids.cuda()
    x = torch.randn(n, 768, generator=g).cuda().to(dtype)
    plan = moe.dispatch(ids, experts, n)
    act = moe.expert_gateup_swiglu(dev.gate, dev.up, x, plan, dev.sh[0], dev.sh[1])
    y = moe.expert_down(dev.down, act, plan, dev.sh[2])
    want = products(dev, x, ids.long(), True)
    assert int(plan.buf[3]) == 0 and err(act, want[0]) < TOL and err(y, want[1]) < TOL
    skipped = (ids.reshape(-1) < 0).nonzero().flatten()
    assert len(skipped) > 50 and not act[skipped].any() and not y[skipped].any()


@pytest.mark.parametrize("dtype", (torch.bfloat16, torch.float16), ids=("bf16", "f16"))
@pytest.mark.parametrize("types,hidden", (((Q4_K,) * 3, 1280), ((IQ3_S,) * 3, 768)), ids=("q4k", "iq3s"))
@pytest.mark.parametrize("n,skip,skew", ((37, 0., False), (77, .2, True), (331, .4, False)))
def test_gathered_rows_change_no_bit(types, hidden, n, skip, skew, dtype):
    """gate/up from the scratch that it accepts, where it gathers token rows, and from a larger one with the rows in slot order: the same rows in
    the same order; a shared expert, skipped ids, counts that do not divide by the loaders' four rows, an expert with most of the tokens"""
    from tqllm_b200 import capi, moe
    lib, experts, topk = capi.lib, 16, 4
    dev = moe.MoeLayer.from_synth(synth.make_layer(synth.LayerShape("gather", hidden, experts, topk, 512, shared=True, types=types), 3, "cuda"))
    g = torch.Generator().manual_seed(n)
    order = torch.rand(n, experts, generator=g)
    if skew:
        order[:, 11] -= 0.9
    ids = order.argsort(1)[:, :topk].to(torch.int32).contiguous()
    ids[torch.rand(n, topk, generator=g) < skip] = -1
    x = torch.randn(n, hidden, generator=g).cuda().to(dtype)
    plan, slots, code = moe.dispatch(ids.cuda(), experts, n), n * topk + n, capi.BF16 if dtype == torch.bfloat16 else capi.F16
    small, large = lib.b2moe_expert_workspace_bytes(dev.gate.type, n, hidden, code), lib.b2moe_expert_slot_workspace_bytes(C.byref(dev.gate.c), slots, code)
    assert small < slots * (2 * hidden + hidden // 8)
    out = []
    for nbytes in (small, large):
        act, ws = torch.zeros(slots, 512, device="cuda"), torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        capi.check(lib.b2moe_expert_gateup_swiglu(*(C.byref(b.c) for b in (dev.gate, dev.up, dev.sh[0], dev.sh[1])), x.data_ptr(), code, plan.buf.data_ptr(), n, topk,
                                                  n, act.data_ptr(), ws.data_ptr(), nbytes, torch.cuda.current_stream().cuda_stream), "gateup")
        assert int(plan.buf[3]) == 0
        out.append(act)
    assert torch.equal(out[0], out[1]) and err(out[0], products(dev, x, ids.cuda().long(), True)[0]) < TOL


def test_decode_kernels_can_be_pinned():
    """the harness reaches the decode kernels at a density where a call takes this form, and they keep their precision there"""
    from tqllm_b200 import capi, moe
    dev = moe.MoeLayer.from_synth(synth.make_layer(synth.LayerShape("pin", 1024, 8, 2, 512, types=(IQ3_S,) * 3), 5, "cuda"))
    x = synth.make_tokens(dev.shape, 120, 6, "cuda")
    for family, exact in (("auto", True), ("decode", True), ("decode_kernels", False)):
        with capi.family(family):
            dev.forward(x)
        art = dev.artefacts()
        act, y = products(dev, x, art["ids"].long(), False)
        assert (err(art["act"], act) < TOL) == exact and (err(art["y"], y) < TOL) == exact and err(art["y"], y) < 1e-3
