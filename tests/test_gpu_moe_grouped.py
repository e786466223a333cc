"""GPU: the sparse MoE block whose experts run as grouped products over device row offsets, against the same block one
expert at a time (the path that a hook on an expert selects): the same bits for every routing (fp32 sums in another order
apart) -- experts without rows, with one row, with more rows than a tile -- and the sort behind it against torch's stable
sort."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

ACT = dict(block_size=128, ebit=2, mbit=2, sc_ebit=5, sc_mbit=3, l2_block_size=32, l2_sc_bit=2, l2_scheme="SIG-1")


def _block(E, top_k, hidden, inter, ops, seed=3):
    import hbq_b200 as H
    g = torch.Generator(device="cuda").manual_seed(seed)
    moe = H.ExpertParallelMoE(hidden, inter, E, top_k=top_k, device="cuda", dtype=torch.float16, ops_factory=ops, local_only=True)
    moe.aq = H.HBQQuantizer(**ACT)
    with torch.no_grad():
        moe.gate.weight.copy_(torch.randn((E, hidden), device="cuda", generator=g))
        for ex in moe.experts:
            for lin in (ex.w1, ex.w3, ex.w2):
                lin.weight.copy_(0.05 * torch.randn(lin.weight.shape, device="cuda", generator=g))
            ex.w2.aq = H.HBQQuantizer(**ACT)
    return moe


def _ops(name):
    import hbq_b200 as H
    return {"fp32": H.FP32AccumMatMul, "fp16": lambda: H.FP16AccumMatMul(group_size=128),
            "fp16_quant": lambda: H.FP16AccumMatMul(group_size=64, quant_block_size=32)}[name]


@pytest.mark.parametrize("ops", ["fp32", "fp16", "fp16_quant"])
@pytest.mark.parametrize("E,top_k,tokens", [(8, 2, 1), (8, 2, 77), (3, 1, 700), (20, 2, 301), (4, 4, 129)])
def test_grouped_experts_equal_one_at_a_time(ops, E, top_k, tokens):
    import hbq_b200 as H
    moe = _block(E, top_k, 256, 640, _ops(ops))
    x = torch.randn((tokens, 256), device="cuda").half()
    with torch.inference_mode():
        assert moe._grouped_model() is not None
        got = moe(x)
        handle = moe.experts[0].register_forward_hook(lambda m, i, o: None)
        assert moe._grouped_model() is None
        want = moe(x)
        handle.remove()
    if ops == "fp32" and tokens < 700:
        # batches of up to 32 rows multiply on a kernel that adds in another order: an fp32 sum that falls on the other
        # side of an fp16 rounding (some 1 % of them, by 2^-11) crosses a threshold of w2's input quantizer once in 2^8
        # times and then moves the value by a step of 2^-3: sqrt(0.01 * 2^-8) * 2^-3 = 8e-4 of the result
        assert (got.float() - want.float()).norm() <= 4e-3 * want.float().norm()
    elif top_k <= 2:                                 # the sum of two fp16 products has one rounding either way
        assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    else:                                            # atomic fp16 additions in any order: one rounding of the sum per choice
        bound = top_k * 2.0 ** -11 * want.abs().float().amax()
        assert (got.float() - want.float()).abs().amax() <= bound
    assert H.gemm_status() == 0


@pytest.mark.parametrize("ops", ["fp16", "fp16_quant"])
@pytest.mark.parametrize("packed", [False, True])
def test_block_quantizer_that_yields_bf16(ops, packed):
    """The accumulation operators convert their operand to fp16, so the grouped products see the same values."""
    moe = _block(4, 2, 256, 640, _ops(ops))
    moe.aq.out_dtype = torch.bfloat16
    moe.packed_dispatch = packed
    x = torch.randn((50, 256), device="cuda").half()
    with torch.inference_mode():
        assert moe._grouped_model() is not None
        got = moe(x)
        moe.experts[0].register_forward_hook(lambda m, i, o: None)
        want = moe(x)
    assert got.dtype == want.dtype == torch.float16
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("which", [0, 2])
def test_an_expert_that_keeps_its_scales(which):
    """Any expert whose quantizer keeps the chosen scales has them after the call: the block runs expert by expert."""
    import hbq_b200 as H
    moe = _block(4, 2, 256, 640, _ops("fp16"))
    x = torch.randn((50, 256), device="cuda").half()
    with torch.inference_mode():
        want = moe(x)
        moe.experts[which].w2.aq = H.HBQQuantizer(keep_l2_scale=True, **ACT)
        assert moe._grouped_model() is None
        got = moe(x)
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    rows = int((moe.route(x)[1] == which).sum())
    assert moe.experts[which].w2.aq.shared_scale.shape == (rows, 640 // 128)


@pytest.mark.parametrize("hidden,inter", [(264, 640), (256, 648), (320, 608), (256, 640)])
def test_sizes_that_the_partial_sum_operator_refuses(hidden, inter):
    """K in whole groups of 64 and N in whole blocks of 32, as the operator of an expert's own layers asks for."""
    moe = _block(4, 2, hidden, inter, _ops("fp16_quant"))
    x = torch.randn((50, hidden), device="cuda").half()
    with torch.inference_mode():
        if hidden % 64 == 0 and inter % 64 == 0:
            assert moe._grouped_model() is not None and moe(x).shape == x.shape
        else:
            assert moe._grouped_model() is None
            with pytest.raises(RuntimeError, match="divisible"):
                moe(x)


def test_expert_ids_of_another_integer_type():
    """A block with a router of its own that returns 32-bit ids: the same result as with 64-bit ones."""
    import hbq_b200 as H

    class Block(H.ExpertParallelMoE):
        def route(self, x2d):
            w, idx = super().route(x2d)
            return w, idx.int()

    moe = _block(8, 2, 256, 640, _ops("fp16"))
    x = torch.randn((77, 256), device="cuda").half()
    with torch.inference_mode():
        want = moe(x)
        moe.__class__ = Block
        got = moe(x)
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("E", [1, 2, 8, 33, 256])
@pytest.mark.parametrize("tokens,top_k", [(1, 1), (31, 2), (512, 2), (1000, 3), (40000, 2)])
def test_route_is_a_stable_sort(E, tokens, top_k):
    from hbq_b200 import _lib
    from hbq_b200.quantizer import _ptr, _stream_ptr
    g = torch.Generator(device="cuda").manual_seed(E + tokens)
    ids = torch.randint(0, E, (tokens, top_k), device="cuda", generator=g)
    if E > 2:
        ids[ids == 1] = 0                             # an expert without rows
    off = torch.empty(E + 1, dtype=torch.int32, device="cuda")
    pos = torch.empty(tokens * top_k, dtype=torch.int32, device="cuda")
    src = torch.empty(tokens * top_k, dtype=torch.int64, device="cuda")
    _lib.check(_lib.lib().hbq_moe_route(_ptr(ids), tokens, top_k, E, _ptr(off), _ptr(src), _ptr(pos), _stream_ptr(ids.device)), "route")
    order = torch.sort(ids.view(-1), stable=True).indices
    assert torch.equal(src, order // top_k)
    assert torch.equal(pos.long()[order], torch.arange(tokens * top_k, device="cuda"))
    counts = torch.bincount(ids.view(-1), minlength=E)
    assert torch.equal(off.long(), torch.cat([counts.new_zeros(1), counts.cumsum(0)]))


@pytest.mark.parametrize("E,tokens,top_k", [(1, 1, 1), (8, 33, 2), (33, 1000, 3), (256, 5000, 2)])
def test_ids_without_an_expert_are_left_out(E, tokens, top_k):
    """Ids below 0, of the number of experts and more, and beyond 32 bits: their copies lie behind every expert's rows,
    have no position and add nothing to their token."""
    from hbq_b200 import _lib
    from hbq_b200.quantizer import _ptr, _stream_ptr
    g = torch.Generator(device="cuda").manual_seed(E + tokens)
    n = tokens * top_k
    ids = torch.randint(0, E, (n,), device="cuda", generator=g)
    odd = torch.tensor([-1, E, -2 ** 31, 2 ** 31, 2 ** 32, 2 ** 32 + E - 1, -2 ** 63, 2 ** 63 - 1], device="cuda")
    hit = torch.rand(n, device="cuda", generator=g) < 0.3
    hit[0] = True
    ids = torch.where(hit, odd[torch.arange(n, device="cuda") % 8], ids)
    valid = (ids >= 0) & (ids < E)
    off = torch.empty(E + 1, dtype=torch.int32, device="cuda")
    pos = torch.empty(n, dtype=torch.int32, device="cuda")
    src = torch.empty(n, dtype=torch.int64, device="cuda")
    s, L = _stream_ptr(ids.device), _lib.lib()
    _lib.check(L.hbq_moe_route(_ptr(ids), tokens, top_k, E, _ptr(off), _ptr(src), _ptr(pos), s), "route")
    order = torch.sort(torch.where(valid, ids, E), stable=True).indices
    count = int(valid.sum())
    assert torch.equal(src, order // top_k)
    assert torch.equal(pos.long()[order], torch.where(torch.arange(n, device="cuda") < count, torch.arange(n, device="cuda"), -1))
    counts = torch.bincount(ids[valid], minlength=E)
    assert torch.equal(off.long(), torch.cat([counts.new_zeros(1), counts.cumsum(0)]))
    hidden = 64
    rows = torch.randn((n, hidden), device="cuda", generator=g).half()
    w = torch.rand((tokens, top_k), device="cuda", generator=g).half()
    out = torch.empty((tokens, hidden), dtype=torch.float16, device="cuda")
    _lib.check(L.hbq_moe_combine(_ptr(rows), _ptr(w), _ptr(pos), tokens, top_k, hidden, _ptr(out), s), "combine")
    parts = torch.where(valid[:, None], rows[pos.long().clamp(min=0)] * w.view(-1, 1), 0).view(tokens, top_k, hidden).float()
    want = torch.zeros((tokens, hidden), device="cuda")
    for j in range(top_k):                               # the kernel's order: fp32 sums of the fp16 products
        want += parts[:, j]
    assert torch.equal(out, want.half())


@pytest.mark.parametrize("offsets", [[0, 200, 1000], [-7, 130, 300], [0, 299, 301], [250, 100, 300], [400, 500, 600], [-9, -5, -1]])
def test_row_offsets_outside_the_rows(offsets):
    """Entries only compute and store the rows that A and C have; what lies around C stays as it was."""
    from hbq_b200 import _lib
    from hbq_b200.gemm import gemm, gemm_grouped
    rows, K, N = 300, 128, 256
    g = torch.Generator(device="cuda").manual_seed(5)
    a = torch.randint(-4, 5, (rows, K), device="cuda", generator=g).half()
    ws = [torch.randint(-3, 4, (N, K), device="cuda", generator=g).half() for _ in range(2)]
    around = torch.full((rows + 2048, N), 7.0, dtype=torch.float16, device="cuda")
    out = around[1024:1024 + rows]
    gemm_grouped(a, torch.tensor(offsets, dtype=torch.int32, device="cuda"), ws, [out, out], range(2), _lib.ACC_FP32)
    want = torch.full_like(around, 7.0)
    for e in range(2):
        r0 = min(max(offsets[e], 0), rows)
        r1 = max(min(offsets[e + 1], rows), r0)
        if r1 > r0:
            want[1024 + r0:1024 + r1] = gemm(a[r0:r1].contiguous(), ws[e], 0, b_is_nk=True, force_simt=True)
    assert torch.equal(around, want)
