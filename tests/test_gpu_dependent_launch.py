"""GPU: kernels that start while the one before them still runs must see everything it wrote and leave everything it
still reads: chains on reused buffers (tokens, packed weights and outputs overwritten in place between calls) enqueued
without a synchronisation, on a side stream and inside a graph, against the same chain synchronised after every call."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _chain(M, sync):
    import hbq_b200 as H
    from hbq_b200.packed_gemm import W4Weight
    N = K = 1024
    g = torch.Generator(device="cuda").manual_seed(M)
    aq = H.HBQQuantizer(128, 2, 2, 5, 3, l2_block_size=8, l2_sc_bit=2, l2_scheme="SIG-1")
    wq = H.HBQQuantizer(128, 2, 1, 5, 3, l2_block_size=8, l2_sc_bit=2, l2_scheme="Mix")
    nv = H.MXFPQuantizer(16, 2, 1, 5, 3)
    ws = [torch.randn((N, K), device="cuda", generator=g).mul_(0.05).half() for _ in range(2)]
    x = torch.randn((M, K), device="cuda", generator=g).half()
    gain = torch.ones(K, dtype=torch.float16, device="cuda")
    steps = []
    wait = torch.cuda.synchronize if sync else (lambda: None)
    w4 = W4Weight.from_packed(wq.quantize_packed(ws[0]))
    for i in range(8):
        w4.data.copy_(W4Weight.from_packed(wq.quantize_packed(ws[i & 1])).data); wait()      # the weight changes in place
        xq = aq.q(x); wait()
        y = w4.matmul(xq); wait()
        z = H.blockquant_ext.gemm_fp32_accum(nv.q(y), ws[i & 1], b_is_nk=True); wait()
        n, _ = H.rmsnorm_quantize(z, gain, 1e-5, aq, residual=y, inplace=False); wait()
        k = H.write_k_cache(n.view(1, M, K), K // 128, aq); wait()
        v = H.write_v_cache(n.view(1, M, K), K // 128, aq); wait()
        x.copy_(H.swiglu_quantize(k.view(M, K), v.view(M, K), aq) + xq); wait()              # the tokens as well
        steps += [xq, y, z, n, k, v]
    return steps + [x]


@pytest.mark.parametrize("M", [1, 5, 33, 100])
def test_chain_without_synchronisation(M):
    want = _chain(M, True)
    torch.cuda.synchronize()
    got = _chain(M, False)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        other = _chain(M, False)
    torch.cuda.synchronize()
    for a, b, c in zip(want, got, other):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16)) and torch.equal(a.view(torch.int16), c.view(torch.int16))
    import hbq_b200 as H
    assert H.gemm_status() == 0


@pytest.mark.parametrize("M", [1, 33])
def test_chain_in_a_graph(M):
    import hbq_b200 as H
    aq = H.HBQQuantizer(128, 2, 2, 5, 3, l2_block_size=8, l2_sc_bit=2, l2_scheme="SIG-1")
    w = torch.randn((1024, 1024), device="cuda").mul_(0.05).half()
    x = torch.zeros((M, 1024), device="cuda").half()

    def steps():
        t = x
        for _ in range(6):
            t = H.blockquant_ext.gemm_fp32_accum(aq.q(t), w, b_is_nk=True)
        return t
    steps()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = steps()
    for _ in range(3):
        x.copy_(torch.randn((M, 1024), device="cuda"))
        g.replay()
        assert torch.equal(out, steps())


class _Buffers:
    """Everything the steps below rewrite in place."""

    def __init__(self):
        import hbq_b200 as H
        from hbq_b200.packed_gemm import W4Weight
        g = torch.Generator(device="cuda").manual_seed(11)
        self.tokens = torch.randn((1, 256, 512), device="cuda", generator=g).half()          # 256 tokens, 4 heads of 128
        ang = torch.rand((1, 256, 128), device="cuda", generator=g) * 6.28
        self.cos, self.sin = ang.cos().half(), ang.sin().half()
        self.act = H.HBQQuantizer(128, 2, 2, 5, 3, l2_block_size=8, l2_sc_bit=2, l2_scheme="SIG-1")
        self.wgt = H.HBQQuantizer(128, 2, 1, 5, 3, l2_block_size=8, l2_sc_bit=2, l2_scheme="Mix")
        self.weights = [torch.randn((512, 512), device="cuda", generator=g).mul_(0.05).half() for _ in range(3)]
        self.gain = torch.ones(512, dtype=torch.float16, device="cuda")
        self.ids = torch.randint(0, 3, (256, 2), device="cuda", generator=g)
        i32 = dict(dtype=torch.int32, device="cuda")
        self.offsets, self.pos = torch.empty(4, **i32), torch.empty(512, **i32)
        self.src = torch.empty(512, dtype=torch.int64, device="cuda")
        self.rows = torch.empty((512, 512), dtype=torch.float16, device="cuda")
        self.share = torch.full((256, 2), 0.5, dtype=torch.float16, device="cuda")
        self.w4 = W4Weight.from_packed(self.wgt.quantize_packed(self.weights[0]))
        self.w4._workspace(64)
        self.start = [t.clone() for t in (self.tokens, self.ids, self.w4.data)]

    def reset(self):
        for t, s in zip((self.tokens, self.ids, self.w4.data), self.start):
            t.copy_(s)


def _block(b, wait):
    """Attention and a sparse block of experts, every output rewritten or its input overwritten by a later step: rotary
    embedding, queries run by run, softmax in place, outputs put in place, routing into the same offsets, grouped
    products, and the decode products beside them."""
    import hbq_b200 as H
    from hbq_b200 import _lib, kvcache
    from hbq_b200.gemm import gemm_grouped
    from hbq_b200.packed_gemm import W4Weight
    from hbq_b200.quantizer import _ptr, _stream_ptr
    L, out = _lib.lib(), []
    for i in range(4):
        x = b.tokens
        q = kvcache.rope_heads(x, 4, b.cos, b.sin); wait()
        runs = kvcache.quantize_q_runs(q.view(1, 256, 512), 4, 2, 128, b.act, b.cos, b.sin); wait()
        p = H.softmax_quantize(runs.view(1, 4, 256, 128), 0.3, b.act); wait()                # in place
        out.append(p.clone()); wait()
        assert kvcache.quantize_head_rows(p.view(1, 4, 256, 128), x.view(1, 256, 4, 128), 0, b.act); wait()      # over the tokens
        k = H.write_k_cache(x, 4, b.act, b.cos, b.sin); wait()
        v = H.write_v_cache(k.view(1, 256, 512), 4, b.act); wait()
        rows = b.rows
        _lib.check(L.hbq_moe_route(_ptr(b.ids), 256, 2, 3, _ptr(b.offsets), _ptr(b.src), _ptr(b.pos), _stream_ptr(x.device)), "route"); wait()
        xs = b.act.q(v.view(256, 512)).index_select(0, b.src); wait()
        gemm_grouped(xs, b.offsets, b.weights, [rows] * 3, range(3), _lib.ACC_GROUPED, 128); wait()
        h = H.swiglu_quantize(rows, xs, b.act); wait()
        gemm_grouped(h, b.offsets, b.weights[::-1], [rows] * 3, range(3), _lib.ACC_FP32); wait()      # over the first products
        y = torch.empty((256, 512), dtype=torch.float16, device=x.device)
        _lib.check(L.hbq_moe_combine(_ptr(rows), _ptr(b.share), _ptr(b.pos), 256, 2, 512, _ptr(y), _stream_ptr(x.device)), "combine"); wait()
        b.ids.copy_((b.ids + i) % 3); wait()                                                  # other offsets in the next round
        n, _ = H.rmsnorm_quantize(y, b.gain, 1e-5, b.act); wait()
        z = torch.cat([b.w4.matmul(n[r:r + 64]) for r in range(0, 256, 64)]); wait()
        b.w4.data.copy_(W4Weight.from_packed(b.wgt.quantize_packed(b.weights[(i + 1) % 3])).data); wait()
        x.copy_((z + n).view(1, 256, 512)); wait()
        out += [q, k, v, xs, h, y, n, z]
    return out + [b.tokens.clone(), b.offsets.clone()]


@pytest.mark.parametrize("how", ["default stream", "side stream", "graph"])
def test_block_without_synchronisation(how):
    import hbq_b200 as H
    b = _Buffers()
    want = _block(b, torch.cuda.synchronize)
    b.reset()
    stream = torch.cuda.current_stream() if how == "default stream" else torch.cuda.Stream()
    torch.cuda.synchronize()
    if how == "graph":
        with torch.cuda.stream(stream):
            _block(b, lambda: None)                       # what is set up once per stream
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            got = _block(b, lambda: None)
        runs = [graph.replay] * 3
    else:
        got = []

        def eager():
            with torch.cuda.stream(stream):
                got[:] = _block(b, lambda: None)
        runs = [eager] * 3
    for run in runs:
        b.reset()
        torch.cuda.synchronize()
        run()
        torch.cuda.synchronize()
        assert len(got) == len(want)
        for i, (g, w) in enumerate(zip(got, want)):
            assert torch.equal(g.view(torch.int16), w.view(torch.int16)), i
    assert H.gemm_status() == 0
