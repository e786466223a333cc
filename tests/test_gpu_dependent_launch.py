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
