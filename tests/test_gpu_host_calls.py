"""GPU: the module's calls against the general path they stand in for, over the forms of tensor that take one or the
other: views, subclasses, parameters, tensors that require a gradient, other streams, biases of other types, empty ones."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


class Tagged(torch.Tensor):
    pass


def _forms(x):
    yield "plain", x
    yield "3d", x.view(3, -1, x.shape[-1])
    yield "transposed", x.t()
    yield "strided", x[:, ::2]
    yield "rows", x[1:5]
    yield "offset", x.view(-1)[8:8 + 128 * 20].view(20, 128)
    yield "unaligned", x.view(-1)[1:1 + 128 * 20].view(20, 128)
    yield "subclass", x.as_subclass(Tagged)
    yield "parameter", torch.nn.Parameter(x)
    yield "grad", x.clone().requires_grad_()
    yield "empty", x[:0]
    yield "bf16", x.bfloat16()


@pytest.mark.parametrize("out_dtype", [None, torch.float16, torch.bfloat16])
def test_quantize_equals_the_general_path(out_dtype):
    import hbq_b200 as H
    x = torch.randn((30, 512), device="cuda").half()
    for q in (H.HBQQuantizer(128, 2, 2, 5, 3, l2_block_size=8, l2_sc_bit=2, l2_scheme="SIG-1"), H.MXFPQuantizer(16, 2, 1, 5, 3),
              H.MXFPQuantizer(32, 2, 1, 5, 3, per_tensor_scale=True), H.MXINTQuantizer(8, 5, 0, 32)):
        q.out_dtype = out_dtype
        for name, t in _forms(x):
            got, want = q.q(t), q._launch(t, True, None)
            assert got.dtype == want.dtype and got.shape == want.shape and got.stride() == want.stride(), name
            assert torch.equal(got.view(torch.int16), want.view(torch.int16)) and not got.requires_grad, name


def test_calls_run_on_the_current_stream():
    import hbq_b200 as H
    q = H.HBQQuantizer(128, 2, 2, 5, 3, l2_block_size=8, l2_sc_bit=2, l2_scheme="SIG-1")
    x = torch.randn((64, 4096), device="cuda").half()
    want = q.q(x)
    torch.cuda.synchronize()
    y = torch.zeros_like(x)
    s = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        z = q.q(y)
    y.copy_(x)
    g.replay()
    assert torch.equal(z, want)


@pytest.mark.parametrize("M", [1, 7, 64, 300])
def test_products_equal_the_general_path(M):
    import hbq_b200 as H
    from hbq_b200.gemm import gemm
    from hbq_b200.packed_gemm import W4Weight
    q = H.HBQQuantizer(128, 2, 1, 5, 3, l2_block_size=8, l2_sc_bit=2, l2_scheme="Mix")
    w = torch.randn((256, 512), device="cuda").half()
    packed = q.quantize_packed(w)
    w4, wq = W4Weight.from_packed(packed), H.dequantize_packed(packed)
    x = torch.randn((M, 512), device="cuda").half()
    wide = torch.randn((M, 1024), device="cuda").half()
    for t in (x, wide[:, ::2], torch.nn.Parameter(x), x.as_subclass(Tagged)):
        for bias in (None, torch.randn(256, device="cuda").half(), torch.randn(256, device="cuda")):
            out = torch.empty((M, 256), dtype=torch.float16, device="cuda")
            for mode, gk, gn in ((0, 0, 0), (2, 128, 0), (3, 128, 32)):
                assert torch.equal(gemm(t, wq, mode, gk, gn, bias=bias, b_is_nk=True), gemm(t, wq, mode, gk, gn, bias=bias, b_is_nk=True, out=out))
                wt = wq.t().contiguous()
                assert torch.equal(gemm(t, wt, mode, gk, gn, bias=bias), gemm(t, wt, mode, gk, gn, bias=bias, out=out))
            if M <= 128:
                assert torch.equal(w4.matmul(t, bias), w4.matmul(t, bias, out=out))
    with pytest.raises(RuntimeError):
        gemm(x, wq[:, :256], 0, b_is_nk=True)
    with pytest.raises(RuntimeError):
        gemm(x.float(), wq, 0, b_is_nk=True)
    with pytest.raises(RuntimeError):
        w4.matmul(x[:, :256])
