"""GPU: the query side of a prefill in runs -- post-RoPE queries stored run by run, a run's attention output quantised into
place -- against the plain quantizer on the same tensors permuted by torch, bit for bit; formats whose block is not one
head are refused."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _quantizer(block, mb, micro):
    import hbq_b200 as H
    return H.HBQQuantizer(block, 2, mb, 5, 3, l2_block_size=micro, l2_sc_bit=2, l2_scheme="SIG-1")


def _data(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(shape, device="cuda", generator=g)
    x.view(-1, 32)[::5] *= 3000.0
    x.view(-1, 32)[1::7] *= 1e-6
    x.view(-1, 32)[2::9] = -0.0
    return x.half()


def _same(a, b):
    return torch.equal(a.contiguous().view(torch.int16), b.contiguous().view(torch.int16))


@pytest.mark.parametrize("D,mb,micro", [(128, 2, 8), (128, 1, 32), (64, 2, 8)])
@pytest.mark.parametrize("B,T,heads,group,run", [(1, 256, 4, 1, 128), (2, 384, 6, 3, 128), (3, 24, 8, 8, 8), (1, 7, 2, 2, 7)])
def test_q_runs(D, mb, micro, B, T, heads, group, run):
    from hbq_b200 import kvcache
    q, x = _quantizer(D, mb, micro), _data((B, T, heads * D), T + D)
    ang = torch.rand((B, T, D), device="cuda", generator=torch.Generator(device="cuda").manual_seed(D)) * 6.28
    for cos, sin in ((ang.cos().half(), ang.sin().half()), (ang[:1].cos().half(), ang[:1].sin().half())):
        got = kvcache.quantize_q_runs(x, heads, group, run, q, cos, sin)
        want = kvcache.write_k_cache(x, heads, q, cos, sin).view(B, heads // group, group, T // run, run, D).permute(3, 0, 1, 2, 4, 5)
        assert _same(got, want.reshape(T // run, B, heads // group, group * run, D))


@pytest.mark.parametrize("D,mb,micro", [(128, 2, 8), (128, 2, 32), (64, 1, 8)])
@pytest.mark.parametrize("B,heads,run,t0,T", [(1, 1, 1, 0, 1), (2, 6, 128, 128, 384), (3, 5, 33, 10, 50)])
def test_head_rows(D, mb, micro, B, heads, run, t0, T):
    from hbq_b200 import kvcache
    q, x = _quantizer(D, mb, micro), _data((B, heads, run, D), T + D)
    out = torch.full((B, T, heads, D), 7.0, device="cuda", dtype=torch.float16)
    want = out.clone()
    assert kvcache.quantize_head_rows(x, out, t0, q)
    want[:, t0:t0 + run] = q.q(x.transpose(1, 2).reshape(B * run, heads * D)).view(B, run, heads, D)
    assert _same(out, want)


def test_formats_that_are_refused():
    import hbq_b200 as H
    from hbq_b200 import kvcache
    x, out = _data((1, 2, 16, 128), 1), torch.zeros((1, 16, 2, 128), device="cuda", dtype=torch.float16)
    cos = torch.ones((1, 16, 128), device="cuda", dtype=torch.float16)
    for q in (_quantizer(64, 2, 8), _quantizer(128, 3, 8), H.MXFPQuantizer(32, 2, 1, 5, 3), H.MXFPQuantizer(128, 2, 1, 5, 3),
              H.HBQQuantizer(128, 2, 1, 5, 3, l2_block_size=8, l2_sc_bit=2, l2_scheme="Mix")):
        assert not kvcache.quantize_head_rows(x, out, 0, q)
        assert kvcache.quantize_q_runs(x.view(1, 16, 256), 2, 1, 8, q, cos, cos) is None
    assert not out.any()


def _attention(o_aq):
    import hbq_b200 as H
    torch.manual_seed(1)
    at = H.QLlamaAttention(H.LlamaArch(hidden=256, heads=2, kv_heads=1, head_dim=128, ffn=256, vocab=64, layers=1), device="cuda")
    for lin in (at.q_proj, at.k_proj, at.v_proj, at.o_proj):
        lin.weight.data.normal_(0, 0.05)
        lin.aq = _quantizer(128, 2, 8)
    at.quant_post_rope_q = True
    at.o_proj.aq = o_aq
    at.query_chunk = 128
    return at


@pytest.mark.parametrize("how", ["method", "forward", "hook", "global hook"])
@pytest.mark.parametrize("T", [128, 256])
def test_output_quantizers_that_do_more_than_their_format(how, T):
    """A quantizer type with a `q` or `forward` of its own, or with hooks, is called at every length, also where the
    attention runs in pieces (two at 256 tokens) whose output its format's kernel could quantise in place."""
    import hbq_b200 as H
    calls = []

    class Method(H.HBQQuantizer):
        def q(self, x):
            calls.append(1)
            return super().q(x)

    class Forward(H.HBQQuantizer):
        def forward(self, x):
            calls.append(1)
            return super().forward(x)

    kind = {"method": Method, "forward": Forward}.get(how, H.HBQQuantizer)
    oq = kind(128, 2, 2, 5, 3, l2_block_size=8, l2_sc_bit=2, l2_scheme="SIG-1")
    handle = None
    if how == "hook":
        handle = oq.register_forward_hook(lambda m, i, o: calls.append(1))
    if how == "global hook":
        handle = torch.nn.modules.module.register_module_forward_hook(lambda m, i, o: calls.append(1) if m is oq else None)
    x = torch.randn((T, 256), device="cuda").half()
    cos = torch.ones((1, T, 128), device="cuda").half()
    try:
        with torch.no_grad():
            got = _attention(oq)(x, 1, T, cos, torch.zeros_like(cos))
    finally:
        if handle is not None:
            handle.remove()
    assert len(calls) == 1
    with torch.no_grad():
        want = _attention(_quantizer(128, 2, 8))(x, 1, T, cos, torch.zeros_like(cos))
    assert _same(got, want)
