"""GPU: the byte-table K- and V-cache writes against the plain quantizer on the rotated / transposed tensor, bit for bit:
rows of one block of 32 to 256 elements, token counts around the 128-token block, odd head counts, per-batch tables,
centring, subnormals, zeros, values next to fp16's largest and infinities."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _data(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(shape, device="cuda", generator=g)
    flat = x.view(-1, 32)
    flat[0::9] *= 30000.0
    flat[1::9] *= 1e-6
    flat[2::9] = 0.0
    flat[3::9, 5] = -0.0
    flat[4::9, 7] = float("inf")
    return x.half()


def _quantizer(block, mb, micro):
    import hbq_b200 as H
    return H.HBQQuantizer(block, 2, mb, 5, 3, l2_block_size=micro, l2_sc_bit=2, l2_scheme="SIG-1")


def _same(a, b, nan=None):
    """Equal bits; where ``nan`` (the quantised tensor is a NaN, whose sign no arithmetic defines) equal magnitudes."""
    if nan is not None:
        a, b = torch.where(nan, a.abs(), a), torch.where(nan, b.abs(), b)
    return torch.equal(a.contiguous().view(torch.int16), b.contiguous().view(torch.int16))


@pytest.mark.parametrize("D,mb,micro", [(32, 2, 8), (64, 1, 8), (64, 2, 32), (128, 2, 8), (128, 1, 32), (128, 2, 16), (256, 2, 64)])
@pytest.mark.parametrize("B,T,heads", [(1, 1, 1), (2, 37, 3), (3, 129, 8)])
def test_k_write_rows_of_one_block(D, mb, micro, B, T, heads):
    from hbq_b200 import kvcache
    q = _quantizer(D, mb, micro)
    k = _data((B, T, heads * D), T + D)
    ang = torch.rand((B, T, D), device="cuda", generator=torch.Generator(device="cuda").manual_seed(D)) * 6.28
    cos, sin = ang.cos().half(), ang.sin().half()
    center = torch.randn((B, heads, 1, D), device="cuda").half()
    x = k.view(B, T, heads, D).transpose(1, 2)
    for c, s in ((cos, sin), (cos[:1], sin[:1])):
        rot = kvcache.apply_rope(x, c, s)
        assert _same(kvcache.write_k_cache(k, heads, q, c, s), q.q(rot.contiguous()), rot.isnan()) and kvcache.fused_last
        assert _same(kvcache.write_k_cache(k, heads, q, c, s, center=center), q.q((rot - center).contiguous()), rot.isnan())
    assert _same(kvcache.write_k_cache(k, heads, q), q.q(x.contiguous()))
    kb = k.bfloat16()
    assert _same(kvcache.write_k_cache(kb, heads, q), q.q(kb.view(B, T, heads, D).transpose(1, 2).contiguous()))


@pytest.mark.parametrize("mb,micro", [(1, 8), (1, 32), (2, 8), (2, 32)])
@pytest.mark.parametrize("B,T,heads,D", [(1, 1, 1, 64), (2, 127, 3, 64), (1, 128, 2, 128), (2, 129, 3, 192), (1, 517, 2, 256)])
def test_v_write_blocks_of_128_tokens(mb, micro, B, T, heads, D):
    from hbq_b200 import kvcache
    q = _quantizer(128, mb, micro)
    v = _data((B, T, heads * D), T + D)
    for t in (v, v.bfloat16()):
        want = q.q(t.view(B, T, heads, D).permute(0, 2, 3, 1).contiguous()).transpose(-1, -2)
        assert _same(kvcache.write_v_cache(t, heads, q), want) and kvcache.fused_last
        assert _same(kvcache.write_v_cache(t, heads, q, token_major=True), want.transpose(1, 2))
