"""GPU: the decode GEMM's weight records against the same rearrangement of the packed planes by torch, for block counts that
end inside a thread's four, and the unquantised rotary embedding against the separate tensor ops, bit for bit."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

VALUE_BYTE = [0x00, 0x38, 0x3C, 0x3E, 0x40, 0x42, 0x44, 0x46]      # top bytes of 0, .5, 1, 1.5, 2, 3, 4, 6 as fp16


@pytest.mark.parametrize("scheme", ["Mix", "FP-1"])
@pytest.mark.parametrize("micro", [8, 32])
@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("N,K", [(128, 128), (256, 384), (128, 640), (384, 1024)])
def test_prepacked_records(N, K, bits, micro, scheme):
    import hbq_b200 as H
    from hbq_b200.packed_gemm import W4Weight
    g = torch.Generator(device="cuda").manual_seed(N + K)
    q = H.HBQQuantizer(128, 2, 1, 5, 3, l2_block_size=micro, l2_sc_bit=2, l2_scheme=scheme)
    p = q.quantize_packed(torch.randn((N, K), device="cuda", generator=g).half())
    nblk, tiles = K // 128, N // 128
    codes = p.codes.view(tiles, 128, nblk, 64).permute(0, 2, 1, 3)                       # [tile, block, row, 64 B]
    if bits == 4:
        body = codes.reshape(tiles, nblk, 128, 4, 16).transpose(2, 3)
    else:
        c = torch.stack([codes & 0xF, codes >> 4], dim=-1).reshape(tiles, nblk, 128, 128).long()
        lut = torch.tensor(VALUE_BYTE, device="cuda")
        body = (lut[c & 7] | ((c & 8) << 4)).to(torch.uint8).view(tiles, nblk, 128, 8, 16).transpose(2, 3)
    side = torch.zeros((tiles, nblk, 128, 8), dtype=torch.uint8, device="cuda")
    l2 = p.l2_packed.view(tiles, 128, nblk, -1).permute(0, 2, 1, 3)
    side[..., :l2.shape[-1]] = l2
    sc = p.scale_u8.view(tiles, 128, nblk).transpose(1, 2).int() << 7
    side[..., 4], side[..., 5] = (sc & 0xFF).to(torch.uint8), (sc >> 8).to(torch.uint8)
    if p.scheme is not None:
        side[..., 6] = p.scheme.view(tiles, 128, nblk).transpose(1, 2) & 1
    want = torch.cat([body.reshape(tiles, nblk, -1), side.view(tiles, nblk, -1)], dim=-1)
    assert torch.equal(W4Weight.from_packed(p, bits).data, want.reshape(-1))


@pytest.mark.parametrize("B,T,heads,D", [(1, 1, 1, 16), (2, 37, 3, 64), (1, 1000, 32, 128), (3, 65, 5, 80), (1, 9, 2, 256)])
@pytest.mark.parametrize("per_batch", [False, True])
def test_rope_without_a_quantizer(B, T, heads, D, per_batch):
    from hbq_b200 import kvcache
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn((B, T, heads * D), device="cuda", generator=g).half()
    x.view(-1, 16)[::7] *= 1e-4
    ang = torch.rand((B if per_batch else 1, T, D), device="cuda", generator=g) * 6.28
    cos, sin = ang.cos().half(), ang.sin().half()
    want = kvcache.apply_rope(x.view(B, T, heads, D).transpose(1, 2), cos, sin)
    with torch.no_grad():
        got = kvcache.rope_heads(x, heads, cos, sin)
    assert got.is_contiguous() and torch.equal(got.view(torch.int16), want.contiguous().view(torch.int16))
    assert kvcache.rope_heads(x.clone().requires_grad_(), heads, cos, sin).requires_grad


@pytest.mark.parametrize("cos_shape,sin_shape", [((1, 1, 64), (1, 1, 64)), ((1, 9, 64), (3, 9, 64)), ((3, 9, 1), (3, 9, 1)), ((9, 64), (9, 64))])
def test_rope_tables_that_broadcast(cos_shape, sin_shape):
    from hbq_b200 import kvcache
    x = torch.randn((3, 9, 2 * 64), device="cuda").half()
    cos, sin = torch.rand(cos_shape, device="cuda").half(), torch.rand(sin_shape, device="cuda").half()
    heads = x.view(3, 9, 2, 64).transpose(1, 2)
    with torch.no_grad():
        try:
            want = kvcache.apply_rope(heads, cos, sin)
        except RuntimeError:
            with pytest.raises(RuntimeError):
                kvcache.rope_heads(x, 2, cos, sin)
            return
        assert torch.equal(kvcache.rope_heads(x, 2, cos, sin), want)


@pytest.mark.parametrize("B,T", [(0, 5), (2, 0)])
def test_rope_of_nothing(B, T):
    from hbq_b200 import kvcache
    x, cos = torch.empty((B, T, 2 * 64), device="cuda").half(), torch.ones((1, T, 64), device="cuda").half()
    with torch.no_grad():
        assert kvcache.rope_heads(x, 2, cos, cos).shape == (B, 2, T, 64)
