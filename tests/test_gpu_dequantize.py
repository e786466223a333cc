"""GPU: packed codes and scales back to the fake-quantised tensor, at the sizes where the kernel's chunk and block
arithmetic can go wrong: one row, one chunk more or less than a CTA's share, padded last blocks, odd lengths, bf16.
The result must equal the tensor the quantizer itself writes, bit for bit."""
import pytest

from util import load_formats, make_quantizer

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

FORMATS = ["mxfp4", "nvfp4", "mxint8", "mxfp_a8", "hbq_a_act", "hbq_e_act", "hbq_a_wgt", "hbq_e_wgt"]


@pytest.mark.parametrize("name", FORMATS)
@pytest.mark.parametrize("rows,K", [(1, 8), (1, 8192), (3, 1016), (5, 333), (9, 8192), (129, 4104), (2, 77)])
@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
def test_dequantize_equals_the_quantizers_tensor(name, rows, K, dtype):
    import hbq_b200 as H
    f = load_formats()
    if name not in f:
        pytest.skip("format not in the fixture")
    q = make_quantizer(f[name])
    x = torch.randn((rows, K), device="cuda", generator=torch.Generator(device="cuda").manual_seed(rows * K))
    x[:, ::7] *= 20
    packed, y = q.quantize_packed(x.to(getattr(torch, dtype)), with_deq=True)
    back = H.dequantize_packed(packed)
    a, b = back.view(torch.int16), y.view(torch.int16).clone()
    if f[name]["kind"] == "mxint":
        b[b == -32768] = 0                   # two's-complement codes cannot carry -0.0
    assert torch.equal(a, b)
    if packed.l2_packed is not None:         # micro-scale plane at an odd address
        raw = torch.empty(packed.l2_packed.numel() + 1, dtype=torch.uint8, device="cuda")
        raw[1:] = packed.l2_packed.flatten()
        packed.l2_packed = raw[1:].view(packed.l2_packed.shape)
        assert torch.equal(H.dequantize_packed(packed).view(torch.int16), a)


@pytest.mark.parametrize("mbit", [0, 1, 2])
def test_codes_beyond_fp16_decode_to_infinity(mbit):
    """Five exponent bits: every code times a scale of one, against the value sign * 2^(e - 15) * (1 + m) in 64 bits rounded
    to fp16 -- the top exponent is 2^16 and more, infinite with any mantissa."""
    import hbq_b200 as H
    q = H.MXFPQuantizer(32, 5, mbit, 5, 3)
    bits = 6 + mbit
    packed = q.quantize_packed(torch.zeros((1 << bits, 32), device="cuda").half())
    packed.codes = torch.arange(1 << bits, device="cuda", dtype=torch.uint8).view(-1, 1).expand(-1, 32).contiguous()
    packed.scale_u8 = torch.full_like(packed.scale_u8, 0x3C00 >> 7)
    c = torch.arange(1 << bits, dtype=torch.float64)
    m, e = c % (1 << mbit), (c // (1 << mbit)) % 32
    mag = torch.where(e == 0, m / (1 << mbit) * 2.0 ** -14, (1 + m / (1 << mbit)) * 2.0 ** (e - 15))
    want = torch.where(c >= 1 << (5 + mbit), -mag, mag).half()
    got = H.dequantize_packed(packed).cpu()
    assert torch.isinf(want).sum() == 2 << mbit
    assert torch.equal(got.view(torch.int16), want.view(-1, 1).expand(-1, 32).contiguous().view(torch.int16))
