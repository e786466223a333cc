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
