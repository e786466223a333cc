"""GPU: the two-table ("Mix") weight formats through the byte-table kernel, every output against the CPU oracle, bit for
bit: block and micro-block geometries with compiled-in and run-time lane counts, blocks of zeros, subnormals, values
next to fp16's largest (products that overflow), row counts that end inside a CTA's share."""
import numpy as np
import pytest

from util import bits, seeded_inputs

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

GEOMETRIES = [(128, 8, 1), (128, 32, 1), (128, 16, 1), (64, 8, 2), (256, 64, 1), (128, 8, 2), (32, 8, 1)]


def _inputs(rows, K, seed):
    x = seeded_inputs("wgt", rows, K, seed).astype(np.float32)
    rng = np.random.default_rng(seed + 1)
    for r in range(0, rows, 7):
        x[r] *= [1.0, 2.0 ** -14, 2.0 ** -18, 3.0e5, 8.0e5, 0.0][(r // 7) % 6]
    x = np.clip(x, -65504, 65504)
    x[:, ::31] = 0.0
    x = x.astype(np.float16)
    x[rng.random(x.shape) < 0.01] = np.float16(-0.0)
    return x


@pytest.mark.parametrize("block,micro,mb", GEOMETRIES)
@pytest.mark.parametrize("rows", [1, 41])
@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
def test_mix_outputs_match_the_oracle(oracle, block, micro, mb, rows, dtype):
    import hbq_b200 as H
    K = 1536 if block != 256 else 1792
    t = torch.from_numpy(_inputs(rows, K, block + micro + rows)).cuda().to(getattr(torch, dtype))
    x = t.half().cpu().numpy()
    o = oracle.quantize(x, oracle.Format(oracle.KIND_HBQ, 2, mb, 5, 3, block, l2_block_size=micro, l2_sc_bit=2, l2_scheme="Mix"))
    kw = dict(block_size=block, ebit=2, mbit=mb, sc_ebit=5, sc_mbit=3, l2_block_size=micro, l2_sc_bit=2, l2_scheme="Mix")
    want = torch.from_numpy(np.ascontiguousarray(o["deq"]).view(np.int16).copy()).view(torch.float16).to(t.dtype)
    q = H.HBQQuantizer(**kw)
    assert torch.equal(q.q(t).cpu().view(torch.int16), want.view(torch.int16))
    qk = H.HBQQuantizer(keep_l2_scale=True, **kw)
    assert torch.equal(qk.q(t).cpu().view(torch.int16), want.view(torch.int16))
    assert np.array_equal(qk.shared_scale.cpu().numpy().view(np.uint16), bits(o["scale"]))
    assert np.array_equal(qk.l2_scale.cpu().numpy().astype(np.uint8), o["l2"])
    assert np.array_equal(qk.blk_l2_scheme.cpu().numpy().astype(np.uint8), o["scheme"])
    if (block // micro) * 2 not in (8, 16, 32):
        return
    for with_deq in (False, True):
        packed = q.quantize_packed(t, with_deq=with_deq)
        packed = packed[0] if with_deq else packed
        pc = packed.codes.cpu().numpy()
        un = np.stack([pc & 0xF, pc >> 4], axis=-1).reshape(rows, -1)
        oc = o["codes"].reshape(rows, -1).astype(np.uint8)
        assert np.array_equal(un, oc & 0xF)
        if mb == 2:
            assert np.array_equal(np.unpackbits(packed.sign.cpu().numpy(), axis=-1, bitorder="little"), oc >> 4)
        assert np.array_equal(packed.scheme.cpu().numpy(), o["scheme"])
        assert torch.equal(H.dequantize_packed(packed).cpu().view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("block,micro,mb", [(128, 8, 1), (128, 32, 2), (32, 8, 1)])
def test_mix_packed_outputs_of_infinite_and_nan_inputs(oracle, block, micro, mb):
    """An infinity takes the largest element value in every packed output and a NaN stays one in the tensor, as in the
    oracle (which leaves a NaN's code open)."""
    import hbq_b200 as H
    x = _inputs(41, 1536, 5)
    rng = np.random.default_rng(6)
    x[rng.random(x.shape) < 0.004] = np.float16(np.inf)
    x[rng.random(x.shape) < 0.004] = np.float16(-np.inf)
    x[3, :block] = np.float16(np.inf)
    x[rng.random(x.shape) < 0.002] = np.float16(np.nan)
    x[5, :block] = np.float16(np.nan)
    ok = ~np.isnan(x)
    o = oracle.quantize(x, oracle.Format(oracle.KIND_HBQ, 2, mb, 5, 3, block, l2_block_size=micro, l2_sc_bit=2, l2_scheme="Mix"))
    q = H.HBQQuantizer(block_size=block, ebit=2, mbit=mb, sc_ebit=5, sc_mbit=3, l2_block_size=micro, l2_sc_bit=2, l2_scheme="Mix")
    packed, deq = q.quantize_packed(torch.from_numpy(x).cuda(), with_deq=True)
    pc = packed.codes.cpu().numpy()
    un = np.stack([pc & 0xF, pc >> 4], axis=-1).reshape(41, -1)
    assert np.array_equal(un[ok], o["codes"].reshape(41, -1).astype(np.uint8)[ok] & 0xF)
    assert np.array_equal(packed.scheme.cpu().numpy(), o["scheme"])
    got = deq.cpu().numpy()
    assert np.array_equal(bits(got)[ok], bits(o["deq"].reshape(41, -1))[ok]) and np.isnan(got[~ok]).all()


@pytest.mark.parametrize("block,micro,mb", [(128, 8, 1), (128, 32, 2), (64, 16, 1), (32, 8, 1)])
def test_mix_tensor_of_infinite_and_nan_inputs_does_not_depend_on_the_outputs(oracle, block, micro, mb):
    """The tensor alone, with the kept scales and with packed outputs: the oracle's values, NaNs included."""
    import hbq_b200 as H
    x = _inputs(41, 1536, 7)
    rng = np.random.default_rng(8)
    x[rng.random(x.shape) < 0.004] = np.float16(np.inf)
    x[rng.random(x.shape) < 0.004] = np.float16(-np.inf)
    x[3, :block] = np.float16(-np.inf)
    x[rng.random(x.shape) < 0.002] = np.float16(np.nan)
    x[5, :block] = np.float16(np.nan)
    ok = ~np.isnan(x)
    want = oracle.quantize(x, oracle.Format(oracle.KIND_HBQ, 2, mb, 5, 3, block, l2_block_size=micro, l2_sc_bit=2, l2_scheme="Mix"))["deq"].reshape(41, -1)
    assert np.isinf(want).any()
    kw = dict(block_size=block, ebit=2, mbit=mb, sc_ebit=5, sc_mbit=3, l2_block_size=micro, l2_sc_bit=2, l2_scheme="Mix")
    t = torch.from_numpy(x).cuda()
    got = [H.HBQQuantizer(**kw).q(t), H.HBQQuantizer(keep_l2_scale=True, **kw).q(t)]
    if (block // micro) * 2 in (8, 16, 32):
        got.append(H.HBQQuantizer(**kw).quantize_packed(t, with_deq=True)[1])
    for y in got:
        y = y.cpu().numpy()
        assert np.array_equal(bits(y)[ok], bits(want)[ok]) and np.isnan(y[~ok]).all()
