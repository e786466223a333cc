"""Timed cases of the library: what a user's program has it do, through the public entry points.

Kinds of case (``case["op"]``):

``decode``   one linear layer of a decode or short mixed step as a serving engine runs it (``HBQLinearMethod.apply``:
             activation quantizer, then the product), 1 to a few hundred rows, with the weight kept as packed codes
             (``packed_weights``) or as the fp16 fake-quantised tensor.
``linear``   one linear layer of a prefill (``QLinear.forward``: activation quantizer, then the GEMM with the
             configuration's accumulation model), hundreds to thousands of rows, fp16 or bf16 activations.
``act``      a block quantizer on an activation tensor: the fake-quantised tensor alone, or packed codes and scales
             together with it (the bandwidth sweep's outputs).
``weight``   putting a checkpoint's weight into the form it is kept and served in: packed codes (encode), the fp16
             tensor back from them (decode), and the decode GEMM's tile order where the format has one.
``kv``       the K- and V-cache writes of one attention block after its projections (rotary embedding, both quantizers).
``model``    the prefill of a decoder: logits of a batch of prompts (Llama-3-8B or Mixtral-8x7B block sizes, few layers).

Sizes are those of the Llama-3-8B and Mixtral-8x7B shapes that the benchmark and the tests use, with row counts from one
token up, odd ones among them.  Everything is random: weights N(0, 0.02), activations N(0, 1) with outlier channels (or
0.5 x Student-t(3) for the bandwidth sweep), token ids uniform.
"""
from __future__ import annotations

import torch

import hbq_b200 as H
from hbq_b200.packed_gemm import W4Weight
from hbq_b200.serving import HBQLinearMethod

# ---- quantisation configurations (the YAML files' fields) ------------------------------------------------------
_BLOCK = dict(act_block_size=128, act_ebit=2, act_mbit=2, act_sc_ebit=5, act_sc_mbit=3, act_l2_sc_bit=2,
              act_l2_scheme="SIG-1", act_per_tensor_scale=False, wgt_block_size=128, wgt_ebit=2, wgt_mbit=1,
              wgt_sc_ebit=5, wgt_sc_mbit=3, wgt_l2_sc_bit=2, wgt_l2_scheme="Mix", wgt_per_tensor_scale=False,
              qk_mx_round=False, scale_allow_subnormal=False)
_MICRO = {"hbq_a": 8, "hbq_e": 32}


def _config(preset: str, accumulation: str = "fp32", kv: bool = False) -> H.PTQConfig:
    """``hbq_a`` / ``hbq_e`` with an accumulation model; ``kv``: also K, V, post-RoPE Q and the attention weights."""
    micro = _MICRO[preset]
    return H.PTQConfig({
        "quantization": dict(xqtype="hbq", wqtype="hbq", quant_attn_wgt=kv, quant_post_rope_q=kv, quant_4b_kv=kv,
                             quant_k_cache=kv, quant_v_cache=kv),
        "block_quant": dict(_BLOCK, act_l2_block_size=micro, wgt_l2_block_size=micro),
        "accumulation": dict(type=accumulation, group_size=128, quant_block_size=32)})


# activation quantizers of the bandwidth sweep
_ACT = {
    "mxfp4": lambda: H.MXFPQuantizer(block_size=32, ebit=2, mbit=1, sc_ebit=5, sc_mbit=0),
    "nvfp4": lambda: H.MXFPQuantizer(block_size=16, ebit=2, mbit=1, sc_ebit=5, sc_mbit=3),
    "mxint8": lambda: H.MXINTQuantizer(nbit=8, sc_ebit=8, sc_mbit=0, block_size=32),
    "mxfp_a8": lambda: H.MXFPQuantizer(block_size=32, ebit=2, mbit=5, sc_ebit=5, sc_mbit=0),
    "hbq_a": lambda: _config("hbq_a").map_act_quantizer(),
    "hbq_e": lambda: _config("hbq_e").map_act_quantizer(),
}
# codes + scales, bytes per element
_PACKED_BYTES = {"mxfp4": 0.5 + 1 / 32, "nvfp4": 0.5 + 1 / 16, "mxint8": 1 + 1 / 32, "mxfp_a8": 1 + 1 / 32,
                 "hbq_a": 0.625 + 1 / 128 + 4 / 128, "hbq_e": 0.625 + 1 / 128 + 1 / 128}
_WGT = {
    "mxfp4": _ACT["mxfp4"],
    "nvfp4": _ACT["nvfp4"],
    "hbq_a": lambda: _config("hbq_a").map_wgt_quantizer(),
    "hbq_e": lambda: _config("hbq_e").map_wgt_quantizer(),
}
_WGT_BYTES = {"mxfp4": 0.5 + 1 / 32, "nvfp4": 0.5 + 1 / 16, "hbq_a": 0.5 + 6 / 128, "hbq_e": 0.5 + 3 / 128}
_KV = {
    "hbq_a": lambda: _config("hbq_a", kv=True).map_kv_quantizer(),
    "hbq_e": lambda: _config("hbq_e", kv=True).map_kv_quantizer(),
    "nvfp4": _ACT["nvfp4"],
}

# linear layers of the two architectures: output features, input features (the fused q/k/v and gate/up among them)
_SHAPES = [(4096, 4096), (1024, 4096), (6144, 4096), (14336, 4096), (4096, 14336), (28672, 4096)]


# ---- the cases ----------------------------------------------------------------------------------------------------
def listed():
    return [
        # a single sequence being decoded: the o projection, the smallest call (latency and launches)
        dict(name="decode_1_packed", op="decode", preset="hbq_a", rows=1, N=4096, K=4096, packed=True),
        # a small decode batch through the up projection
        dict(name="decode_8_packed", op="decode", preset="hbq_e", rows=8, N=14336, K=4096, packed=True),
        # a decode batch of odd size through the down projection
        dict(name="decode_33_packed", op="decode", preset="hbq_a", rows=33, N=4096, K=14336, packed=True),
        # the same step of an engine that keeps the fp16 tensors: fused q/k/v projection
        dict(name="decode_19_fp16", op="decode", preset="hbq_e", rows=19, N=6144, K=4096, packed=False),
        # prefill with INT8 partial sums: the benchmark's layer, bf16 activations
        dict(name="linear_psum_bf16", op="linear", preset="hbq_e", accumulation="fp16_quant", rows=4096, N=14336, K=4096,
             dtype="bf16"),
        # a prompt of odd length through the down projection, fp16 accumulation in groups of 128
        dict(name="linear_grouped_ragged", op="linear", preset="hbq_e", accumulation="fp16", rows=1913, N=4096, K=14336,
             dtype="fp16"),
        # the bandwidth sweep's tensor: packed codes + scales + the dequantised tensor
        dict(name="act_hbq_a_packed", op="act", format="hbq_a", rows=8192, K=8192, dtype="bf16", packed=True),
        # a prompt's hidden states through a one-level format, fake-quantised only
        dict(name="act_nvfp4", op="act", format="nvfp4", rows=3001, K=4096, dtype="fp16", packed=False),
        # quantising a checkpoint's weight and keeping it packed
        dict(name="weight_hbq_a", op="weight", format="hbq_a", N=14336, K=4096),
        # cache writes of four prompts of odd length
        dict(name="kv_hbq_a", op="kv", format="hbq_a", B=4, T=1999, heads=8, D=128),
        # prefill of two prompts, everything quantised (attention weights, Q, K, V as well)
        dict(name="llama_prefill", op="model", arch="llama", layers=2, B=2, T=2048),
        # prefill of one prompt that fills no tile evenly through a mixture-of-experts layer
        dict(name="mixtral_prefill", op="model", arch="mixtral", layers=1, B=1, T=1000),
    ]


def _spread(rng, lo: int, hi: int) -> int:
    """A whole number spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    op = rng.choice(["decode", "decode", "linear", "linear", "act", "act", "weight", "kv", "model"])
    if op == "decode":
        N, K = rng.choice(_SHAPES)
        return dict(op=op, preset=rng.choice(["hbq_a", "hbq_e"]), rows=_spread(rng, 1, 384), N=N, K=K,
                    packed=rng.random() < 0.6)
    if op == "linear":
        N, K = rng.choice(_SHAPES)
        return dict(op=op, preset=rng.choice(["hbq_a", "hbq_e"]), accumulation=rng.choice(["fp16_quant", "fp16", "fp32"]),
                    rows=_spread(rng, 256, 4096), N=N, K=K, dtype=rng.choice(["fp16", "bf16"]))
    if op == "act":
        K = rng.choice([4096, 8192, 14336, 1024]) if rng.random() < 0.8 else rng.randint(1000, 8192)
        return dict(op=op, format=rng.choice(sorted(_ACT)), rows=_spread(rng, 16, 8192), K=K,
                    dtype=rng.choice(["fp16", "bf16"]), packed=rng.random() < 0.5)
    if op == "weight":
        N, K = rng.choice(_SHAPES)
        return dict(op=op, format=rng.choice(sorted(_WGT)), N=N, K=K)
    if op == "kv":
        return dict(op=op, format=rng.choice(sorted(_KV)), B=rng.randint(1, 8), T=_spread(rng, 100, 4096),
                    heads=rng.choice([8, 32]), D=128)
    arch = rng.choice(["llama", "llama", "mixtral"])
    return dict(op=op, arch=arch, layers=rng.randint(1, 2) if arch == "llama" else 1, B=rng.randint(1, 2),
                T=rng.choice([512, 1024, 2048]) if rng.random() < 0.5 else 8 * rng.randint(25, 190))   # multiples of 8: the model's grain


# ---- inputs ---------------------------------------------------------------------------------------------------------
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _activations(rows: int, K: int, g: torch.Generator, gain: float = 30.0) -> torch.Tensor:
    """N(0, 1) with about 0.5 % outlier channels."""
    x = torch.randn((rows, K), device="cuda", generator=g)
    x[:, torch.randperm(K, device="cuda", generator=g)[: max(1, K // 200)]] *= gain
    return x


def _weight(N: int, K: int, g: torch.Generator) -> torch.Tensor:
    return torch.randn((N, K), device="cuda", generator=g).mul_(0.02).half()


_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}


def _arch(case) -> H.LlamaArch:
    arch = H.mixtral_8x7b() if case["arch"] == "mixtral" else H.LlamaArch(vocab=32000)
    arch.layers = case["layers"]
    return arch


def prepare(case, seed):
    g = _gen(seed)
    op = case["op"]
    st = {"op": op}
    if op == "decode":
        cfg = _config(case["preset"])
        method = HBQLinearMethod(cfg.map_act_quantizer(), cfg.map_wgt_quantizer(), packed_weights=case["packed"])
        layer = torch.nn.Module()
        layer.weight = torch.nn.Parameter(_weight(case["N"], case["K"], g), requires_grad=False)
        method.process_weights_after_loading(layer)
        st.update(method=method, layer=layer, x=_activations(case["rows"], case["K"], g).half())
    elif op == "linear":
        cfg = _config(case["preset"], case["accumulation"])
        lin = H.QLinear(case["K"], case["N"], bias=False, check_finite=False, device="cuda", dtype=torch.float16)
        lin.weight.data = _weight(case["N"], case["K"], g)
        lin.weight.requires_grad_(False)
        cfg.apply_to_linear(lin)
        if lin.ops is None:
            lin.ops = H.FP32AccumMatMul()
        lin.aq.out_dtype = torch.float16
        st.update(lin=lin, x=_activations(case["rows"], case["K"], g).to(_DTYPES[case["dtype"]]))
    elif op == "act":
        shape = (case["rows"], case["K"])
        t = torch.randn(shape, device="cuda", generator=g)
        chi = torch.zeros(shape, device="cuda")
        for _ in range(3):
            chi.add_(torch.randn(shape, device="cuda", generator=g).square_())
        x = t.div_(chi.div_(3.0).sqrt_()).mul_(0.5).to(_DTYPES[case["dtype"]])
        st.update(q=_ACT[case["format"]](), x=x, packed=case["packed"])
    elif op == "weight":
        st.update(q=_WGT[case["format"]](), w=_weight(case["N"], case["K"], g), tiled=case["format"].startswith("hbq"))
    elif op == "kv":
        B, T, Hh, D = case["B"], case["T"], case["heads"], case["D"]
        inv = 1.0 / (500000.0 ** (torch.arange(0, D, 2, dtype=torch.float32, device="cuda") / D))
        f = torch.outer(torch.arange(T, dtype=torch.float32, device="cuda"), inv)
        emb = torch.cat((f, f), dim=-1)
        st.update(q=_KV[case["format"]](), heads=Hh, cos=emb.cos().half()[None], sin=emb.sin().half()[None],
                  k=_activations(B * T, Hh * D, g, 8.0).half().view(B, T, Hh * D),
                  v=torch.randn((B, T, Hh * D), device="cuda", generator=g).half())
    else:
        arch = _arch(case)
        model = H.QLlamaModel(arch, device="cuda", parallel=False)
        model.init_weights(seed=seed)
        model.apply_ptq(_config("hbq_e") if case["arch"] == "mixtral" else _config("hbq_a", kv=True))
        st.update(model=model, ids=torch.randint(0, arch.vocab, (case["B"], case["T"]), device="cuda", generator=g))
    return st


# ---- one pass ---------------------------------------------------------------------------------------------------------
def _planes(p):
    return {n: getattr(p, n) for n in ("codes", "sign", "scale_u8", "l2_packed", "scheme") if getattr(p, n) is not None}


def run(state):
    op = state["op"]
    with torch.inference_mode():
        if op == "decode":
            return state["method"].apply(state["layer"], state["x"])
        if op == "linear":
            return state["lin"](state["x"])
        if op == "act":
            if not state["packed"]:
                return state["q"].q(state["x"])
            packed, deq = state["q"].quantize_packed(state["x"], with_deq=True)
            return dict(_planes(packed), deq=deq)
        if op == "weight":
            packed = state["q"].quantize_packed(state["w"])
            out = dict(_planes(packed), weight=H.dequantize_packed(packed))
            if state["tiled"]:
                out["tiles"] = W4Weight.from_packed(packed).data
            return out
        if op == "kv":
            return (H.write_k_cache(state["k"], state["heads"], state["q"], state["cos"], state["sin"]),
                    H.write_v_cache(state["v"], state["heads"], state["q"]))
        return state["model"](state["ids"])


# ---- what a pass cannot do without ------------------------------------------------------------------------------------
def work(case):
    op = case["op"]
    if op in ("decode", "linear"):
        M, N, K = case["rows"], case["N"], case["K"]
        wbytes = 0.5 + 6 / 128 if case.get("packed") else 2.0
        return {"bytes": N * K * wbytes + 2.0 * M * (K + N), "flops": 2.0 * M * N * K}
    if op == "act":
        n = case["rows"] * case["K"]
        return {"bytes": n * (4.0 + (_PACKED_BYTES[case["format"]] if case["packed"] else 0.0)), "flops": 0.0}
    if op == "weight":
        n = case["N"] * case["K"]
        return {"bytes": n * (4.0 + _WGT_BYTES[case["format"]] + (0.5625 if case["format"].startswith("hbq") else 0.0)),
                "flops": 0.0}
    if op == "kv":
        n = case["B"] * case["T"] * case["heads"] * case["D"]
        return {"bytes": 8.0 * n + 4.0 * case["T"] * case["D"], "flops": 0.0}
    a = _arch(case)
    B, T = case["B"], case["T"]
    tokens = B * T
    attn = a.hidden * a.head_dim * (2 * a.heads + 2 * a.kv_heads)
    experts = a.num_experts if a.num_experts else 1
    active = a.top_k if a.num_experts else 1
    mlp = 3 * a.hidden * a.ffn
    flops = 2.0 * tokens * (a.layers * (attn + active * mlp) + a.hidden * a.vocab)
    flops += a.layers * 2.0 * B * a.heads * T * T * a.head_dim               # causal: half of both attention products
    nbytes = 2.0 * (a.layers * (attn + experts * mlp) + a.hidden * a.vocab) + 2.0 * tokens * (a.hidden + a.vocab)
    return {"bytes": nbytes, "flops": flops}


# ---- how far another correct implementation may be ----------------------------------------------------------------------
def tolerance(case):
    op = case["op"]
    if op in ("act", "weight", "kv"):
        return "exact"                       # the quantizers are defined bit for bit
    if op == "model":
        # the same model with its linear layers in 64-bit arithmetic: 3.5e-2 to 6.8e-2.  A sum that lands on the other
        # side of an fp16 rounding moves a value by half an ulp, but where that value meets a threshold of a 5-bit (or
        # 4-bit) code it moves by a whole step, and in the second layer nearly every value has felt one.
        return {"rel": 2e-1}
    # one linear layer: 5e-5 against 64-bit sums of the same fp16 operands, nothing at all for the accumulation models
    # against sums taken in another order (a group's products add up exactly)
    return {"rel": 2e-4}
