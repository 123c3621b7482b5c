"""The work that a user of this library has it do, as cases with sizes: what one pass runs, the bytes and operations it
cannot do without, and how closely two correct implementations agree on its outputs.

A pass is the linear layers of one block (or one linear, or the packing of one weight) called through ``linear.py`` in the
order in which the model code calls them, on buffers that the caller owns. Attention and everything else between the
linears is not part of this library: its results are inputs here.
"""
from __future__ import annotations

import importlib

import torch

_pkg = importlib.import_module("comfyui-backend-but-rust_b200")
L = _pkg.linear
F = _pkg.ffi

_DT = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


# ---- the cases ------------------------------------------------------------------------------------------------------------

def listed():
    return [
        # The adaLN modulation linear of a DiT block: one conditioning vector, a large weight. The smallest call there is.
        {"name": "modulation_m1", "kind": "modulation", "M": 1, "K": 3072, "N": 18432},
        # Cross-attention K and V of an SDXL U-Net block: two prompts of 77 tokens, fp16.
        {"name": "cross_kv_m154", "kind": "cross_kv", "M": 154, "K": 2048, "N": 1280},
        # One ConvRot int8 linear through QuantLinear.forward on a few hundred rows (a context embedder, a short prompt).
        {"name": "linear_m333_bf16", "kind": "linear", "M": 333, "K": 3072, "N": 3072, "dtype": "bf16"},
        # W6A8 video-DiT block on few tokens, from the packed weights (no room for a decoded copy).
        {"name": "w6a8_block_m64", "kind": "w6_block", "M": 64, "hidden": 5120, "ffn": 13824, "form": "packed"},
        # The SDXL U-Net's two transformer block widths at 1024 x 1024, CFG batch 2, fp16, quantized at load.
        {"name": "unet_block_1280", "kind": "unet_block", "images": 2, "pixels": 1024, "C": 1280, "head": 64},
        {"name": "unet_block_640", "kind": "unet_block", "images": 2, "pixels": 4096, "C": 640, "head": 64},
        # A SwiGLU DiT block with gated attention output on an odd number of tokens (a non-square image).
        {"name": "swiglu_block_m1111", "kind": "swiglu_block", "M": 1111, "hidden": 3072, "ffn": 8192},
        # A Qwen-Image-shaped MMDiT block at 1024 x 1024: adaLN, QKV, attention-out, MLP with GELU-tanh.
        {"name": "dit_block_m4352", "kind": "dit_block", "M": 4352, "hidden": 3072, "mlp": 12288},
        # The same at 2048 x 2048, the largest.
        {"name": "dit_block_m16896", "kind": "dit_block", "M": 16896, "hidden": 3072, "mlp": 12288},
        # W6A8 video-DiT block, 5 frames of 512 x 512: decode each weight, then the int8 linears.
        {"name": "w6a8_block_m2048", "kind": "w6_block", "M": 2048, "hidden": 5120, "ffn": 13824, "form": "decode"},
        # The MLP of a text encoder layer, weight-only int8 in f32: RMS norm, gate-up, SwiGLU, down onto the residual stream.
        {"name": "text_encoder_m512", "kind": "text_mlp", "M": 512, "hidden": 2560, "ffn": 9728},
        # A linear's weight at load (int8 ConvRot, fp16 U-Net, W6A8) and when a LoRA is baked into it (back to the original
        # basis, then packed again with stochastic rounding).
        {"name": "pack_weights_5120", "kind": "pack", "N": 5120, "K": 5120},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    """One more case of the same ranges; no drawn case costs more than the largest listed one."""
    kind = rng.choice(["modulation", "cross_kv", "linear", "linear", "w6_packed", "unet_block", "unet_block", "swiglu_block",
                       "dit_block", "dit_block", "w6_decode", "text_mlp", "pack"])
    if kind == "modulation":
        K = 256 * rng.randint(4, 20)
        return {"kind": kind, "M": rng.choice([1, 1, 2, 3, rng.randint(4, 8)]), "K": K, "N": rng.choice([2, 3, 6, 9]) * K + 8 * rng.randint(0, 3)}
    if kind == "cross_kv":
        return {"kind": kind, "M": rng.choice([77, 154, 231, 308, rng.randint(16, 512)]), "K": rng.choice([768, 1024, 2048]),
                "N": rng.choice([320, 640, 1280])}
    if kind == "linear":
        dtype = rng.choice(["bf16", "bf16", "f16", "f32"])
        K = 64 * rng.randint(5, 80) if dtype == "f16" else 256 * rng.randint(2, 24)
        N = rng.choice([64, 8 * rng.randint(40, 1800), 256 * rng.randint(2, 40)])
        return {"kind": kind, "M": _log(rng, 9, 8192), "K": K, "N": N, "dtype": dtype}
    if kind in ("w6_packed", "w6_decode"):
        h = 256 * rng.randint(8, 20)
        return {"kind": "w6_block", "M": _log(rng, 10, 192) if kind == "w6_packed" else _log(rng, 200, 5000), "hidden": h,
                "ffn": 256 * (round(h * rng.choice([2.5, 2.7, 4.0])) // 256), "form": "packed" if kind == "w6_packed" else "decode"}
    if kind == "unet_block":
        C, head = rng.choice([(320, 40), (640, 64), (640, 80), (1280, 64), (1280, 160)])
        side = {320: (24, 96), 640: (16, 72), 1280: (8, 40)}[C]
        return {"kind": kind, "images": rng.choice([1, 2, 2, 4]), "pixels": rng.randint(*side) * rng.randint(*side), "C": C, "head": head}
    if kind == "swiglu_block":
        h = 256 * rng.randint(6, 16)
        return {"kind": kind, "M": _log(rng, 200, 5500), "hidden": h, "ffn": 256 * (round(h * rng.choice([2.67, 3.0, 4.0])) // 256)}
    if kind == "dit_block":
        h = 256 * rng.randint(6, 12)
        return {"kind": kind, "M": _log(rng, 300, 16896), "hidden": h, "mlp": 4 * h}
    if kind == "text_mlp":
        h = 256 * rng.randint(4, 14)
        return {"kind": kind, "M": _log(rng, 20, 1024), "hidden": h, "ffn": 256 * (round(h * rng.choice([2.67, 3.8, 4.0])) // 256)}
    return {"kind": "pack", "N": 8 * rng.randint(80, 1600), "K": 256 * rng.randint(2, 24)}


# ---- inputs ---------------------------------------------------------------------------------------------------------------

class _Make:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.dev = torch.device("cuda")
        self.g = torch.Generator(device=self.dev).manual_seed(seed)

    def randn(self, *shape):
        return torch.randn(*shape, generator=self.g, device=self.dev)

    def activations(self, M, K, dtype=torch.bfloat16):
        """N(0, 1) with heavy-tailed channels: a channel's scale is |t(3)|, between 0.2 and 50."""
        t = self.randn(K).abs() / (self.randn(3, K).square().sum(0) / 3.0).sqrt()
        return (self.randn(M, K) * t.clamp(0.2, 50.0)).to(dtype)

    def bias(self, N, dtype=torch.bfloat16):
        return (self.randn(N) * 0.01).to(dtype)

    def convrot(self, N, K, dtype=torch.bfloat16, bias=True):
        """An int8 ConvRot linear: (codes, scales, bias)."""
        q, s = L.convrot_requant(self.randn(N, K) * 0.02, 0)
        return q, s, self.bias(N, dtype) if bias else None

    def fp16(self, N, K, rotate):
        """A U-Net linear quantized at load from fp16."""
        q, s = L.sd_quant_rows((self.randn(N, K) * 0.02).half(), rotate)
        return q, s, self.bias(N, torch.float16)

    def w6(self, N, K):
        """A W6A8 linear: (packed codes, group scales, channel scales, bias)."""
        return (*L.w6_requant((self.randn(N, K) * 0.015).bfloat16(), 1), self.bias(N))

    def empty(self, *shape, dtype=torch.bfloat16):
        return torch.empty(shape, dtype=dtype, device=self.dev)

    def codes(self, M, K):
        """Where a quantizer writes: codes and row scales."""
        return self.empty(M, K, dtype=torch.int8), self.empty(M, dtype=torch.float32)


def _rot(K):
    """The U-Net's rotation group for rows of K values."""
    return 256 if K % 256 == 0 else 64 if K % 64 == 0 else 0


def _prepare_modulation(c, m):
    M, K, N = c["M"], c["K"], c["N"]
    return {"x": m.activations(M, K), "w": m.convrot(N, K), "a": m.codes(M, K), "out": m.empty(M, N)}


def _run_modulation(s):
    q, sc, b = s["w"]
    a, xs = L.quant_rows(s["x"], F.PRO_SILU, 1, q=s["a"][0], scales=s["a"][1])
    return L.int8_gemm(a, q, xs, sc, b, out=s["out"])


def _prepare_cross_kv(c, m):
    K, N = c["K"], c["N"]
    return {"ctx": m.randn(c["M"], K).half(), "k": m.fp16(N, K, 256), "v": m.fp16(N, K, 256)}


def _run_cross_kv(s):
    a, xs = L.sd_quant_rows(s["ctx"], 256)
    return [L.int8_gemm(a, q, xs, sc, b, out_dtype=torch.float16) for q, sc, b in (s["k"], s["v"])]


def _prepare_linear(c, m):
    dt = _DT[c["dtype"]]
    w = (m.randn(c["N"], c["K"]) * 0.02).to(dt)
    lin = L.QuantLinear.from_float(w, m.bias(c["N"], dt), _rot(c["K"]) if dt == torch.float16 else 256)
    return {"x": m.activations(c["M"], c["K"], dt), "lin": lin}


def _run_linear(s):
    return s["lin"].forward(s["x"])


def _prepare_w6_block(c, m):
    M, h, f = c["M"], c["hidden"], c["ffn"]
    s = {"form": c["form"], "x": m.activations(M, h), "attn": m.randn(M, h).bfloat16(), "ones": torch.ones(h, dtype=torch.bfloat16, device=m.dev),
         "qkv_w": m.w6(3 * h, h), "out_w": m.w6(h, h), "up_w": m.w6(f, h), "down_w": m.w6(h, f), "a": m.codes(M, h), "af": m.codes(M, f),
         "qkv": m.empty(M, 3 * h), "x1": m.empty(M, h), "x2": m.empty(M, h), "h": m.empty(M, f)}
    if c["form"] == "decode":
        s["parts"] = m.empty(f // 64, M, dtype=torch.float32)
    return s


def _run_w6_block(s):
    def quant(x, pro=F.PRO_PLAIN):
        a = s["a"] if x.shape[1] == s["a"][0].shape[1] else s["af"]
        return L.quant_rows(x, pro, 1, q=a[0], scales=a[1], eps=1e-6)

    packed = s["form"] == "packed"

    def linear(a, xs, w, **kw):
        q6, rel, ch, b = w
        if packed:
            return L.w6a8_gemm(a, q6, rel, xs, ch, b, **kw)
        return L.int8_gemm(a, L.w6_decode(q6, rel, a.shape[1]), xs, ch, b, **kw)

    linear(*quant(s["x"], F.PRO_RMS), s["qkv_w"], out=s["qkv"])
    linear(*quant(s["attn"]), s["out_w"], rscale=s["ones"], resid=s["x"], out=s["x1"])
    a, xs = quant(s["x1"], F.PRO_RMS)
    if packed:
        a, xs = quant(linear(a, xs, s["up_w"], act=F.ACT_GELU_TANH, out=s["h"]))
    else:
        q6, rel, ch, b = s["up_w"]
        L.int8_gemm_act_rot(a, L.w6_decode(q6, rel, a.shape[1]), xs, ch, b, act=F.ACT_GELU_TANH, out=s["h"], amax_part=s["parts"])
        a, xs = L.quant_rows_rotated(s["h"], s["parts"], q=s["af"][0], scales=s["af"][1])
    linear(a, xs, s["down_w"], rscale=s["ones"], resid=s["x1"], out=s["x2"])
    return [s["qkv"], s["x2"]]


def _prepare_unet_block(c, m):
    C, P, images = c["C"], c["pixels"], c["images"]
    M, heads = P * images, C // c["head"]
    padded = -(-c["head"] // 64) * 64          # the attention kernel's head width
    h = torch.float16
    norm = lambda: (1.0 + 0.1 * m.randn(C), 0.1 * m.randn(C))  # noqa: E731
    attn = lambda: m.randn(M, heads, padded).half() if padded != c["head"] else m.randn(M, C).half()  # noqa: E731
    return {"x": m.activations(M, C, h).view(images, P, C), "groups": 32, "head": c["head"], "gn": norm(), "ln1": norm(), "ln2": norm(),
            "ln3": norm(), "attn1": attn(), "attn2": attn(), "ones": torch.ones(C, dtype=h, device=m.dev), "r": _rot(C), "r4": _rot(4 * C),
            "in_w": m.fp16(C, C, _rot(C)), "qkv_w": m.fp16(3 * C, C, _rot(C)), "o1_w": m.fp16(C, C, _rot(C)), "q_w": m.fp16(C, C, _rot(C)),
            "o2_w": m.fp16(C, C, _rot(C)), "up_w": m.fp16(8 * C, C, _rot(C)), "down_w": m.fp16(C, 4 * C, _rot(4 * C)),
            "out_w": m.fp16(C, C, _rot(C)), "t": m.empty(M, C, dtype=h), "qkv": m.empty(M, 3 * C, dtype=h), "q": m.empty(M, C, dtype=h),
            "h": m.empty(M, 8 * C, dtype=h), "y": m.empty(M, C, dtype=h)}


def _run_unet_block(s):
    r, t, ones = s["r"], s["t"], s["ones"]

    def linear(a, w, **kw):
        q, sc, b = w
        return L.int8_gemm(a[0], q, a[1], sc, b, **kw)

    def heads(attn):
        return L.sd_unpad_quant_rows(attn, s["head"], r) if attn.dim() == 3 else L.sd_quant_rows(attn, r)

    linear(L.sd_group_norm_quant_rows(s["x"], *s["gn"], s["groups"], 1e-6, r), s["in_w"], out=t)
    linear(L.sd_ln_quant_rows(t, *s["ln1"], 1e-5, r), s["qkv_w"], out=s["qkv"])
    linear(heads(s["attn1"]), s["o1_w"], rscale=ones, resid=t, out=t)
    linear(L.sd_ln_quant_rows(t, *s["ln2"], 1e-5, r), s["q_w"], out=s["q"])
    linear(heads(s["attn2"]), s["o2_w"], rscale=ones, resid=t, out=t)
    linear(L.sd_ln_quant_rows(t, *s["ln3"], 1e-5, r), s["up_w"], out=s["h"])
    linear(L.sd_geglu_quant_rows(s["h"], s["r4"]), s["down_w"], rscale=ones, resid=t, out=t)
    linear(L.sd_quant_rows(t, r), s["out_w"], rscale=ones, resid=s["x"].view(t.shape), out=s["y"])
    return [s["qkv"], s["q"], s["y"]]


def _prepare_swiglu_block(c, m):
    M, h, f = c["M"], c["hidden"], c["ffn"]
    return {"x": m.activations(M, h), "attn": m.randn(M, h).bfloat16(), "n1": 1.0 + 0.1 * m.randn(h), "n2": 1.0 + 0.1 * m.randn(h), "f": f,
            "ones": torch.ones(h, dtype=torch.bfloat16, device=m.dev), "qkvg_w": m.convrot(4 * h, h, bias=False), "out_w": m.convrot(h, h, bias=False),
            "gu_w": m.convrot(2 * f, h, bias=False), "down_w": m.convrot(h, f, bias=False), "a": m.codes(M, h), "af": m.codes(M, f),
            "qkvg": m.empty(M, 4 * h), "gu": m.empty(M, 2 * f), "x1": m.empty(M, h), "x2": m.empty(M, h)}


def _run_swiglu_block(s):
    h, f = s["x"].shape[1], s["f"]
    q, sc = s["a"]

    def linear(a, w, **kw):
        return L.int8_gemm(a[0], w[0], a[1], w[1], w[2], **kw)

    linear(L.quant_rows(s["x"], F.PRO_RMS, 1, norm_w=s["n1"], eps=1e-6, q=q, scales=sc), s["qkvg_w"], out=s["qkvg"])
    # the attention result times the sigmoid of the gate logits, which are the last quarter of the projection's rows
    linear(L.quant_rows(s["attn"], F.PRO_GATE, 1, g=s["qkvg"][:, 3 * h:], q=q, scales=sc), s["out_w"], rscale=s["ones"], resid=s["x"], out=s["x1"])
    linear(L.quant_rows(s["x1"], F.PRO_RMS, 1, norm_w=s["n2"], eps=1e-6, q=q, scales=sc), s["gu_w"], out=s["gu"])
    linear(L.quant_rows(s["gu"], F.PRO_SWIGLU, 1, K=f, up_offset=f, q=s["af"][0], scales=s["af"][1]), s["down_w"], rscale=s["ones"],
           resid=s["x1"], out=s["x2"])
    return [s["qkvg"], s["x2"]]


def _prepare_dit_block(c, m):
    M, h, f = c["M"], c["hidden"], c["mlp"]
    return {"x": m.activations(M, h), "attn": m.randn(M, h).bfloat16(), "cond": m.randn(1, h).bfloat16(), "ada_w": m.convrot(6 * h, h),
            "qkv_w": m.convrot(3 * h, h), "out_w": m.convrot(h, h), "up_w": m.convrot(f, h), "down_w": m.convrot(h, f), "ac": m.codes(1, h),
            "a": m.codes(M, h), "af": m.codes(M, f), "mod": m.empty(1, 6 * h), "qkv": m.empty(M, 3 * h), "x1": m.empty(M, h),
            "x2": m.empty(M, h), "h": m.empty(M, f), "parts": m.empty(f // 64, M, dtype=torch.float32)}


def _run_dit_block(s):
    x, h = s["x"], s["x"].shape[1]
    a, xs = s["a"]

    def linear(a, w, **kw):
        return L.int8_gemm(a[0], w[0], a[1], w[1], w[2], **kw)

    linear(L.quant_rows(s["cond"], F.PRO_SILU, 1, q=s["ac"][0], scales=s["ac"][1]), s["ada_w"], out=s["mod"])
    shift1, scale1, gate1, shift2, scale2, gate2 = s["mod"].view(6, h).unbind(0)
    linear(L.quant_rows(x, F.PRO_LN_MOD, 1, eps=1e-6, mod_scale=scale1, mod_shift=shift1, q=a, scales=xs), s["qkv_w"], out=s["qkv"])
    linear(L.quant_rows(s["attn"], F.PRO_PLAIN, 1, q=a, scales=xs), s["out_w"], rscale=gate1, resid=x, out=s["x1"])
    L.quant_rows(s["x1"], F.PRO_LN_MOD, 1, eps=1e-6, mod_scale=scale2, mod_shift=shift2, q=a, scales=xs)
    q, sc, b = s["up_w"]
    L.int8_gemm_act_rot(a, q, xs, sc, b, act=F.ACT_GELU_TANH, out=s["h"], amax_part=s["parts"])
    linear(L.quant_rows_rotated(s["h"], s["parts"], q=s["af"][0], scales=s["af"][1]), s["down_w"], rscale=gate2, resid=s["x1"], out=s["x2"])
    return [s["mod"], s["qkv"], s["x2"]]


def _prepare_text_mlp(c, m):
    M, h, f = c["M"], c["hidden"], c["ffn"]
    scratch = (m.empty(4 * M * max(h, f), dtype=torch.uint8), m.empty(4 * f * h, dtype=torch.uint8))
    return {"embeds": m.randn(M, h), "norm": 1.0 + 0.1 * m.randn(h), "gu_w": m.convrot(2 * f, h, bias=False), "down_w": m.convrot(h, f, bias=False),
            "stream": m.empty(M, h, dtype=torch.float32), "gu": m.empty(M, 2 * f, dtype=torch.float32), "scratch": scratch, "f": f}


def _run_text_mlp(s):
    stream = s["stream"].copy_(s["embeds"])    # the residual stream starts at the embeddings; the layer adds to it
    L.wo8_linear(stream, s["gu_w"][0], s["gu_w"][1], F.PRO_RMS, norm_w=s["norm"], eps=1e-6, out=s["gu"], scratch=s["scratch"])
    L.wo8_linear(s["gu"], s["down_w"][0], s["down_w"][1], F.PRO_SWIGLU, K=s["f"], up_offset=s["f"], out=stream, beta=1.0, scratch=s["scratch"])
    return stream


def _prepare_pack(c, m):
    w = m.randn(c["N"], c["K"]) * 0.02
    return {"bf16": w.bfloat16(), "f32": w, "f16": w.half(), "rotate": _rot(c["K"])}


def _run_pack(s):
    q, sc = L.convrot_requant(s["bf16"], 0)
    back = L.convrot_dequant(q, sc, torch.bfloat16)
    return [q, sc, back, *L.convrot_requant(back, 17), *L.convrot_requant(s["f32"], 0), *L.sd_quant_rows(s["f16"], s["rotate"]),
            *L.w6_requant(s["bf16"], 17)]


_PREPARE = {"modulation": _prepare_modulation, "cross_kv": _prepare_cross_kv, "linear": _prepare_linear, "w6_block": _prepare_w6_block,
            "unet_block": _prepare_unet_block, "swiglu_block": _prepare_swiglu_block, "dit_block": _prepare_dit_block,
            "text_mlp": _prepare_text_mlp, "pack": _prepare_pack}
_RUN = {"modulation": _run_modulation, "cross_kv": _run_cross_kv, "linear": _run_linear, "w6_block": _run_w6_block,
        "unet_block": _run_unet_block, "swiglu_block": _run_swiglu_block, "dit_block": _run_dit_block, "text_mlp": _run_text_mlp,
        "pack": _run_pack}


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, _Make(seed))
    state["run"] = _RUN[case["kind"]]
    return state


def run(state):
    return state["run"](state)


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------

def work(case):
    """Inputs and weights read once, results written once (what stays inside a block, such as the hidden activations of an
    MLP, is not counted); two operations per multiply-add of the products. The packing passes have no product: the four
    stages of a 256-wide rotation are 28 operations a value."""
    kind, c = case["kind"], case
    if kind == "modulation":
        M, K, N = c["M"], c["K"], c["N"]
        return {"bytes": 2 * M * K + N * K + 6 * N + 2 * M * N, "flops": 2 * M * N * K}
    if kind == "cross_kv":
        M, K, N = c["M"], c["K"], c["N"]
        return {"bytes": 2 * M * K + 2 * (N * K + 6 * N + 2 * M * N), "flops": 4 * M * N * K}
    if kind == "linear":
        M, K, N, e = c["M"], c["K"], c["N"], 4 if c["dtype"] == "f32" else 2
        return {"bytes": e * M * K + N * K + (4 + e) * N + e * M * N, "flops": 2 * M * N * K}
    if kind == "w6_block":
        M, h, f = c["M"], c["hidden"], c["ffn"]
        weights = 4 * h * h + 2 * h * f
        return {"bytes": weights * 25 // 32 + 6 * (5 * h + f) + 2 * M * 6 * h, "flops": 2 * M * weights}
    if kind == "unet_block":
        C, M = c["C"], c["images"] * c["pixels"]
        weights = 20 * C * C                    # in, qkv 3, out, q, out, up 8, down 4, out
        padded = -(-c["head"] // 64) * 64 * (C // c["head"])
        return {"bytes": weights + 6 * 17 * C + 8 * 4 * C + 2 * M * (C + 2 * padded + 3 * C + C + C), "flops": 2 * M * weights}
    if kind == "swiglu_block":
        M, h, f = c["M"], c["hidden"], c["ffn"]
        weights = 5 * h * h + 3 * h * f
        return {"bytes": weights + 4 * (6 * h + 2 * f) + 8 * h + 2 * M * 7 * h, "flops": 2 * M * weights}
    if kind == "dit_block":
        M, h, f = c["M"], c["hidden"], c["mlp"]
        weights = 4 * h * h + 2 * h * f
        return {"bytes": weights + 6 * h * h + 6 * (11 * h + f) + 14 * h + 2 * M * 6 * h, "flops": 2 * M * weights + 12 * h * h}
    if kind == "text_mlp":
        M, h, f = c["M"], c["hidden"], c["ffn"]
        return {"bytes": 3 * h * f + 4 * (2 * f + h) + 4 * h + 8 * M * h, "flops": 6 * M * h * f}
    N, K = c["N"], c["K"]
    stored = N * K + 4 * N
    w6 = N * K * 25 // 32 + 4 * N
    # inputs: the weight in bf16, f32 and fp16 (bf16 once for both of its packings); results: three int8 packings, the bf16
    # weight back in its original basis, the baked packing, the W6 packing
    return {"bytes": (2 + 4 + 2) * N * K + 4 * stored + 2 * N * K + w6, "flops": 28 * 6 * N * K}


def tolerance(case):
    """Integer results are the same in every correct implementation. Floating ones differ where a result is rounded to 16 bits
    (one in some thousand values lands on the other side of a boundary when sums are formed in another order) and where such
    a value passes through a quantizer again, which makes neighbouring codes of it; the figures are about four times what
    the path shows against the same steps with sums, norms and activations in 64 bits."""
    kind = case["kind"]
    if kind == "pack":              # seen: codes 3e-5, scales 6e-8, the weight back in its original basis 2e-5 (one bf16 step)
        return {"rel": 8e-5, "max": 3e-2, "differ": 2e-4}
    if kind == "text_mlp":          # seen: 5e-6 (the activation's two bf16 terms)
        return {"rel": 2e-5, "max": 2e-4}
    if kind in ("modulation", "linear", "cross_kv"):      # seen: 4e-6 with 16-bit results, one step at most
        return {"rel": 1e-6} if case.get("dtype") == "f32" else {"rel": 2e-5, "max": 1e-2}
    return {"rel": 6e-3, "max": 0.2}                      # seen: 1.5e-3 and 0.05, from codes that differ by one
