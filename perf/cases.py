"""What this framework is timed on: the FP8 layers of a SigLIP encoder as a program calls them, from one image to a
thousand, through ``siglip_b200.Engine``.

A case is one pass of one of these programs (``kind``):

  embed     pixels -> patch unfold + quantisation -> patch-embed GEMM + positional table (what opens an encoder)
  block     every GEMM of an encoder block and what feeds them: LayerNorm -> QKV projection; the attention output
            (another library's, bf16) -> quantise -> output projection + residual; LayerNorm -> FC1 + GELU -> FC2 + residual
  fc1, fc2  one layer on operands that are already e4m3, the calls of the per-layer bench
  mlp       FC1 + GELU -> e4m3 -> FC2 + residual as one call, with a static scale between the layers
  dynamic   the same MLP with a dynamic scale: FC1 -> bf16 -> abs-max -> quantise -> FC2
  host_mlp  the MLP as one call on pinned host operands

Programs that run a layer after a layer (block, mlp, dynamic, embed) own their activation buffers; single layers let the
framework allocate their output.  Sizes are those of the two encoders the repository is configured for (768 / 3072 at
196 tokens of 16 x 16 pixels, 1152 / 4304 at 729 tokens of 14 x 14) and generic ones.
"""
from __future__ import annotations

import functools
import math

import torch

from siglip_b200 import Engine, synth
from siglip_b200 import lib as L

LN_SCALE = 8.0 / 448.0        # static scales of a calibrated model: LayerNorm outputs stay within +-8,
ATTN_SCALE = 4.0 / 448.0      # attention outputs (averages of values) within +-4,
PIXEL_SCALE = 1.0 / 448.0     # normalised pixels within +-1,
HIDDEN_SCALE = 0.0125         # GELU outputs within 5.6
EPS = 1e-6


def listed() -> list:
    return [
        # one image through the smaller encoder's patch embedding: an interactive request, launches and latency
        dict(name="embed_1", kind="embed", images=1, height=224, width=224, patch=16, d=768, pixels="f32"),
        # a small serving batch of the same
        dict(name="embed_32", kind="embed", images=32, height=224, width=224, patch=16, d=768, pixels="f32"),
        # bulk embedding of a data set with the larger encoder: K = 588 and a frame that the patches do not divide
        dict(name="embed_256", kind="embed", images=256, height=384, width=384, patch=14, d=1152, pixels="bf16"),
        # one image through a block of the larger encoder: eight dependent calls, none of which fills the GPU
        dict(name="block_1", kind="block", rows=729, d=1152, ff=4304, flags=0),
        # a batch of eight through a block of the smaller encoder, GELU through the hardware tanh
        dict(name="block_8_small", kind="block", rows=8 * 196, d=768, ff=3072, flags=L.SL8_FLAG_GELU_HW_TANH),
        # seven images packed to the tokens that a mask left over: a ragged row count
        dict(name="block_ragged", kind="block", rows=5003, d=1152, ff=4304, flags=0),
        # the per-layer bench, 64 images: FC1 to bf16, FC2
        dict(name="fc1_64", kind="fc1", rows=64 * 729, d=1152, ff=4304, out="bf16", flags=0),
        dict(name="fc2_64", kind="fc2", rows=64 * 729, d=1152, ff=4304),
        # an ordinary batch and a whole data-set shard through the MLP
        dict(name="mlp_16", kind="mlp", rows=16 * 729, d=1152, ff=4304, flags=0),
        dict(name="mlp_1024", kind="mlp", rows=1024 * 729, d=1152, ff=4304, flags=0),
        # a model without calibrated scales
        dict(name="dynamic_8", kind="dynamic", rows=8 * 729, d=1152, ff=4304, flags=0),
        # a caller whose activations live in host memory
        dict(name="host_mlp_16", kind="host_mlp", rows=16 * 729, d=1152, ff=4304, flags=0),
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["embed", "embed", "block", "block", "block", "fc1", "fc2", "mlp", "mlp", "dynamic", "host_mlp"])
    # the two encoders' widths twice as often as a width of no model's
    d, ff = rng.choice([(768, 3072), (768, 3072), (1152, 4304), (1152, 4304), (16 * rng.randint(24, 100), 16 * rng.randint(64, 300))])
    flags = rng.choice([0, 0, 0, L.SL8_FLAG_GELU_HW_TANH])
    if kind == "embed":
        patch = rng.choice([14, 16])
        # square frames of the usual resolutions, or a frame of any shape
        h, w = rng.choice([(224, 224), (256, 256), (384, 384), (rng.randint(64, 512), rng.randint(64, 512))])
        pixels = rng.choice(["f32", "bf16"])
        images = _log(rng, 1, max(1, min(512, 250_000_000 // (h * w * 3))))
        return dict(kind=kind, images=images, height=h, width=w, patch=patch, d=d, pixels=pixels)
    if kind == "fc1":
        return dict(kind=kind, rows=_log(rng, 50, 100_000), d=d, ff=ff, out=rng.choice(["bf16", "e4m3"]), flags=flags)
    if kind == "fc2":
        return dict(kind=kind, rows=_log(rng, 50, 200_000), d=d, ff=ff)
    if kind == "host_mlp":
        return dict(kind=kind, rows=_log(rng, 500, 30_000), d=d, ff=ff, flags=flags)
    if kind == "mlp":        # up to the shard of a data set, whatever the width
        return dict(kind=kind, rows=_log(rng, 50, 746_496 * 1152 * 4304 // max(d * ff, 1152 * 4304)), d=d, ff=ff, flags=flags)
    return dict(kind=kind, rows=_log(rng, 50, 100_000), d=d, ff=ff, flags=flags)


@functools.lru_cache(maxsize=None)
def _engine() -> Engine:
    return Engine(0)          # a program keeps one handle per GPU


def _codes(rows: int, cols: int) -> torch.Tensor:
    """An e4m3 activation buffer: rows on 128-byte lines."""
    return torch.zeros((rows, synth.pitch128(cols)), dtype=torch.uint8, device="cuda").view(torch.float8_e4m3fn)[:, :cols]


def _scalar(v: float) -> torch.Tensor:
    return torch.tensor([v], dtype=torch.float32, device="cuda")


class _Maker:
    """Seeded weights and activations, all on the GPU."""

    def __init__(self, seed: int):
        self.g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape, std: float = 1.0) -> torch.Tensor:
        return torch.randn(shape, generator=self.g, device="cuda") * std

    def bf16(self, rows: int, cols: int, std: float = 1.0) -> torch.Tensor:
        return self.normal(rows, cols, std=std).to(torch.bfloat16)

    def layer(self, n: int, k: int) -> dict:
        w, s = synth.quantize_e4m3(self.normal(n, k, std=0.02))
        return dict(w=w, scale_b=_scalar(s), bias=self.normal(n, std=0.01).to(torch.bfloat16))

    def act(self, rows: int, cols: int, scale: float, gelu: bool = False) -> torch.Tensor:
        """e4m3 codes of an activation with a static scale, made in slices so that a large one fits beside itself."""
        out = _codes(rows, cols)
        for r in range(0, rows, 65536):
            n = min(65536, rows - r)
            x = self.normal(n, cols)
            if gelu:
                x = torch.nn.functional.gelu(x * 0.68, approximate="tanh")
            out[r:r + n].copy_((x / scale).clamp_(-448.0, 448.0).to(torch.float8_e4m3fn))
        return out


def _host(t: torch.Tensor) -> torch.Tensor:
    """Pinned copy in host memory, row pitch kept."""
    if t.dim() == 2 and t.stride(0) != t.shape[1]:
        full = torch.as_strided(t, (t.shape[0], t.stride(0)), (t.stride(0), 1))
        return full.cpu().pin_memory()[:, :t.shape[1]]
    return t.cpu().pin_memory()


def prepare(case: dict, seed: int) -> dict:
    c, m, kind = case, _Maker(seed), case["kind"]
    s = dict(eng=_engine(), kind=kind, flags=c.get("flags", 0))
    if kind == "embed":
        h, w, p, d = c["height"], c["width"], c["patch"], c["d"]
        gh, gw = h // p, w // p
        px = torch.rand((c["images"], 3, h, w), generator=m.g, device="cuda") * 2 - 1
        s["pixels"] = px if c["pixels"] == "f32" else px.to(torch.bfloat16)
        rows, k = c["images"] * gh * gw, 3 * p * p
        s.update(patch=p, period=gh * gw, scale=_scalar(PIXEL_SCALE), proj=m.layer(d, k), A=_codes(rows, k),
                 D=torch.empty((rows, d), dtype=torch.bfloat16, device="cuda"))
        s["table"] = s["eng"].make_table(m.normal(d, std=0.01), m.normal(gh * gw, d, std=0.02))
        return s
    rows, d, ff = c["rows"], c["d"], c["ff"]
    if kind == "block":
        s["x"], s["attn"] = m.bf16(rows, d), m.bf16(rows, d, std=0.5)
        s.update(qkv=m.layer(3 * d, d), out=m.layer(d, d), fc1=m.layer(ff, d), fc2=m.layer(d, ff),
                 ln1=(1 + m.normal(d, std=0.1), m.normal(d, std=0.1)), ln2=(1 + m.normal(d, std=0.1), m.normal(d, std=0.1)),
                 ln_scale=_scalar(LN_SCALE), attn_scale=_scalar(ATTN_SCALE), hidden_scale=_scalar(HIDDEN_SCALE))
        # the activation buffers of a serving loop
        s.update(a=_codes(rows, d), q=torch.empty((rows, 3 * d), dtype=torch.bfloat16, device="cuda"), o=_codes(rows, d),
                 y=torch.empty((rows, d), dtype=torch.bfloat16, device="cuda"), hidden=_codes(rows, ff),
                 D=torch.empty((rows, d), dtype=torch.bfloat16, device="cuda"))
        return s
    if kind == "fc1":
        s.update(A=m.act(rows, d, LN_SCALE), fc1=m.layer(ff, d), scale_a=_scalar(LN_SCALE), out=c["out"],
                 hidden_scale=_scalar(HIDDEN_SCALE))
        return s
    if kind == "fc2":
        s.update(A=m.act(rows, ff, HIDDEN_SCALE, gelu=True), fc2=m.layer(d, ff), scale_a=_scalar(HIDDEN_SCALE),
                 residual=m.bf16(rows, d))
        return s
    s.update(A=m.act(rows, d, LN_SCALE), fc1=m.layer(ff, d), fc2=m.layer(d, ff), scale_a=_scalar(LN_SCALE),
             hidden_scale=_scalar(HIDDEN_SCALE), residual=m.bf16(rows, d))
    if kind == "host_mlp":
        for k in ("fc1", "fc2"):
            s[k] = dict(w=_host(s[k]["w"]), scale_b=float(s[k]["scale_b"]), bias=_host(s[k]["bias"]))
        s.update(A=_host(s["A"]), residual=_host(s["residual"]), D=torch.empty((rows, d), dtype=torch.bfloat16).pin_memory())
        return s
    s.update(hidden=_codes(rows, ff), D=torch.empty((rows, d), dtype=torch.bfloat16, device="cuda"))
    if kind == "dynamic":
        s["h"] = torch.empty((rows, ff), dtype=torch.bfloat16, device="cuda")
    return s


def run(s: dict):
    eng, kind, flags = s["eng"], s["kind"], s["flags"]
    if kind == "embed":
        p = s["proj"]
        eng.patchify_quantize(s["pixels"], s["patch"], s["scale"], out=s["A"])
        return eng.patch_embed(s["A"], p["w"], s["table"], period=s["period"], scale_a=s["scale"], scale_b=p["scale_b"], out=s["D"])
    if kind == "block":
        qkv, out, fc1, fc2, ln = s["qkv"], s["out"], s["fc1"], s["fc2"], s["ln_scale"]
        eng.layernorm_quantize(s["x"], *s["ln1"], EPS, ln, out=s["a"])
        eng.linear_bias(s["a"], qkv["w"], qkv["bias"], scale_a=ln, scale_b=qkv["scale_b"], out=s["q"])
        eng.quantize_e4m3(s["attn"], s["attn_scale"], out=s["o"])
        eng.fc2_residual(s["o"], out["w"], out["bias"], s["x"], scale_a=s["attn_scale"], scale_b=out["scale_b"], out=s["y"])
        eng.layernorm_quantize(s["y"], *s["ln2"], EPS, ln, out=s["a"])
        eng.mlp_chain(s["a"], fc1["w"], fc1["bias"], fc2["w"], fc2["bias"], s["y"], scale_a=ln, scale_w1=fc1["scale_b"],
                      scale_w2=fc2["scale_b"], hidden_scale=s["hidden_scale"], hidden=s["hidden"], out=s["D"], flags=flags)
        return s["q"], s["D"]
    if kind == "fc1":
        p = s["fc1"]
        if s["out"] == "bf16":
            return eng.fc1_gelu(s["A"], p["w"], p["bias"], scale_a=s["scale_a"], scale_b=p["scale_b"], flags=flags)
        return eng.fc1_gelu(s["A"], p["w"], p["bias"], scale_a=s["scale_a"], scale_b=p["scale_b"],
                            out_dtype=torch.float8_e4m3fn, out_scale=s["hidden_scale"], flags=flags)
    if kind == "fc2":
        p = s["fc2"]
        return eng.fc2_residual(s["A"], p["w"], p["bias"], s["residual"], scale_a=s["scale_a"], scale_b=p["scale_b"])
    fc1, fc2 = s["fc1"], s["fc2"]
    if kind == "host_mlp":
        return eng.mlp_chain_host(s["A"], fc1["w"], fc1["bias"], fc2["w"], fc2["bias"], s["residual"], s["D"], scale_a=LN_SCALE,
                                  scale_w1=fc1["scale_b"], scale_w2=fc2["scale_b"], hidden_scale=HIDDEN_SCALE, flags=flags)
    if kind == "mlp":
        return eng.mlp_chain(s["A"], fc1["w"], fc1["bias"], fc2["w"], fc2["bias"], s["residual"], scale_a=s["scale_a"],
                             scale_w1=fc1["scale_b"], scale_w2=fc2["scale_b"], hidden_scale=s["hidden_scale"],
                             hidden=s["hidden"], out=s["D"], flags=flags)
    eng.fc1_gelu(s["A"], fc1["w"], fc1["bias"], scale_a=s["scale_a"], scale_b=fc1["scale_b"], out=s["h"], flags=flags)
    amax, scale = eng.amax_scale(s["h"])
    eng.quantize_e4m3(s["h"], scale, out=s["hidden"])
    eng.fc2_residual(s["hidden"], fc2["w"], fc2["bias"], s["residual"], scale_a=scale, scale_b=fc2["scale_b"], out=s["D"])
    return scale, s["D"]


def work(case: dict) -> dict:
    """Inputs once, outputs once; 2 M N K for each GEMM.  What passes between the layers of one program is not counted."""
    c, kind = case, case["kind"]
    if kind == "embed":
        gh, gw = c["height"] // c["patch"], c["width"] // c["patch"]
        rows, k, d = c["images"] * gh * gw, 3 * c["patch"] ** 2, c["d"]
        pixel = 4 if c["pixels"] == "f32" else 2
        return {"bytes": rows * k * pixel + d * k + 2 * gh * gw * d + 2 * rows * d, "flops": 2 * rows * d * k}
    rows, d, ff = c["rows"], c["d"], c["ff"]
    if kind == "fc1":
        return {"bytes": rows * d + ff * d + 2 * ff + rows * ff * (2 if c["out"] == "bf16" else 1), "flops": 2 * rows * d * ff}
    if kind == "fc2":
        return {"bytes": rows * ff + ff * d + 2 * d + 4 * rows * d, "flops": 2 * rows * d * ff}
    mlp = {"bytes": rows * d + 2 * ff * d + 2 * (ff + d) + 4 * rows * d, "flops": 4 * rows * d * ff}
    if kind == "block":      # x and the attention output in, QKV and the new stream out, four weights
        return {"bytes": 2 * 2 * rows * d + 2 * 3 * rows * d + 2 * rows * d + 4 * d * d + 2 * ff * d, "flops": mlp["flops"] + 8 * rows * d * d}
    return mlp


def tolerance(case: dict):
    """Measured against every kind in float64 with the same roundings (e4m3 between layers, bf16 out): bf16 outputs differ by
    one ulp in few places (2-norm 2e-5 for one GEMM; 2.4e-4, largest 0.02, after a block, whose e4m3 codes flip at ties too)."""
    if case["kind"] == "fc1" and case["out"] == "e4m3":
        return {"rel": 1e-3, "max": 0.25}      # one e4m3 code is an eighth of a value
    return {"rel": 1e-3, "max": 0.08 if case["kind"] == "block" else 0.04}
