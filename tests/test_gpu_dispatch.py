"""The variant the dispatch picks gives bit for bit what one fixed variant gives, whatever the shape: every variant adds the
K = 32 steps of an element in the same order and its epilogues differ in layout only."""
import pytest
import torch

import siglip_b200
from siglip_b200 import lib as L, synth

pytestmark = pytest.mark.gpu
DEV = "cuda"
GENERAL = 6       # 128 x 128 tiles on single CTAs: serves every layer and output type

# (kind of call, the variant its cost picks, shapes): every row of the cost model, at row counts and widths that end in the
# middle of a tile and K that ends in the middle of a block.
CASES = [("gelu", 18, (1, 16, 16), (769, 400, 592)), ("gelu", 14, (9473, 144, 80), (5121, 1296, 592)), ("gelu", 15, (9473, 144, 2128)),
         ("tanh", 18, (127, 144, 80)), ("tanh", 3, (9473, 144, 1616)), ("tanh", 15, (9473, 144, 80)), ("tanh", 2, (20001, 528, 2128)),
         ("none", 18, (129, 400, 592)), ("none", 3, (9473, 144, 592)), ("none", 2, (9473, 1040, 1104)), ("none", 1, (20001, 272, 4176)),
         ("fc2", 18, (1, 16, 16), (2369, 528, 592)), ("fc2", 19, (20001, 16, 1616)), ("fc2", 3, (9473, 144, 80)), ("fc2", 17, (9473, 656, 80)),
         ("fc2", 1, (16001, 656, 1616)), ("pe", 18, (127, 144, 80)), ("pe", 17, (9473, 144, 80))]


def _codes(g, rows, cols):
    full = torch.randint(0, 256, (rows, synth.pitch128(cols)), generator=g, device=DEV, dtype=torch.uint8) & 0xBF      # |v| < 2, no NaN
    return full[:, :cols]


@pytest.mark.parametrize("kind,variant,shape", [(kind, v, s) for kind, v, *shapes in CASES for s in shapes])
def test_the_picked_variant_agrees_with_the_general_one(engine, kind, variant, shape):
    M, N, K = shape
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    A, B = _codes(g, M, K), _codes(g, N, K)
    bias = torch.randn(N, generator=g, device=DEV).to(torch.bfloat16)
    s = torch.full((1,), 0.05, device=DEV)
    kw = dict(scale_a=s, scale_b=s)
    e4m3 = dict(out_dtype=torch.uint8, out_scale=s)
    side = torch.randn((M, N), generator=g, device=DEV).to(torch.bfloat16)
    op, flags = {"gelu": (1, 0), "tanh": (1, L.SL8_FLAG_GELU_HW_TANH), "none": (1, L.SL8_FLAG_NO_ACTIVATION), "fc2": (2, 0), "pe": (0, 0)}[kind]
    calls = {"gelu": [lambda: engine.fc1_gelu(A, B, bias, **kw), lambda: engine.fc1_gelu(A, B, None, **e4m3, **kw)],
             "tanh": [lambda: engine.fc1_gelu(A, B, bias.float(), flags=flags, **kw), lambda: engine.fc1_gelu(A, B, bias, flags=flags, **e4m3, **kw)],
             "none": [lambda: engine.linear_bias(A, B, None, **kw), lambda: engine.linear_bias(A, B, bias, **e4m3, **kw)],
             "fc2": [lambda: engine.fc2_residual(A, B, bias, side, **kw)],
             "pe": [lambda: engine.patch_embed(A, B, side[:100], row_phase=3, **kw),
                    lambda: engine.patch_embed(A, B, engine.padded_table(side[:100]), period=min(M, 100), row_phase=3, **kw)]}[kind]
    for i, call in enumerate(calls):
        out_dtype = 1 if i == 1 and op == 1 else 0
        assert engine.query_config(op, M, N, K, out_dtype, flags)["variant_id"] == variant != GENERAL
        got = call()
        engine.set_variant(GENERAL)
        try:
            want = call()
        finally:
            engine.set_variant(-1)
        engine.device_status()
        assert torch.equal(got.view(torch.uint8), want.view(torch.uint8)), f"{kind}, call {i} at {M} x {N} x {K}"


def test_the_pick_follows_the_ctas_a_launch_may_use(engine, monkeypatch):
    """A handle held to eight CTAs (or pairs) has many rounds of tiles where the whole chip has less than one."""
    for op, M, N, K, whole, held in ((2, 2048, 768, 768, 18, 17), (1, 4096, 512, 1600, 18, 15)):
        assert engine.query_config(op, M, N, K)["variant_id"] == whole
        monkeypatch.setenv("SL8_MAX_CLUSTERS", "8")
        with siglip_b200.Engine(0) as few:
            cfg = few.query_config(op, M, N, K)
        monkeypatch.delenv("SL8_MAX_CLUSTERS")
        assert cfg["variant_id"] == held and cfg["grid"] == 8 * cfg["cta_group"]
