"""The variant the dispatch picks gives bit for bit what one fixed variant gives, whatever the shape: every variant adds the
K = 32 steps of an element in the same order and its epilogues differ in layout only.  Shapes on both sides of the lines the
cost model draws: one tile, a last tile of 16 columns, a full round of tiles and one tile more, K of one step and many blocks."""
import pytest
import torch

import siglip_b200
from siglip_b200 import lib as L, synth

pytestmark = pytest.mark.gpu
DEV = "cuda"
GENERAL = 6       # 128 x 128 tiles on single CTAs: serves every layer and output type

SHAPES = [(1, 16, 16), (127, 144, 80), (129, 400, 592), (768, 1152, 1152), (2049, 1040, 512), (2368, 2048, 128), (2369, 2064, 128),
          (3700, 1152, 4304), (7000, 768, 3072), (9473, 512, 1600)]


def _codes(g, rows, cols):
    full = torch.randint(0, 256, (rows, synth.pitch128(cols)), generator=g, device=DEV, dtype=torch.uint8) & 0xBF      # |v| < 2, no NaN
    return full[:, :cols]


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_the_picked_variant_agrees_with_the_general_one(engine, M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    A, B = _codes(g, M, K), _codes(g, N, K)
    bias = torch.randn(N, generator=g, device=DEV).to(torch.bfloat16)
    side = torch.randn((M, N), generator=g, device=DEV).to(torch.bfloat16)
    s = torch.full((1,), 0.05, device=DEV)
    kw = dict(scale_a=s, scale_b=s)
    calls = [lambda: engine.fc1_gelu(A, B, bias, **kw), lambda: engine.fc1_gelu(A, B, bias, out_dtype=torch.uint8, out_scale=s, **kw),
             lambda: engine.fc1_gelu(A, B, bias.float(), flags=L.SL8_FLAG_GELU_HW_TANH, **kw), lambda: engine.linear_bias(A, B, None, **kw),
             lambda: engine.linear_bias(A, B, bias, out_dtype=torch.uint8, out_scale=s, **kw), lambda: engine.fc2_residual(A, B, bias, side, **kw),
             lambda: engine.patch_embed(A, B, side[:100], row_phase=3, **kw) if M >= 100 else engine.patch_embed(A, B, side, **kw)]
    for i, call in enumerate(calls):
        got = call()
        engine.set_variant(GENERAL)
        try:
            want = call()
        finally:
            engine.set_variant(-1)
        engine.device_status()
        assert torch.equal(got.view(torch.uint8), want.view(torch.uint8)), f"call {i} at {M} x {N} x {K}"


def test_the_pick_follows_the_ctas_a_launch_may_use(engine, monkeypatch):
    """A handle held to eight CTAs (or pairs) has many rounds of tiles where the whole chip has less than one."""
    for op, M, N, K, whole, held in ((2, 2048, 768, 768, 18, 17), (1, 4096, 512, 1600, 18, 15)):
        assert engine.query_config(op, M, N, K)["variant_id"] == whole
        monkeypatch.setenv("SL8_MAX_CLUSTERS", "8")
        with siglip_b200.Engine(0) as few:
            cfg = few.query_config(op, M, N, K)
        monkeypatch.delenv("SL8_MAX_CLUSTERS")
        assert cfg["variant_id"] == held and cfg["grid"] == 8 * cfg["cta_group"]
