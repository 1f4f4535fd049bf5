"""The variant the dispatch picks gives bit for bit what one fixed variant gives, whatever the shape: every variant adds the
K = 32 steps of an element in the same order and its epilogues differ in layout only."""
import pytest
import torch

import siglip_b200
from siglip_b200 import lib as L, sweep, synth

pytestmark = pytest.mark.gpu
DEV = "cuda"
GENERAL = 6       # 128 x 128 tiles on single CTAs: serves every layer and output type

# Row counts and widths that end in the middle of a tile and K that ends in the middle of a block, from one row of one narrow tile up:
# between them they reach every row of the cost model (tests/test_tooling.py).
SHAPES = {
    "gelu": [(1, 16, 16), (769, 400, 592), (9473, 144, 80), (5121, 1296, 592), (9473, 144, 2128), (769, 2320, 592), (300, 2064, 1616), (129, 416, 16),
             (5003, 528, 1104), (5003, 528, 4176), (9001, 784, 4176), (5003, 3088, 80)],
    "tanh": [(1300, 3088, 592), (127, 144, 80), (9473, 144, 1616), (9473, 144, 80), (20001, 528, 2128), (1300, 2320, 4176), (700, 656, 592), (129, 416, 272),
             (5003, 784, 4176), (4000, 1600, 4176)],
    "none": [(129, 400, 592), (9473, 144, 592), (9473, 1040, 1104), (20001, 272, 4176), (769, 2320, 3072), (3001, 2320, 16), (16001, 2320, 1616),
             (700, 528, 1104), (129, 416, 16), (4000, 784, 1104), (5003, 1296, 4176)],
    "fc2": [(1, 16, 16), (2369, 528, 592), (20001, 16, 1616), (9473, 144, 80), (9473, 656, 80), (16001, 656, 1616), (5121, 784, 3072), (1300, 2064, 16),
            (700, 528, 16), (129, 416, 16), (5003, 1296, 4176), (7001, 1040, 4176)],
    "pe": [(127, 144, 80), (9473, 144, 80), (769, 1552, 4176), (3001, 2320, 16), (700, 784, 2128), (129, 416, 16), (7001, 1040, 2128)],
}


def _codes(g, rows, cols):
    full = torch.randint(0, 256, (rows, synth.pitch128(cols)), generator=g, device=DEV, dtype=torch.uint8) & 0xBF      # |v| < 2, no NaN
    return full[:, :cols]


@pytest.mark.parametrize("kind,shape", [(kind, s) for kind, shapes in SHAPES.items() for s in shapes])
def test_the_picked_variant_agrees_with_the_general_one(engine, kind, shape):
    M, N, K = shape
    variant = sweep.cheapest(kind.upper(), M, N, K)
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
    for cls, op, M, N, K in (("FC2", 2, 2048, 768, 768), ("GELU", 1, 4096, 512, 1600)):
        whole, held = sweep.cheapest(cls, M, N, K), sweep.cheapest(cls, M, N, K, clusters=8)
        assert whole != held
        assert engine.query_config(op, M, N, K)["variant_id"] == whole
        monkeypatch.setenv("SL8_MAX_CLUSTERS", "8")
        with siglip_b200.Engine(0) as few:
            cfg = few.query_config(op, M, N, K)
        monkeypatch.delenv("SL8_MAX_CLUSTERS")
        assert cfg["variant_id"] == held and cfg["grid"] == 8 * cfg["cta_group"]
