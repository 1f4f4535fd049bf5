"""Tiles of 64 columns (variant 20) and of 192 (variant 21): bit for bit what the general variant gives."""
import pytest
import torch

from tests import test_gpu_dispatch as dispatch

pytestmark = pytest.mark.gpu
DEV = "cuda"

@pytest.mark.parametrize("variant", [20, 21])
@pytest.mark.parametrize("M,N,K", [(1, 16, 16), (129, 64, 80), (257, 80, 592), (385, 192, 1168), (300, 208, 4304), (2500, 400, 144)])
def test_tile_edges(engine, variant, M, N, K):
    """One row, one narrow column of tiles, remainders of either width, a K that ends in the middle of a block, several rounds of tiles."""
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    A, B = dispatch._codes(g, M, K), dispatch._codes(g, N, K)
    s = torch.full((1,), 0.05, device=DEV)
    kw = dict(scale_a=s, scale_b=s)
    bias = torch.randn(N, generator=g, device=DEV).to(torch.bfloat16)
    side = torch.randn((M + 130, N), generator=g, device=DEV).to(torch.bfloat16)
    period = min(M, 100)
    calls = [lambda: engine.fc1_gelu(A, B, bias, **kw), lambda: engine.fc1_gelu(A, B, bias.float(), out_dtype=torch.uint8, out_scale=s, **kw),
             lambda: engine.linear_bias(A, B, None, **kw), lambda: engine.fc2_residual(A, B, bias, side[:M], **kw),
             lambda: engine.patch_embed(A, B, side[:period], period=period, row_phase=period // 2, **kw),
             lambda: engine.patch_embed(A, B, engine.padded_table(side[:period]), period=period, **kw)]
    for i, call in enumerate(calls):
        got = []
        for v in (variant, dispatch.GENERAL):
            engine.set_variant(v)
            try:
                got.append(call())
            finally:
                engine.set_variant(-1)
            engine.device_status()
        assert torch.equal(got[0].view(torch.uint8), got[1].view(torch.uint8)), f"call {i} at {M} x {N} x {K}"


def test_the_listed_variants_are_those_a_handle_takes(engine):
    from siglip_b200.layers import num_variants
    from siglip_b200.lib import SL8Error
    for v in range(num_variants()):
        engine.set_variant(v)
        assert engine.query_config(1, 5000, 1152, 4304)["variant_id"] == v
    engine.set_variant(-1)
    with pytest.raises(SL8Error):
        engine.set_variant(num_variants())
