"""CPU-side checks of the drop-in boundary: the library builds, loads, exports every symbol
the header declares, and the entry points that need no GPU behave."""
import ctypes as C
import re
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def lib():
    from siglip_b200 import build
    build.build()
    import siglip_b200.lib as L
    return L.load_library()


def header_symbols():
    text = (ROOT / "include" / "siglip_fp8.h").read_text()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(sl8_[a-z0-9_]+)\s*\(", text)))


def test_header_and_binding_agree(lib):
    import siglip_b200.lib as L
    syms = header_symbols()
    assert len(syms) >= 16
    assert sorted(L.SIGNATURES) == syms
    for s in syms:
        assert hasattr(lib, s), f"libsiglip_fp8.so does not export {s}"


def test_version_and_variants(lib):
    from siglip_b200.layers import num_variants, describe_variant
    assert b"sm_100a" in lib.sl8_version()
    n = num_variants()
    assert n >= 4
    seen = set()
    for v in range(n):
        c = describe_variant(v)
        assert c["variant_id"] == v and c["cta_group"] in (1, 2) and c["tile_m"] == 128 * c["cta_group"]
        assert c["tile_n"] in (64, 128, 192, 256) and c["tile_k"] in (128, 256) and c["smem_bytes"] <= 232448
        seen.add((c["cta_group"], c["tile_n"], c["stages"], c["epi_warps"], c["staging_buffers"]))
    assert len(seen) == n
    with pytest.raises(Exception):
        describe_variant(n)


def test_query_config_without_handle(lib):
    import siglip_b200.lib as L
    cfg = L.Config()
    assert lib.sl8_query_config(None, L.SL8_OP_FC1_GELU, L.SL8_OUT_BF16, 46656, 4304, 1152, C.byref(cfg)) == 0
    assert cfg.tile_n == 256 and cfg.grid in (148, 296 // 2)
    assert lib.sl8_query_config(None, L.SL8_OP_FC2_RESIDUAL, L.SL8_OUT_BF16, 46656, 1152, 4304, C.byref(cfg)) == 0
    assert cfg.tile_n in (192, 256) and cfg.cta_group == 2     # (2 % apart)
    assert lib.sl8_query_config(None, L.SL8_OP_FC2_RESIDUAL, L.SL8_OUT_BF16, 729, 1152, 4304, C.byref(cfg)) == 0
    assert cfg.tile_n == 64 and cfg.cta_group == 1        # too few 256-wide tiles for 148 SMs
    assert lib.sl8_query_config(None, 7, 0, 10, 16, 16, C.byref(cfg)) == L.SL8_ERR_INVALID_VALUE


def test_the_reported_tile_is_the_one_the_grid_walks(lib):
    """Rows and columns of a tile, as reported, give the tiles of a call: one CTA (pair) each until the GPU is full."""
    import siglip_b200.lib as L
    from siglip_b200.layers import describe_variant
    from siglip_b200.sweep import variant_tiles
    tiles = variant_tiles()
    cfg = L.Config()
    for v in range(lib.sl8_num_variants()):
        c = describe_variant(v)
        assert (c["cta_group"], c["tile_n"]) == tiles[v]
    for op, n, k in ((L.SL8_OP_PATCH_EMBED, 768, 768), (L.SL8_OP_FC1_GELU, 3072, 768), (L.SL8_OP_FC2_RESIDUAL, 1152, 4304), (L.SL8_OP_FC2_RESIDUAL, 1600, 4800)):
        for m in (1, 196, 729, 1568, 5003, 46656):
            assert lib.sl8_query_config(None, op, L.SL8_OUT_BF16, m, n, k, C.byref(cfg)) == 0
            count = -(-m // cfg.tile_m) * -(-n // cfg.tile_n)
            assert cfg.grid == min(count, 148 // cfg.cta_group) * cfg.cta_group, (op, m, n, k)


def test_what_the_query_names_can_be_described(lib):
    """The variant of a call, by its id, is among those that are listed, and described as the query does (shared memory and grid
    are the call's own)."""
    import siglip_b200.lib as L
    from siglip_b200.build import variant_ids
    from siglip_b200.layers import describe_variant, num_variants
    assert variant_ids() == list(range(num_variants()))
    cfg = L.Config()
    named = set()
    for op, n, k in ((L.SL8_OP_PATCH_EMBED, 1152, 588), (L.SL8_OP_FC1_GELU, 1600, 512), (L.SL8_OP_FC2_RESIDUAL, 1152, 4304), (L.SL8_OP_FC2_RESIDUAL, 768, 3072)):
        for m in (1, 300, 729, 1568, 2187, 3136, 5003, 11664, 46656):
            assert lib.sl8_query_config(None, op, L.SL8_OUT_BF16, m, n, k, C.byref(cfg)) == 0
            listed = describe_variant(cfg.variant_id)
            for field in ("cta_group", "tile_m", "tile_n", "tile_k", "stages", "epi_warps", "staging_buffers"):
                assert listed[field] == getattr(cfg, field), (op, m, field)
            named.add(cfg.tile_n)
    assert 192 in named          # (FC2 1152 x 4304 at 5 003 rows)


def test_null_handle_is_rejected(lib):
    import siglip_b200.lib as L
    assert lib.sl8_destroy(None) == L.SL8_ERR_INVALID_VALUE
    assert lib.sl8_set_variant(None, 0) == L.SL8_ERR_INVALID_VALUE
    assert lib.sl8_fc1_gelu_fp8(None, None, 0, None, 0, None, None, None, None, 0, 0, None, 1, 16, 16, 0, None) \
        == L.SL8_ERR_INVALID_VALUE


def test_create_without_gpu_reports_no_device(lib):
    import torch
    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    import siglip_b200
    with pytest.raises(siglip_b200.SL8Error) as e:
        siglip_b200.Engine(0)
    assert e.value.code == siglip_b200.lib.SL8_ERR_NO_DEVICE
    assert "no CUDA device" in str(e.value)
