"""The switches of a measurement build (compiled with -DSL8_DIAG) that leave operand copies out: every launch still comes to its end,
so what a stage's barrier is told to expect is what comes.  The library as it ships refuses them."""
import pytest
import torch

from siglip_b200 import lib as L, synth

pytestmark = pytest.mark.gpu
DEV = "cuda"
SKIP_LOAD, SKIP_A, SKIP_B = 0x1000, 0x8000, 0x10000


# a CTA's share of B has 256, 128, 96 and 64 rows (with 64 the producer of B brings a quarter of A), singly and in pairs
@pytest.mark.parametrize("variant", [0, 1, 6, 7, 19, 20, 21])
@pytest.mark.parametrize("flags", [SKIP_A, SKIP_B, SKIP_A | SKIP_B, SKIP_LOAD])
def test_what_is_left_out_is_not_waited_for(engine, variant, flags):
    a, b = (synth.quantize_e4m3(torch.randn((r, 592), device=DEV))[0] for r in (700, 400))
    out = torch.empty((700, 400), dtype=torch.bfloat16, device=DEV)
    engine.set_variant(variant)
    try:
        engine.fc1_gelu(a, b, None, out=out, flags=flags)
    except L.SL8Error as e:
        assert "unknown flag bits" in str(e)
    else:
        engine.device_status()
    finally:
        engine.set_variant(-1)
