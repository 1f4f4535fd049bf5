"""Quantise with 32 bytes per load: bit for bit what the oracle gives, at run lengths, pitches and base addresses on either side of
where these loads are taken."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _matrix(rows, cols, dtype, pad, shift, seed):
    """rows x cols with a pitch of cols + pad, `shift` elements behind a 256-byte boundary; values over the whole range of e4m3."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    flat = torch.randn(shift + rows * (cols + pad), generator=g, device=DEV) * torch.exp(torch.randn(shift + rows * (cols + pad), generator=g, device=DEV) * 2)
    return flat.to(dtype)[shift:].view(rows, cols + pad)[:, :cols]


# one vector, a row and a bit, several vectors in flight (more than one wave of blocks), more than 64 MiB
@pytest.mark.parametrize("rows,cols", [(1, 16), (5, 48), (257, 1152), (331, 1160), (9000, 768), (46656, 768)])
@pytest.mark.parametrize("pad,shift", [(0, 0), (16, 0), (8, 0), (0, 8), (0, 16)])
def test_quantize(engine, oracle, rows, cols, pad, shift):
    x = _matrix(rows, cols, torch.bfloat16, pad, shift, rows + cols)
    x[rows // 2, cols - 1] = -3.0e4
    scale = torch.full((1,), 0.03125, device=DEV)
    q = engine.quantize_e4m3(x, scale)
    engine.device_status()
    pick = torch.linspace(0, rows - 1, min(rows, 300), device=DEV).long()          # every row of the small ones
    assert np.array_equal(q.view(torch.uint8)[pick].cpu().numpy(), oracle.quantize_rows(x[pick].float().cpu().numpy(), 0.03125))
    narrow = engine.quantize_e4m3(x, scale, out=torch.empty((rows, cols + 8), dtype=torch.uint8, device=DEV)[:, :cols])
    assert torch.equal(q.view(torch.uint8), narrow.view(torch.uint8))              # codes on 8-byte boundaries

