"""The patch unfold with three, four and six chunks in flight per thread, last rounds full and cut short: bit for bit the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
# strips of up to 3, 4, 6, 7, 9, 11, 12, 21 steps; patches that are whole chunks, pairs and odd; image rows on chunk boundaries and off them
@pytest.mark.parametrize("W,P", [(128, 16), (160, 16), (224, 16), (128, 14), (160, 14), (384, 14), (512, 14), (512, 16), (250, 14), (333, 16), (301, 7), (224, 7)])
def test_batches(engine, oracle, dtype, W, P):
    images, C, H = 3, 3, 2 * P + 3
    g = torch.Generator(device=DEV).manual_seed(W + P)
    pixels = (torch.rand((images, C, H, W), generator=g, device=DEV) * 2 - 1).to(dtype)
    pixels = pixels.repeat(60, 1, 1, 1) if W % 16 == 0 else pixels                 # many strips: whole patch rows per block
    scale = torch.tensor([1.0 / 448.0], device=DEV)
    A = engine.patchify_quantize(pixels, P, scale)
    engine.device_status()
    K, pitch = C * P * P, A.stride(0)
    row_bytes = pitch if pitch - K < 128 else (K + 15) // 16 * 16
    ref = oracle.patchify_quantize(pixels.float().cpu().numpy(), P, float(scale.item()), lda=pitch, row_bytes=row_bytes)
    assert np.array_equal(torch.as_strided(A, (A.shape[0], pitch), (pitch, 1)).cpu().numpy()[:, :row_bytes], ref[:, :row_bytes])
