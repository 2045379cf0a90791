"""hgb_local_op SUM with 7 x 7 to 13 x 13 masks on 16-bit storage, on both sides of the
rule that takes large batches of 9 x 9 and 11 x 11 to TMA (tiles of 64 x 64 against four
per SM), rows that TMA can address and rows that it cannot: the bits of the FP32 oracle
(fused multiply-adds in row-major order) rounded once to the storage type."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("k", [7, 9, 11, 13])
@pytest.mark.parametrize("large", [False, True])
def test_16bit_masks(gpu, oracle, large, k, dtype):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    h, w = 67, 133  # 2 x 3 tiles
    n = -(-4 * sms // 6) if large else 3
    rng = np.random.default_rng(k)
    img = torch.from_numpy(rng.random((3, h, w), dtype=np.float32)).to(dtype)
    mask = rng.normal(0, 1.0 / k, (k, k)).astype(np.float32)
    of = torch.arange(n, device="cuda") % 3
    for boundary in (0, 1, 2, 3, 4):
        refs = torch.stack([torch.from_numpy(oracle.local_op(img[b].float().numpy(), mask=mask, boundary=boundary, const=0.5,
                                                             contract=1)).to(dtype) for b in range(3)]).cuda()
        for row in (136, 137):
            x = torch.zeros((n, h, row), dtype=dtype, device="cuda")
            x[:, :, :w] = img.cuda()[of]
            y = torch.zeros((n, h, row), dtype=dtype, device="cuda")
            gpu.local_op(x[:, :, :w], y[:, :, :w], mask=mask, boundary=boundary, const=0.5)
            assert torch.equal(y[:, :, :w], refs[of]), (boundary, row)
            assert not y[:, :, w:].any()
