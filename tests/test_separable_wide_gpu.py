"""hgb_separable on 16-bit images that TMA stages: eight outputs per lane and two
rows per warp in the row pass, at sizes around the 128 x 32 tile and the lanes'
eight columns, for every tap count, against the FP32 kernel on the widened image
rounded to the storage type.  Both fold the same taps in the same order in FP32, so
the results are equal bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("k", [3, 5, 7, 9, 11, 13, 15])
@pytest.mark.parametrize("boundary", [1, 2, 3, 4])
def test_wide_row_pass_equals_fp32_rounded(gpu, dtype, k, boundary):
    rng = np.random.default_rng(k + 20 * boundary)
    row, col = rng.normal(0, 1, k).astype(np.float32), rng.normal(0, 1, k).astype(np.float32)
    for n, h, w in ((1, 31, 120), (2, 33, 136), (1, 64, 264), (3, 95, 128), (1, 16, 16), (1, 32, 8)):
        if min(h, w) < k // 2 + 1:
            continue
        x = torch.from_numpy(rng.random((n, h, w), dtype=np.float32)).cuda().to(dtype)
        y, y32 = torch.empty_like(x), torch.empty((n, h, w), device="cuda")
        gpu.separable(x, y, row, col, boundary=boundary, const=0.5)
        gpu.separable(x.float(), y32, row, col, boundary=boundary, const=0.5)
        torch.cuda.synchronize()
        assert torch.equal(y, y32.to(dtype)), (n, h, w)
