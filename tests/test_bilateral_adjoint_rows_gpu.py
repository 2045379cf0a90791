"""hgb_bilateral_adjoint on row pairs: heights whose interior starts or ends on either
row of a pair (odd and even radii), widths around the tile and the groups of four,
the smallest images of the packed form, with each gradient asked for alone as well.
Tolerance: that of the FP32 range weights and sums against the FP64 oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 2e-3  # of the largest gradient, and of dL/dsigma_r (floor 1e-4 where its terms cancel)


@pytest.mark.parametrize("size", [3, 5, 7, 9, 11, 13])
@pytest.mark.parametrize("h,w", [(32, 32), (33, 66), (34, 131), (47, 35)])
def test_row_pairs_vs_fp64_oracle(gpu, oracle, size, h, w):
    for boundary, const in ((1, 0.0), (4, 0.5)):
        rng = np.random.default_rng(size * 1000 + h + boundary)
        x = rng.random((2, h, w), dtype=np.float32)
        g = rng.normal(0, 1, (2, h, w)).astype(np.float32)
        sm = oracle.spatial_mask(size, size / 4.0)
        xd, gd = torch.from_numpy(x).cuda(), torch.from_numpy(g).cuda()
        gi, gs = gpu.bilateral_adjoint(xd, gd, sm, 0.2, boundary, const)
        torch.cuda.synchronize()
        gi, gs, ref_gs = gi.cpu().numpy(), float(gs.item()), 0.0
        for b in range(2):
            a, sg = oracle.bilateral_adjoint(x[b], g[b], sm.astype(np.float64), 0.2, boundary, const)
            ref_gs += sg
            assert np.max(np.abs(gi[b] - a)) <= TOL * np.max(np.abs(a))
        assert abs(gs - ref_gs) <= max(TOL * abs(ref_gs), 1e-4)
