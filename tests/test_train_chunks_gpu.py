"""hgb_conv_bilateral_mse on batches whose tiles are claimed in chunks of more
than one, the last chunk shorter than the others, with odd image heights (the
last row pair of the bilateral adjoint half in the band): the batch of repeated
images against the single images' results, each of which is checked against the
FP64 oracle elsewhere.  The batch's loss, mask and sigma gradients are the mean
of the singles'; image b's input gradient is its single gradient over the batch
size.  Tolerances: FP32 partials of a few thousand terms each (1e-6 of their
absolute sum) combined in FP64; the gradients' sums cancel by up to two orders."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("boundary", [1, 3, 4])
@pytest.mark.parametrize("w, h, reps", [(190, 131, 243), (259, 37, 441)])
def test_chunked_batch_is_the_mean_of_its_images(gpu, oracle, w, h, reps, boundary):
    rng = np.random.default_rng(w + boundary)
    x3 = torch.from_numpy(rng.random((3, h, w), dtype=np.float32)).cuda()
    t3 = torch.from_numpy(rng.random((3, h, w), dtype=np.float32)).cuda()
    mask = rng.normal(0, 0.02, (7, 7)).astype(np.float32)
    mask[3, 3] += 0.8
    md = torch.from_numpy(mask).cuda()
    sd = torch.tensor([0.15], dtype=torch.float32, device="cuda")
    sm = oracle.spatial_mask(9, 2.0)
    single = [[r.double().cpu().numpy().copy() for r in
               gpu.conv_bilateral_mse(x3[i:i + 1].contiguous(), t3[i:i + 1].contiguous(), md, sd, sm, boundary, 0)]
              for i in range(3)]
    x, t = x3.repeat(reps, 1, 1), t3.repeat(reps, 1, 1)
    n = x.shape[0]
    loss, gx, gm, gs = gpu.conv_bilateral_mse(x, t, md, sd, sm, boundary, 0)
    torch.cuda.synchronize()
    assert abs(loss.item() / np.mean([s[0] for s in single]) - 1) <= 1e-6
    for got, k in ((gm, 2), (gs, 3)):
        want = np.mean([s[k] for s in single], axis=0)
        assert np.linalg.norm(got.double().cpu().numpy() - want) <= 1e-4 * np.linalg.norm(want)
    for b in (0, 1, n // 2, n - 2, n - 1):
        want = single[b % 3][1][0] / n
        assert np.linalg.norm(gx[b].double().cpu().numpy() - want) <= 1e-5 * np.linalg.norm(want)
