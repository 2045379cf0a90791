"""GPU parity of the tiled line adjoints (line_adjoint_kernels.cuh) with the FP64
restatements: hgb_separable_adjoint and hgb_local_op_adjoint with 1 x K and
K x 1 masks, at the edges of the 64 x 32 tiles and on images smaller than the
reach.

Tolerances, from FP32 rounding (u = 2^-24): a gradient pixel folds at most
(K + K (K - 1)) <= 225 fused multiply-adds per pass over a few pre-images, the
usual error of such a sum being a few u: 2e-6 relative (L2).  A tap gradient
folds 16 products per thread, a warp and a CTA tree (about 9 more additions),
then FP64: at most 25 u = 1.5e-6 of the sum of the absolute products, 3e-6 with
the rounding of t and g_t themselves."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (3, 5), (32, 64), (31, 63), (33, 65), (40, 134)]


def _close(got, ref):
    return np.linalg.norm(got - ref) <= 2e-6 * max(np.linalg.norm(ref), 1e-30)


@pytest.mark.parametrize("boundary", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("k", [3, 5, 7, 9, 11, 13, 15])
def test_separable_adjoint_tiles(gpu, oracle, k, boundary):
    rng = np.random.default_rng(100 * k + boundary)
    for h, w in SIZES:
        img = rng.random((h, w)).astype(np.float32)
        gout = rng.normal(0, 1, (h, w)).astype(np.float32)
        row, col = (rng.normal(0, 0.4, k).astype(np.float32) for _ in "rc")
        gi, gr, gc = gpu.separable_adjoint(torch.from_numpy(img).cuda(), torch.from_numpy(gout).cuda(), row, col,
                                           boundary=boundary, const=0.25)
        ri, rr, rc = oracle.separable_adjoint(img, gout, row, col, boundary, 0.25)
        assert _close(gi.cpu().numpy(), ri), (h, w)
        # |g_t| <= sum |col| |g| and |t| <= sum |row| |x|, each pixel reached at most by K taps per axis
        most = np.abs(gout).sum() * max(np.abs(row).sum(), 1.0) * max(np.abs(col).sum(), 1.0) * max(1.0, img.max())
        assert np.abs(gr.cpu().numpy() - rr).max() <= 3e-6 * most, (h, w)
        assert np.abs(gc.cpu().numpy() - rc).max() <= 3e-6 * most, (h, w)
        # each output alone (the other kernels' forms)
        x, g = torch.from_numpy(img).cuda(), torch.from_numpy(gout).cuda()
        only, _, _ = gpu.separable_adjoint(x, g, row, col, boundary=boundary, const=0.25, want_grad_taps=False)
        assert torch.equal(only, gi)
        _, r2, c2 = gpu.separable_adjoint(x, g, row, col, boundary=boundary, const=0.25, want_grad_in=False)
        assert torch.equal(r2, gr) and torch.equal(c2, gc)


@pytest.mark.parametrize("boundary", [1, 2, 3, 4])
@pytest.mark.parametrize("shape", [(1, 3), (9, 1), (1, 15), (13, 1)])
def test_line_mask_adjoint(gpu, oracle, shape, boundary):
    rng = np.random.default_rng(sum(shape) + boundary)
    for h, w in SIZES:
        img = rng.random((2, h, w + 3)).astype(np.float32)
        gout = rng.normal(0, 1, (2, h, w)).astype(np.float32)
        m = rng.normal(0, 0.4, shape).astype(np.float32)
        x = torch.from_numpy(img).cuda()[:, :, :w]  # rows that start off 16-byte boundaries
        g = torch.from_numpy(gout).cuda()
        host = gpu.local_op_adjoint(g, m, boundary=boundary, inp=x)
        dev = gpu.local_op_adjoint(g, torch.from_numpy(m).cuda(), boundary=boundary, inp=x)
        assert torch.equal(host[0], dev[0]) and torch.equal(host[1], dev[1])
        ref_m = 0.0
        for b in range(2):
            ri, rm = oracle.local_op_adjoint(img[b][:, :w], gout[b], m, boundary)
            assert _close(host[0][b].cpu().numpy(), ri), (h, w)
            ref_m = ref_m + rm
        assert np.abs(host[1].cpu().numpy() - ref_m).max() <= 3e-6 * np.abs(gout).sum()


@pytest.mark.parametrize("boundary", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("k", [3, 5, 7])
def test_square_mask_adjoint_tiles(gpu, oracle, k, boundary):
    """conv_adjoint.cu at the edges of its 64 x 8 and 64 x 32 tiles, on images smaller
    than the mask and on rows off 16-byte boundaries: each gradient alone and both.
    Pixels fold K^2 products (and a few pre-images), tap gradients at most 16 per
    thread and tile, a warp and a CTA tree: the bounds of the line masks hold."""
    rng = np.random.default_rng(10 * k + boundary)
    for h, w in SIZES + [(8, 64), (9, 66)]:
        img = rng.random((2, h, w + 1)).astype(np.float32)
        gout = rng.normal(0, 1, (2, h, w)).astype(np.float32)
        m = rng.random((k, k)).astype(np.float32)
        x, g = torch.from_numpy(img).cuda()[:, :, :w], torch.from_numpy(gout).cuda()
        gi, gm = gpu.local_op_adjoint(g, torch.from_numpy(m).cuda(), boundary=boundary, inp=x)
        alone, _ = gpu.local_op_adjoint(g, m, boundary=boundary, want_grad_mask=False)
        _, gm2 = gpu.local_op_adjoint(g, m, boundary=boundary, inp=x, want_grad_in=False)
        assert torch.equal(gi, alone) and torch.equal(gm, gm2)
        ref_m = 0.0
        for b in range(2):
            ri, rm = oracle.local_op_adjoint(img[b][:, :w], gout[b], m, boundary)
            # positive masks and random signs: compare with the sum of the magnitudes too
            scale = np.linalg.norm(oracle.local_op_adjoint(img[b][:, :w], np.abs(gout[b]), m, boundary)[0])
            assert np.linalg.norm(gi[b].cpu().numpy() - ri) <= 2e-6 * scale, (h, w)
            ref_m = ref_m + rm
        assert np.abs(gm.cpu().numpy() - ref_m).max() <= 3e-6 * np.abs(gout).sum(), (h, w)
