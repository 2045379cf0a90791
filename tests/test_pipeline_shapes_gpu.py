"""Launch shapes of the fused Harris and Unsharp kernels and the word staging that Harris
and Sobel share, at the sizes where they change: Harris tiles of 8, 16 and 64 rows, Unsharp
strips of one and two pairs per lane with one to many rows per warp, byte images of every
row alignment whose edges fall on each byte of a word.  Whole numbers: equal bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(8, 9), (64, 64), (590, 336), (480, 640), (600, 800), (300, 1500), (2428, 192), (720, 1280), (1080, 1920)]


@pytest.mark.parametrize("hw", SIZES)
def test_harris_every_tile_height(gpu, oracle, hw):
    rng = np.random.default_rng(hw[0])
    img = np.kron(rng.integers(0, 256, (hw[0] // 4 + 1, hw[1] // 4 + 1)), np.ones((4, 4)))[:hw[0], :hw[1]]
    img = (img + rng.integers(0, 4, hw)).clip(0, 255).astype(np.uint8)
    for boundary in (0, 1, 2, 3, 4):
        out = gpu.harris(torch.from_numpy(img).cuda(), boundary=boundary)
        assert np.array_equal(out.cpu().numpy(), oracle.harris(img, boundary)), boundary


@pytest.mark.parametrize("hw", SIZES + [(1, 1), (3, 61), (5, 121), (31, 60), (40, 119)])
def test_unsharp_every_shape(gpu, oracle, hw):
    rng = np.random.default_rng(hw[1])
    rgba = rng.integers(0, 256, hw + (4,), dtype=np.uint8)
    for boundary in (0, 1, 2, 3, 4):
        out = gpu.unsharp(torch.from_numpy(rgba).cuda(), boundary=boundary)
        assert np.array_equal(out.cpu().numpy(), oracle.unsharp(rgba, boundary)[0]), boundary


@pytest.mark.parametrize("offset", [0, 1, 2, 3])  # of the first pixel from a word
@pytest.mark.parametrize("w", [1, 2, 3, 4, 5, 7, 8, 9, 12, 13, 126, 127, 128, 129, 131, 133, 143, 144, 145, 149, 257])
def test_word_staging_at_every_edge(gpu, oracle, w, offset):
    h, pitch = 37, 263
    rng = np.random.default_rng(w)
    img = rng.integers(0, 256, (h, w), dtype=np.uint8)
    buf = torch.full((h * pitch + 8,), 201, dtype=torch.uint8, device="cuda")
    x = buf[offset:offset + h * pitch].view(h, pitch)[:, :w]
    x.copy_(torch.from_numpy(img))
    for boundary in (1, 2, 3, 4):
        ref = oracle.sobel_mag(img, boundary=boundary, const=17)
        out = gpu.sobel_mag(x, torch.zeros((h, w), dtype=torch.uint8, device="cuda"), boundary=boundary, const=17)
        assert np.array_equal(out.cpu().numpy(), ref), boundary
        out = gpu.harris(x, torch.zeros((h, w), dtype=torch.uint8, device="cuda"), threshold=50.0, boundary=boundary)
        assert np.array_equal(out.cpu().numpy(), oracle.harris(img, boundary, threshold=50.0)), boundary
