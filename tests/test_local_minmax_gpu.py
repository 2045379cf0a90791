"""GPU parity of the tiled MIN / MAX Domain kernels (local_minmax.cu), bit for
bit: the oracle folds every output's cells in row-major order from FLT_MAX /
FLT_MIN, and minima and maxima round nothing, so every path must give the same
bits (the 16-bit and byte storages write the folded value through one
rounding of a value that they already hold, which changes nothing)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DISC5 = np.array([[0, 1, 1, 1, 0], [1, 1, 1, 1, 1], [1, 1, 1, 1, 1], [1, 1, 1, 1, 1], [0, 1, 1, 1, 0]], np.uint8)
RING3 = np.array([[1, 1, 1], [1, 0, 1], [1, 1, 1]], np.uint8)  # its middle row is no run: the general kernel
DOMAINS = {
    "square3": np.ones((3, 3), np.uint8), "disc5": DISC5, "square7": np.ones((7, 7), np.uint8),
    "cross3": np.array([[0, 1, 0], [1, 1, 1], [0, 1, 0]], np.uint8), "row7": np.ones((1, 7), np.uint8),
    "col5": np.ones((5, 1), np.uint8), "gap5": DISC5 * np.array([[1], [0], [1], [0], [1]], np.uint8), "ring3": RING3,
}
SIZES = [(1, 1), (3, 5), (32, 64), (31, 63), (33, 65), (70, 131)]


def _bits(a):
    return np.ascontiguousarray(a).view({1: np.uint8, 2: np.uint16, 4: np.uint32}[a.itemsize])


@pytest.mark.parametrize("red", [1, 2])
@pytest.mark.parametrize("boundary", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("name", sorted(DOMAINS))
def test_domain_minmax_f32(gpu, oracle, name, boundary, red):
    rng = np.random.default_rng(17 * boundary + red)
    for h, w in SIZES:
        img = (rng.random((h, w)) - 0.25).astype(np.float32)
        got = gpu.local_op(torch.from_numpy(img).cuda(), domain=DOMAINS[name], reduce=red, boundary=boundary, const=0.5)
        ref = oracle.local_op(img, domain=DOMAINS[name], reduce=red, boundary=boundary, const=0.5)
        assert np.array_equal(_bits(got.cpu().numpy()), _bits(ref)), (name, h, w)


@pytest.mark.parametrize("red", [1, 2])
@pytest.mark.parametrize("dtype", [torch.uint8, torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("pad", [0, 3, 4])  # elements behind each row: every row alignment
def test_domain_minmax_types_and_pitches(gpu, oracle, dtype, pad, red):
    rng = np.random.default_rng(5 + pad)
    for h, w in [(37, 141), (80, 250)]:
        buf = torch.from_numpy(rng.integers(0, 256, (2, h, w + pad)).astype(np.float32)).to(dtype).cuda()
        x = buf[:, :, :w]
        y = torch.zeros_like(buf)[:, :, :w]
        gpu.local_op(x, y, domain=DISC5, reduce=red, boundary=3)
        for b in range(2):
            ref = oracle.local_op(x[b].float().cpu().numpy(), domain=DISC5, reduce=red, boundary=3)
            assert np.array_equal(y[b].float().cpu().numpy(), ref), (h, w, pad)


@pytest.mark.parametrize("red", [1, 2])
def test_domain_minmax_special_values(gpu, oracle, red):
    """NaNs and negative zeros follow the stated fold (a NaN is replaced by the
    next cell, equal values by the later one); infinities and denormals too."""
    rng = np.random.default_rng(3)
    img = rng.normal(0, 1, (70, 200)).astype(np.float32)
    at = rng.integers(0, img.size, 400)
    img.flat[at] = rng.choice(np.array([np.nan, np.inf, -np.inf, -0.0, 0.0, 1e-40, -1e-40], np.float32), 400)
    img[:, 128:] = np.abs(img[:, 128:])
    img[:, 128:][~np.isfinite(img[:, 128:])] = np.inf  # tiles without NaNs beside tiles with them
    for dom in (DISC5, DOMAINS["square3"]):
        got = gpu.local_op(torch.from_numpy(img).cuda(), domain=dom, reduce=red, boundary=1).cpu().numpy()
        ref = oracle.local_op(img, domain=dom, reduce=red, boundary=1)
        assert np.array_equal(np.isnan(got), np.isnan(ref))
        ok = ~np.isnan(ref)
        assert np.array_equal(_bits(got)[ok], _bits(ref)[ok])


def test_domain_minmax_windows(gpu, oracle):
    rng = np.random.default_rng(8)
    img = rng.random((90, 150)).astype(np.float32)
    out = torch.zeros((100, 160), device="cuda")
    acc, it = (11, 7, 101, 66), (3, 5, 101, 66)
    gpu.local_op(torch.from_numpy(img).cuda(), out, domain=DISC5, reduce=2, boundary=2, acc=acc, iter_space=it)
    ref = np.zeros((100, 160), np.float32)
    oracle.local_op(img, domain=DISC5, reduce=2, boundary=2, acc=acc, out=ref, iter_space=it)
    assert np.array_equal(_bits(out.cpu().numpy()), _bits(ref))


@pytest.mark.parametrize("boundary", [1, 2, 3, 4])
def test_domain_minmax_space_larger_than_window(gpu, oracle, boundary):
    """Outputs beyond the accessor window read through the boundary at any distance."""
    rng = np.random.default_rng(boundary)
    img = rng.random((90, 150)).astype(np.float32)
    out = torch.zeros((100, 160), device="cuda")
    acc, it = (11, 7, 40, 30), (3, 5, 75, 61)
    gpu.local_op(torch.from_numpy(img).cuda(), out, domain=DISC5, reduce=2, boundary=boundary, acc=acc, iter_space=it,
                 const=0.3)
    ref = np.zeros((100, 160), np.float32)
    oracle.local_op(img, domain=DISC5, reduce=2, boundary=boundary, acc=acc, out=ref, iter_space=it, const=0.3)
    assert np.array_equal(_bits(out.cpu().numpy()), _bits(ref))


@pytest.mark.parametrize("red", [1, 2])
@pytest.mark.parametrize("boundary", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("name", ["square3", "disc5", "square7", "row7", "col5", "ring3"])
def test_domain_minmax_adjoint_tiles(gpu, oracle, name, boundary, red):
    """The tiled select / gather kernels at the edges of their 64 x 32 tiles and
    on images smaller than the window (pre-images on both sides of the image);
    small integers give ties.  At most 49 FP32 additions of a few pre-images
    per pixel: 2e-6 relative (L2) against the FP64 gather."""
    rng = np.random.default_rng(31 * boundary + red)
    for h, w in [(2, 3)] + SIZES:
        img = rng.integers(0, 9, (h, w)).astype(np.float32) if w % 2 else rng.random((h, w)).astype(np.float32)
        gout = rng.normal(0, 1, (h, w)).astype(np.float32)
        got = gpu.minmax_adjoint(torch.from_numpy(img).cuda(), torch.from_numpy(gout).cuda(), red, domain=DOMAINS[name],
                                 boundary=boundary, const=0.5).cpu().numpy()
        _, ref = oracle.minmax_adjoint(img, gout, red, domain=DOMAINS[name], boundary=boundary, const=0.5)
        assert np.linalg.norm(got - ref) <= 2e-6 * max(np.linalg.norm(ref), 1e-30), (name, h, w)
