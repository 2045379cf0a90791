"""The forms that large images and batches take.  Most operators pick rows per thread
(or columns, or the kernel) from the number of tiles against the number of SMs; the
other tests' images are small and take the small forms.  Here a batch of copies of
three small ragged images has as many tiles as the rule asks for, counted from the
device's SMs, so the oracle stays cheap: every copy of an image gives the same result,
and sums over the batch are the images' sums times their copies.

Tolerances are those of the small forms (test_line_adjoint_gpu.py, derived there from
FP32 rounding): 2e-6 relative (L2) for gradient pixels, 3e-6 of the sum of magnitudes
for tap gradients.  adj_fused_kernel chains 4 products per thread and tile through at
most 7 tiles, 8 warp sums and 5 exchanges: 41 u = 2.5e-6 of the sum.  Whole numbers,
minima and maxima, and forms that fold the same terms in the same order are equal bit
for bit."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SMS = 4 * 38  # replaced by the device's number when there is one
if torch.cuda.is_available():
    SMS = torch.cuda.get_device_properties(0).multi_processor_count
H, W = 67, 133  # 3 x 3 tiles of 64 x 32, 3 x 2 of 64 x 64, 3 x 5 of 64 x 16, 2 x 1 of 128 x 128
DISC5 = np.array([[0, 1, 1, 1, 0], [1, 1, 1, 1, 1], [1, 1, 1, 1, 1], [1, 1, 1, 1, 1], [0, 1, 1, 1, 0]], np.uint8)
DOMAINS = {"square3": np.ones((3, 3), np.uint8), "disc5": DISC5, "square7": np.ones((7, 7), np.uint8),
           "gap5": DISC5 * np.array([[1], [0], [1], [0], [1]], np.uint8)}


def _batch(per_image, tiles):
    return -(-tiles // per_image)


def _copies(images, n, pad=0):
    """n images on the device, image b a copy of images[b % 3]; `pad` elements behind each row."""
    k, h, w = images.shape
    buf = torch.zeros((n, h, w + pad), dtype=images.dtype, device="cuda")
    buf[:, :, :w] = images.cuda()[torch.arange(n, device="cuda") % k]
    return buf[:, :, :w]


def _check_copies(got):
    """Every copy equals the first of its image; the three firsts as numpy arrays."""
    first = got[:3][torch.arange(got.shape[0], device="cuda") % 3]
    assert torch.equal(got, first)
    return [got[b].double().cpu().numpy() for b in range(3)]


def _weights(n):
    return [len(range(b, n, 3)) for b in range(3)]


def _close(got, ref, scale=None):
    return np.linalg.norm(got - ref) <= 2e-6 * max(np.linalg.norm(ref) if scale is None else scale, 1e-30)


def _floats(seed, h=H, w=W, signed=False):
    rng = np.random.default_rng(seed)
    a = rng.normal(0, 1, (3, h, w)) if signed else rng.random((3, h, w))
    return torch.from_numpy(a.astype(np.float32))


@pytest.mark.parametrize("boundary", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("k", [3, 5, 7])
@pytest.mark.parametrize("h,w", [(41, 132), (33, 64)])
def test_fused_square_mask_adjoint(gpu, oracle, k, boundary, h, w):
    """adj_fused_kernel: both gradients, rows of whole 16 bytes, four 64 x 32 tiles per SM."""
    n = _batch(math.ceil(w / 64) * math.ceil(h / 32), 4 * SMS)
    img, gout = _floats(k, h, w), _floats(k + 100, h, w, True)
    m = np.random.default_rng(k).random((k, k)).astype(np.float32)
    x, g = _copies(img, n), _copies(gout, n)
    gi, gm = gpu.local_op_adjoint(g, m, boundary=boundary, inp=x)
    _, again = gpu.local_op_adjoint(g, torch.from_numpy(m).cuda(), boundary=boundary, inp=x)
    assert torch.equal(gm, again)
    got, ref_m = _check_copies(gi), 0.0
    for b, c in enumerate(_weights(n)):
        ri, rm = oracle.local_op_adjoint(img[b].numpy(), gout[b].numpy(), m, boundary)
        scale = np.linalg.norm(oracle.local_op_adjoint(img[b].numpy(), gout[b].abs().numpy(), m, boundary)[0])
        assert _close(got[b], ri, scale), b
        ref_m = ref_m + c * rm
    assert np.abs(gm.cpu().numpy() - ref_m).max() <= 3e-6 * g.abs().double().sum().item()


@pytest.mark.parametrize("k", [3, 5, 7])
@pytest.mark.parametrize("step", [-1, 0])
def test_square_mask_adjoint_about_the_line(gpu, oracle, step, k):
    """The last batch of the tiled kernel and the first of the fused one: 1.5 (3 x 3) or 4 tiles per SM."""
    h, w = 41, 132  # 6 tiles
    n = _batch(6, -(-3 * SMS // 2) if k == 3 else 4 * SMS) + step
    img, gout = _floats(k + 4, h, w), _floats(k + 104, h, w, True)
    m = np.random.default_rng(k).random((k, k)).astype(np.float32)
    x, g = _copies(img, n), _copies(gout, n)
    gi, gm = gpu.local_op_adjoint(g, m, boundary=3, inp=x)
    got, ref_m = _check_copies(gi), 0.0
    for b, c in enumerate(_weights(n)):
        ri, rm = oracle.local_op_adjoint(img[b].numpy(), gout[b].numpy(), m, 3)
        scale = np.linalg.norm(oracle.local_op_adjoint(img[b].numpy(), gout[b].abs().numpy(), m, 3)[0])
        assert _close(got[b], ri, scale), b
        ref_m = ref_m + c * rm
    assert np.abs(gm.cpu().numpy() - ref_m).max() <= 3e-6 * g.abs().double().sum().item()


@pytest.mark.parametrize("boundary", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("k", [3, 5, 7])
def test_square_mask_adjoint_four_rows(gpu, oracle, k, boundary):
    """conv_adjoint_kernel with four rows per thread, at least three tiles per CTA (six CTAs an SM at most)."""
    n = _batch(9, 3 * 6 * SMS)
    img, gout = _floats(k + 1), _floats(k + 101, signed=True)
    m = np.random.default_rng(k).random((k, k)).astype(np.float32)
    x, g = _copies(img, n, pad=2), _copies(gout, n)
    gi, gm = gpu.local_op_adjoint(g, m, boundary=boundary, inp=x)
    alone, _ = gpu.local_op_adjoint(g, m, boundary=boundary, want_grad_mask=False)
    _, gm2 = gpu.local_op_adjoint(g, torch.from_numpy(m).cuda(), boundary=boundary, inp=x, want_grad_in=False)
    assert torch.equal(gi, alone) and torch.equal(gm, gm2)
    got, ref_m = _check_copies(gi), 0.0
    for b, c in enumerate(_weights(n)):
        ri, rm = oracle.local_op_adjoint(img[b].numpy(), gout[b].numpy(), m, boundary)
        scale = np.linalg.norm(oracle.local_op_adjoint(img[b].numpy(), gout[b].abs().numpy(), m, boundary)[0])
        assert _close(got[b], ri, scale), b
        ref_m = ref_m + c * rm
    assert np.abs(gm.cpu().numpy() - ref_m).max() <= 3e-6 * g.abs().double().sum().item()


@pytest.mark.parametrize("boundary", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("k", [3, 5, 7, 9, 11, 13, 15])
def test_line_adjoints_four_rows(gpu, oracle, k, boundary):
    """line_adjoint_kernel with four rows per thread, every form (rows, columns, columns of the
    recomputed row pass), three tiles per CTA or more (16 CTAs of 128 threads an SM at most)."""
    n = _batch(9, 3 * 16 * SMS)
    img, gout = _floats(k + 2), _floats(k + 102, signed=True)
    rng = np.random.default_rng(k)
    row, col = (rng.normal(0, 0.4, k).astype(np.float32) for _ in "rc")
    x, g = _copies(img, n, pad=1), _copies(gout, n)
    total = g.abs().double().sum().item()
    # separable: the column pass with the recomputed rows, then the row pass
    gi, gr, gc = gpu.separable_adjoint(x, g, row, col, boundary=boundary, const=0.25)
    only, _, _ = gpu.separable_adjoint(x, g, row, col, boundary=boundary, const=0.25, want_grad_taps=False)
    assert torch.equal(gi, only)
    got, ref_r, ref_c = _check_copies(gi), 0.0, 0.0
    for b, c in enumerate(_weights(n)):
        ri, rr, rc = oracle.separable_adjoint(img[b].numpy(), gout[b].numpy(), row, col, boundary, 0.25)
        assert _close(got[b], ri), b
        ref_r, ref_c = ref_r + c * rr, ref_c + c * rc
    most = total * max(np.abs(row).sum(), 1.0) * max(np.abs(col).sum(), 1.0)
    assert np.abs(gr.cpu().numpy() - ref_r).max() <= 3e-6 * most
    assert np.abs(gc.cpu().numpy() - ref_c).max() <= 3e-6 * most
    # a single line, taps on the host and on the device
    for m in (row[None, :], col[:, None]):
        m = np.ascontiguousarray(m)
        gi, gm = gpu.local_op_adjoint(g, m, boundary=boundary, inp=x)
        di, dm = gpu.local_op_adjoint(g, torch.from_numpy(m).cuda(), boundary=boundary, inp=x)
        assert torch.equal(gi, di) and torch.equal(gm, dm)
        got, ref_m = _check_copies(gi), 0.0
        for b, c in enumerate(_weights(n)):
            ri, rm = oracle.local_op_adjoint(img[b].numpy(), gout[b].numpy(), m, boundary)
            assert _close(got[b], ri), b
            ref_m = ref_m + c * rm
        assert np.abs(gm.cpu().numpy() - ref_m).max() <= 3e-6 * total


@pytest.mark.parametrize("red", [1, 2])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.uint8])
@pytest.mark.parametrize("name", sorted(DOMAINS))
@pytest.mark.parametrize("per_image", [9, 6])  # tiles of 32 and of 64 rows: four and eight rows per thread
def test_minmax_domain_tall_tiles(gpu, oracle, per_image, name, dtype, red):
    n = _batch(per_image, 4 * SMS)
    assert per_image == 6 or 6 * n < 4 * SMS
    rng = np.random.default_rng(red)
    img = torch.from_numpy(rng.integers(0, 200, (3, H, W)).astype(np.float32)).to(dtype)
    for boundary in (0, 1, 2, 3, 4):
        for pad in (0, 3):
            x = _copies(img, n, pad)
            got = gpu.local_op(x, torch.zeros_like(x), domain=DOMAINS[name], reduce=red, boundary=boundary, const=7.0)
            for b, y in enumerate(_check_copies(got)):
                ref = oracle.local_op(img[b].float().numpy(), domain=DOMAINS[name], reduce=red, boundary=boundary,
                                      const=7.0)
                assert np.array_equal(y, ref), (boundary, pad, b)


@pytest.mark.parametrize("red", [1, 2])
@pytest.mark.parametrize("boundary", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("name", sorted(DOMAINS))
@pytest.mark.parametrize("per_image", [15, 9])  # tiles of 16 and of 32 rows: two and four rows per thread
def test_minmax_adjoint_tall_tiles(gpu, oracle, per_image, name, boundary, red):
    n = _batch(per_image, 8 * SMS)
    assert per_image == 9 or 9 * n < 8 * SMS
    rng = np.random.default_rng(boundary)
    img = torch.from_numpy(rng.integers(0, 9, (3, H, W)).astype(np.float32))  # ties
    gout = _floats(boundary + 3, signed=True)
    gi = gpu.minmax_adjoint(_copies(img, n), _copies(gout, n), red, domain=DOMAINS[name], boundary=boundary, const=4.0)
    for b, got in enumerate(_check_copies(gi)):
        _, ref = oracle.minmax_adjoint(img[b].numpy(), gout[b].numpy(), red, domain=DOMAINS[name], boundary=boundary,
                                       const=4.0)
        assert _close(got, ref), b


@pytest.mark.parametrize("boundary", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("pad", [0, 11])  # rows that TMA cannot address, and rows of 144 bytes that it can
def test_sobel_tall_tiles(gpu, oracle, pad, boundary):
    h = 131  # 2 x 2 tiles of 128 x 128
    n = _batch(4, 4 * SMS)
    img = torch.from_numpy(np.random.default_rng(boundary).integers(0, 256, (3, h, W), dtype=np.uint8))
    x, y = _copies(img, n, pad), torch.zeros((n, h, W + pad), dtype=torch.uint8, device="cuda")[:, :, :W]
    s = torch.zeros(1, dtype=torch.int64, device="cuda")
    m = torch.zeros(1, dtype=torch.int32, device="cuda")
    gpu.sobel_mag(x, y, boundary=boundary, const=17, sum_out=s, max_out=m)
    total, most = 0, 0
    for b, (got, c) in enumerate(zip(_check_copies(y), _weights(n))):
        ref = oracle.sobel_mag(img[b].numpy(), boundary=boundary, const=17)
        assert np.array_equal(got, ref), b
        total, most = total + c * int(ref.astype(np.uint64).sum()), max(most, int(ref.max()))
    assert s.item() == total and m.item() == most


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("size", [3, 5, 7, 9, 11, 13])
def test_bilateral_four_columns(gpu, oracle, size, dtype):
    """Four columns per thread (from four 64 x 32 tiles per SM on) against the two-column form of a
    single image, which the oracle checks elsewhere: the same taps in the same order."""
    n = _batch(9, 4 * SMS)
    img = _floats(size).to(dtype)
    sm = oracle.spatial_mask(size, size / 4.0)
    for boundary in (0, 1, 2, 3, 4):
        for pad in (0, 3):
            x = _copies(img, n, pad)
            y = torch.zeros((n, H, W + pad), dtype=dtype, device="cuda")[:, :, :W]
            gpu.bilateral(x, y, sm, 0.15, boundary=boundary, const=0.5)
            _check_copies(y)
            for b in range(3):
                one = gpu.bilateral(x[b], torch.zeros_like(x[b]), sm, 0.15, boundary=boundary, const=0.5)
                assert torch.equal(one, y[b]), (boundary, pad, b)


@pytest.mark.parametrize("boundary", [0, 1, 2, 3, 4])
def test_harris_tall_tiles_and_unsharp_long_segments(gpu, oracle, boundary):
    """64-row tiles of the Harris kernel; segments of the Unsharp kernel longer than two rows (two
    strips of 120 columns per image, at most 64 warps an SM: 11 rows each or more)."""
    n = _batch(4, 4 * SMS)
    rng = np.random.default_rng(boundary)
    img = torch.from_numpy(rng.integers(0, 256, (3, H, W), dtype=np.uint8).repeat(2, axis=2)[:, :, :W].copy())
    got = gpu.harris(_copies(img, n, 3), boundary=boundary, threshold=300.0)
    for b, y in enumerate(_check_copies(got)):
        assert np.array_equal(y, oracle.harris(img[b].numpy(), boundary=boundary, threshold=300.0)), b
    rgba = rng.integers(0, 256, (3, H, W, 4), dtype=np.uint8)
    of = torch.arange(5 * SMS, device="cuda") % 3
    out = gpu.unsharp(torch.from_numpy(rgba).cuda()[of].contiguous(), boundary=boundary)
    assert torch.equal(out, out[:3][of])
    for b in range(3):
        assert np.array_equal(out[b].cpu().numpy(), oracle.unsharp(rgba[b], boundary=boundary)[0]), b
