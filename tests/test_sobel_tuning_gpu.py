"""hgb_sobel_mag on small images follows the tuner: with tuning on a call stores a
choice for its shape, and a loaded choice of any form, the low tiles' number included,
gives the oracle's bits (whole numbers: no tolerance)."""
import json

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _pitched(img):
    h, w = img.shape
    dev = torch.zeros((h, (w + 15) // 16 * 16), dtype=torch.uint8, device="cuda")
    dev[:, :w] = torch.from_numpy(img).cuda()
    return dev[:, :w]


def test_small_images_are_tuned(gpu, oracle, tmp_path):
    from hipacc_gb300 import _lib as L

    img = np.random.default_rng(0).integers(0, 256, (75, 333), dtype=np.uint8)
    ref = oracle.sobel_mag(img, boundary=3)
    x = _pitched(img)
    f = tmp_path / "choices.json"
    try:
        L.call("hgb_autotune_clear")
        L.call("hgb_autotune_enable", 1)
        out = gpu.sobel_mag(x, torch.zeros_like(x))
        L.call("hgb_autotune_enable", 0)
        assert L.load().hgb_autotune_count() == 1
        L.call("hgb_autotune_save", str(f).encode())
        assert list(json.loads(f.read_text())) == ["sobel3:512x128x1"]
        assert np.array_equal(out.cpu().numpy(), ref)
    finally:
        L.call("hgb_autotune_enable", 0)
        L.call("hgb_autotune_clear")


@pytest.mark.parametrize("cfg", [0, 1, 2, 3, 4, 5, 6])  # 6 is none: the untuned form
@pytest.mark.parametrize("hw", [(1, 64), (33, 129), (31, 300), (257, 390), (700, 1300)])
def test_every_form_by_a_loaded_choice(gpu, oracle, cfg, hw, tmp_path):
    from hipacc_gb300 import _lib as L

    h, w = hw
    img = np.random.default_rng(h + cfg).integers(0, 256, hw, dtype=np.uint8)
    x = _pitched(img)
    f = tmp_path / "choices.json"
    f.write_text(json.dumps({"sobel3:%dx%dx1" % (1 << w.bit_length(), 1 << h.bit_length()): [cfg, 0.0]}))
    s = torch.zeros(1, dtype=torch.int64, device="cuda")
    m = torch.zeros(1, dtype=torch.int32, device="cuda")
    try:
        L.call("hgb_autotune_clear")
        L.call("hgb_autotune_load", str(f).encode())
        for boundary in (1, 2, 3, 4):
            ref = oracle.sobel_mag(img, boundary=boundary, const=17)
            out = gpu.sobel_mag(x, torch.zeros_like(x), boundary=boundary, const=17, sum_out=s, max_out=m)
            assert np.array_equal(out.cpu().numpy(), ref), boundary
            assert s.item() == int(ref.astype(np.uint64).sum()) and m.item() == int(ref.max())
    finally:
        L.call("hgb_autotune_clear")
