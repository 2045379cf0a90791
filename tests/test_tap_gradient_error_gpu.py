"""The FP32 rounding in the tap gradients of the tiled adjoints does not grow with the
image: images that give every CTA ten to thirty tiles, rows off 16-byte boundaries,
against FP64.

Bound.  A sum s rounds to FP32 with an error of standard deviation 0.416 u |s| (u =
2^-24; uniform within half an ulp, mantissas logarithmically spread).  Products of
random sign: a partial sum of n of them has variance n sigma^2, so a level in which
all N products are in partial sums of any size adds (0.416 u)^2 N sigma^2, and a
chain of L additions (L + 1) / 2 times that.  A thread's chain within a tile is 16
long in conv_adjoint.cu, 8 and an addition of two in the line kernels; three FP32
exchanges and the rounding of the result follow: 12.5 and 9.5 levels.  The errors'
root mean square over taps and draws may be 1.5 times as large.  (A chain through all
tiles of a CTA is 3.5 to 6.4 u sqrt(sum p^2); the bounds are 2.2 and 1.9.)"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _exact(x, g, mh, mw):
    """Tap gradients with CLAMP and the sums of the squared products, FP64."""
    h, w = x.shape[1:]
    xp = torch.nn.functional.pad(x[:, None], (mw // 2, mw // 2, mh // 2, mh // 2), mode="replicate")[:, 0]
    s = torch.zeros((2, mh, mw), dtype=torch.float64)
    for i in range(mh):
        for j in range(mw):
            for b in range(x.shape[0]):
                p = xp[b, i:i + h, j:j + w].double() * g[b].double()
                s[0, i, j] += p.sum().item()
                s[1, i, j] += (p * p).sum().item()
    return s


@pytest.mark.parametrize("want_in", [False, True])
@pytest.mark.parametrize("n,h,w,mh,mw", [(1, 6001, 6003, 7, 7), (2, 3001, 3003, 3, 3), (40, 1021, 1019, 1, 9),
                                         (16, 1031, 1999, 9, 1)])
def test_error_does_not_grow_with_the_image(gpu, n, h, w, mh, mw, want_in):
    levels = 12.5 if mh == mw else 9.5
    mask = np.full((mh, mw), 1.0 / (mh * mw), np.float32)
    gen = torch.Generator(device="cuda").manual_seed(mh + 10 * mw)
    scaled = []
    for _ in range(2 if mh == mw == 7 else 5):
        x = torch.rand((n, h, w), device="cuda", generator=gen)
        g = torch.randn((n, h, w), device="cuda", generator=gen)
        _, gm = gpu.local_op_adjoint(g, mask, boundary=gpu.CLAMP, inp=x, want_grad_in=want_in)
        ref, squares = _exact(x, g, mh, mw)
        scaled.append(((gm.double().cpu() - ref) / (2.0 ** -24 * squares.sqrt())).flatten())
    rms = torch.cat(scaled).pow(2).mean().sqrt().item()
    print(f"{mh}x{mw}: {rms:.2f} u sqrt(sum p^2), bound {1.5 * 0.416 * levels ** 0.5:.2f}")
    assert rms <= 1.5 * 0.416 * levels ** 0.5
