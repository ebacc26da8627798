"""Global NCC of images on a large offset: the moments are as accurate as sums
in float64, whose own error grows with the square of mean / sigma."""

import pytest
import torch

from nanodrr_gb300.registration import ncc_score

pytestmark = pytest.mark.gpu


# Root mean square over 32 planes of the error against centred float64. Sums of
# the raw moments in float64, in the kernel's order, give 1.0e-8 and 6e-7 at a
# mean of 1e4 and 1e5 sigma (numpy); the float32 rounding of the score adds
# 2e-8. Four times the first, plus the second. (Pairs of floats without a
# shift: 8e-8 and 8e-6.)
@pytest.mark.parametrize("offset,tol", [(0.0, 4e-8), (1e3, 4e-8), (1e4, 6e-8), (1e5, 2.5e-6)])
@pytest.mark.parametrize("shape", [(128, 128), (97, 131)])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_offset(shape, offset, tol, sign):
    g = torch.Generator().manual_seed(11)
    n1, n2 = torch.randn(32, 1, *shape, generator=g), torch.randn(32, 1, *shape, generator=g)
    x1, x2 = (n1 + offset).float(), sign * (0.6 * n1 + 0.8 * n2 + 0.7 * offset).float()
    s = ncc_score(x1.cuda(), x2.cuda(), 1e-7).cpu().double()
    a, b = (x.double() - x.double().mean((2, 3), keepdim=True) for x in (x1, x2))
    eps = float(torch.tensor(1e-7))
    r = (a * b).mean((1, 2, 3)) / ((a * a).mean((1, 2, 3)) + eps).sqrt() / ((b * b).mean((1, 2, 3)) + eps).sqrt()
    assert float((s - r).square().mean().sqrt()) <= tol


@pytest.mark.parametrize("first", [0.0, -3e5, 7.0])
def test_a_first_pixel_unlike_the_others(first):
    """The shift is a pixel of the image, whatever its value."""
    g = torch.Generator().manual_seed(12)
    x1 = torch.rand(4, 1, 40, 61, generator=g) + 50.0
    x2 = 0.5 * x1 + torch.rand(4, 1, 40, 61, generator=g)
    x1[..., 0, 0], x2[..., 0, 0] = first, 1.0
    s = ncc_score(x1.cuda(), x2.cuda(), 1e-7).cpu().double()
    a, b = (x.double() - x.double().mean((2, 3), keepdim=True) for x in (x1, x2))
    r = (a * b).mean((1, 2, 3)) / ((a * a).mean((1, 2, 3)) + 1e-7).sqrt() / ((b * b).mean((1, 2, 3)) + 1e-7).sqrt()
    assert float((s - r).abs().max()) <= 1.2e-7  # two float32 roundings


def test_constant_images_score_zero():
    x = torch.full((2, 1, 33, 50), 0.1, device="cuda", requires_grad=True)
    y = torch.rand(2, 1, 33, 50).cuda()
    s = ncc_score(x, y, 1e-4)
    s.sum().backward()
    assert float(s.detach().abs().max()) <= 1e-6 and bool(torch.isfinite(x.grad).all())
