"""Global NCC moments in float pairs: chunk edges, several planes, and pixel
ranges where the products leave float's range (summed in float64)."""

import pytest
import torch

from nanodrr_gb300.registration import ncc_score
from oracle.ncc_oracle import ncc_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (2, 1, 1, 1023), (1, 3, 4, 256), (3, 1, 25, 41), (2, 2, 200, 211)])
@pytest.mark.parametrize("scale", [1.0, 1e-17, 1e17])
def test_moments_over_chunks_and_ranges(shape, scale):
    g = torch.Generator().manual_seed(shape[-1])
    x1 = ((torch.rand(shape, generator=g) + 3.0) * scale).float()
    x2 = (x1 + torch.rand(shape, generator=g) * scale).float()
    eps = float(scale) ** 2 * 1e-6 if scale < 1 else 1e-7
    s = ncc_score(x1.cuda(), x2.cuda(), eps)
    r = ncc_oracle(x1.double(), x2.double(), eps=float(torch.tensor(eps, dtype=torch.float32)))
    # one float32 rounding per plane score and one of the mean
    assert float((s.cpu().double() - r).abs().max()) <= 1e-6


def test_a_nan_pixel_reaches_its_own_score_only():
    x = torch.rand(3, 1, 40, 40)
    y = x.clone()
    y[1, 0, 3, 3] = float("nan")
    s = ncc_score(y.cuda(), x.cuda())
    assert torch.isnan(s).tolist() == [False, True, False]
