"""Local NCC (window kernels) against the float64 restatement that unfolds the
windows: window sizes around the four-window split, images of one window, one
tile and ragged tiles, several channels, both gradients, 16-bit images."""

import pytest
import torch

from nanodrr_gb300.registration import NormalizedCrossCorrelation2d
from oracle.ncc_oracle import ncc_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,shape", [
    (1, (1, 1, 5, 7)), (2, (2, 1, 2, 33)), (3, (1, 2, 18, 35)), (4, (1, 1, 4, 4)), (5, (2, 3, 20, 36)),
    (13, (2, 1, 13, 61)), (16, (1, 1, 47, 50)), (128, (1, 1, 128, 130)),
])
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 1e-2)])
def test_local_ncc(p, shape, dtype, tol):
    g = torch.Generator().manual_seed(p)
    x1 = (torch.rand(shape, generator=g) + 2.0).to(dtype).cuda().requires_grad_(True)
    x2 = (x1.detach().cpu().float() * 0.5 + torch.rand(shape, generator=g)).to(dtype).cuda().requires_grad_(True)
    go = torch.randn(shape[0], generator=g).to(dtype)
    s = NormalizedCrossCorrelation2d(patch_size=p, eps=1e-3)(x1, x2)
    s.backward(go.cuda())
    d1, d2 = (x.detach().cpu().double().requires_grad_(True) for x in (x1, x2))
    r = ncc_oracle(d1, d2, patch_size=p, eps=1e-3)
    r.backward(go.double())
    # float32 (bfloat16) roundings of the inputs' eps, the score and the gradients
    assert s.dtype == dtype and float((s.detach().cpu().double() - r.detach()).abs().max()) <= tol
    for a, b in ((x1.grad, d1.grad), (x2.grad, d2.grad)):
        assert a.dtype == dtype and float((a.cpu().double() - b).abs().max()) <= tol * max(float(b.abs().max()), 1e-6)


def test_windows_that_do_not_fit_are_refused():
    x = torch.rand(1, 1, 6, 9, device="cuda")
    with pytest.raises(RuntimeError):
        NormalizedCrossCorrelation2d(patch_size=7)(x, x)
    with pytest.raises(ValueError):
        NormalizedCrossCorrelation2d(patch_size=3)(x, x[..., :8])
    # above the kernels' largest window the images are unfolded
    y = torch.rand(1, 1, 131, 131, device="cuda")
    assert abs(float(NormalizedCrossCorrelation2d(patch_size=130)(y, y)) - 1.0) < 1e-4
