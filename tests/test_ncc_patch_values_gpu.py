"""Local NCC where windows hold NaN, infinities or one value: the windows
around them, against the unfolded windows."""

import pytest
import torch

from nanodrr_gb300.registration import NormalizedCrossCorrelation2d, _to_patches, ncc_patch_score, ncc_score

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("at", [(0, 0), (20, 33), (39, 60), (17, 60)])
@pytest.mark.parametrize("p", [2, 5])
def test_a_bad_pixel_stays_in_its_windows(value, at, p):
    g = torch.Generator().manual_seed(p)
    x = torch.rand(2, 1, 40, 61, generator=g)
    y = x + torch.rand(2, 1, 40, 61, generator=g)
    x[1, 0, at[0], at[1]] = value
    results = []
    for f in (lambda a, b: ncc_patch_score(a, b, p, 1e-3),
              lambda a, b: ncc_score(_to_patches(a, p), _to_patches(b, p), 1e-3)):
        a, b = x.cuda().requires_grad_(True), y.cuda().requires_grad_(True)
        s = f(a, b)
        results.append([s.detach(), *torch.autograd.grad(s.sum(), (a, b))])
    touched = torch.zeros(2, 1, 40, 61, dtype=torch.bool)
    touched[1, 0, max(0, at[0] - p + 1) : at[0] + p, max(0, at[1] - p + 1) : at[1] + p] = True
    for i, (got, want) in enumerate(zip(*results)):
        bad = torch.isnan(got).cpu()
        assert torch.equal(bad, torch.isnan(want).cpu())
        assert torch.equal(bad, torch.tensor([False, True]) if i == 0 else touched)
        # both round the float64 sums to float32 once
        ok = ~bad
        d = (got.cpu() - want.cpu())[ok].abs().max()
        assert float(d) <= 1e-5 * float(want.cpu()[ok].abs().max())


def test_windows_of_one_value():
    """The variance of 0.1 (inexact) over a window is zero up to rounding; eps
    alone scales it."""
    g = torch.Generator().manual_seed(0)
    x = torch.full((1, 1, 24, 30), 0.1)
    x[..., 15:, :] = torch.rand(1, 1, 9, 30, generator=g)
    y = torch.rand(1, 1, 24, 30, generator=g)
    a, b = x.cuda().requires_grad_(True), y.cuda().requires_grad_(True)
    s = ncc_patch_score(a, b, 5, 1e-4)
    s.sum().backward()
    c, d = x.double().requires_grad_(True), y.double().requires_grad_(True)
    from oracle.ncc_oracle import ncc_oracle

    r = ncc_oracle(c, d, patch_size=5, eps=1e-4)
    r.sum().backward()
    assert float((s.detach().cpu().double() - r.detach()).abs().max()) <= 1e-5
    for u, v in ((a.grad, c.grad), (b.grad, d.grad)):
        assert float((u.cpu().double() - v).abs().max()) <= 1e-5 * float(v.abs().max())


def test_a_window_size_of_true_is_refused():
    x = torch.rand(1, 1, 8, 8, device="cuda")
    with pytest.raises(TypeError):
        NormalizedCrossCorrelation2d(patch_size=True)(x, x)
