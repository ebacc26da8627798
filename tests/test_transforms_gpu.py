"""Renders whose poses are batched by torch.func.vmap or are fake: the affine
is a tensor expression there, as it has no pointer to launch with."""

import pytest
import torch
from torch._subclasses import FakeTensorMode

import nanodrr_gb300 as nd

pytestmark = pytest.mark.gpu
H, W = 9, 11


def _scene(B=3):
    g = torch.Generator().manual_seed(1)
    sub = nd.Subject.from_volume(torch.rand(14, 15, 16, generator=g).cuda(), (4.0, 4.0, 4.0), convert_to_mu=False)
    sub._image_hu = sub._image_hu.detach().clone().requires_grad_(True)
    rt = nd.make_rt_inv(40.0 * torch.rand(B, 3, generator=g), torch.tensor([[0.0, 200.0, 0.0]]).expand(B, 3)).cuda()
    return sub, rt, nd.make_k_inv(400.0, 9.0, 9.0, 0.0, 0.0, H, W).cuda(), torch.tensor([400.0], device="cuda")


@pytest.mark.parametrize("layout", ["quad", "plain"])
def test_vmap_over_poses(layout):
    sub, rt, k, s = _scene()
    sub.layout = layout
    one = lambda r: nd.render(sub, k, r[None], s, H, W, n_samples=40)[0]  # noqa: E731
    results = []
    for imgs in (torch.func.vmap(one)(rt), nd.render(sub, k, rt, s, H, W, n_samples=40)):
        (gvol,) = torch.autograd.grad(imgs.square().sum(), sub._image_hu)
        results.append((imgs.detach(), gvol))
    (ia, va), (ib, vb) = results
    assert torch.equal(ia, ib)
    # scattered sums add in no fixed order
    assert float((va - vb).abs().max()) <= 1e-5 * float(vb.abs().max())


def test_fake_calibration_step():
    sub, rt, k, s = _scene()
    sub.layout = "plain"
    with FakeTensorMode(allow_non_fake_inputs=True) as mode:
        kf = mode.from_tensor(k).requires_grad_(True)
        img = nd.render(sub, kf, mode.from_tensor(rt), mode.from_tensor(s), H, W, n_samples=40)
        assert tuple(img.shape) == (3, 1, H, W)
        (g,) = torch.autograd.grad(img.sum(), kf)
        assert g.shape == k.shape
