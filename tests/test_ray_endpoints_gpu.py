"""Ray endpoints given to render without their batch dimension."""

import pytest
import torch

import nanodrr_gb300 as nd
from nanodrr_gb300.renderer import _camera_rays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 2])
@pytest.mark.parametrize("ortho", [False, True])
@pytest.mark.parametrize("grad", [False, True])
def test_source_without_a_batch(B, ortho, grad):
    g = torch.Generator().manual_seed(1)
    H, W = 7, 9
    sub = nd.Subject.from_volume(torch.rand(14, 15, 16, generator=g).cuda(), (4.0, 4.0, 4.0), convert_to_mu=False)
    rt = nd.make_rt_inv(40.0 * torch.rand(B, 3, generator=g), torch.tensor([[0.0, 200.0, 0.0]]).expand(B, 3)).cuda()
    k, s = nd.make_k_inv(400.0, 9.0, 9.0, 0.0, 0.0, H, W).cuda(), torch.tensor([400.0], device="cuda")
    src, tgt = _camera_rays(k, s, H, W, ortho, k.device, torch.float32)
    rt.requires_grad_(grad)
    want = nd.render(sub, k, rt, s, H, W, n_samples=40, src=src, tgt=tgt)
    got = nd.render(sub, k, rt, s, H, W, n_samples=40, src=src[0], tgt=tgt)
    assert torch.equal(got, want)
