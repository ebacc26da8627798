"""The one-launch ray set-up and affine against the tensor expressions they
stand for: bitwise forward, gradients of shared and per-pose cameras."""

import pytest
import torch

import nanodrr_gb300 as nd
from nanodrr_gb300.renderer import (
    _affine_product,
    _camera_affine_op,
    _make_src,
    _make_tgt,
    _ray_setup_op,
    _ray_setup_takes,
)

pytestmark = pytest.mark.gpu


def _camera(n_k, n_s, H, W, seed):
    g = torch.Generator().manual_seed(seed)
    k = nd.make_k_inv(1000.0, 1.3, 1.1, 3.0, -2.0, H, W) * (1 + 0.02 * torch.rand(n_k, 3, 3, generator=g))
    s = 900.0 + 200.0 * torch.rand(n_s, generator=g)
    return k.cuda().requires_grad_(True), s.cuda().requires_grad_(True), g


@pytest.mark.parametrize("n_k,n_s", [(1, 1), (3, 1), (1, 3), (3, 3)])
@pytest.mark.parametrize("H,W,S", [(1, 1, 2), (1, 2, 3), (3, 5, 383), (47, 61, 500)])
@pytest.mark.parametrize("ortho", [False, True])
def test_ray_setup_is_the_tensor_expression(n_k, n_s, H, W, S, ortho):
    k, s, g = _camera(n_k, n_s, H, W, 7 * H + n_k)
    B = 3
    rt = torch.eye(4, device="cuda").expand(B, 4, 4)
    assert _ray_setup_takes(k, s, H, W, rt)
    got = _ray_setup_op(k, s, B, H, W, S, ortho)
    tgt = _make_tgt(k, s, H, W, k.device, torch.float32)
    src = _make_src(ortho, tgt, s)
    step = (tgt - src).norm(dim=-1) / float(S - 1)
    want = (src.expand(B, -1, -1), tgt.expand(B, -1, -1), step.expand(B, -1))
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    ups = [torch.randn(t.shape, generator=g).cuda() for t in want]
    if not ortho:  # a pinhole's source does not depend on the camera
        ups[0].zero_()
    grads = [torch.autograd.grad([t for t in out if t.requires_grad], (k, s),
                                 [u for t, u in zip(out, ups) if t.requires_grad], retain_graph=True)
             for out in (got, want)]
    # both sum a few thousand float32 terms of either sign: relative to the
    # sum of their magnitudes (float64), 1e-6
    mag = torch.autograd.grad([t.abs() for t in want[1:]], (k, s), [u.abs() for u in ups[1:]])
    for a, b, m in zip(*grads, mag):
        assert a.shape == b.shape
        assert float((a - b).abs().max()) <= 1e-5 * max(float(m.abs().max()), float(b.abs().max()))


@pytest.mark.parametrize("B", [1, 5, 33])
def test_affine_is_the_tensor_expression(B):
    g = torch.Generator().manual_seed(B)
    w2v = torch.randn(4, 4, generator=g).cuda()
    rt = torch.randn(B, 4, 4, generator=g).cuda().requires_grad_(True)
    M, M_lo = _camera_affine_op(w2v, rt)
    ref = _affine_product(w2v[:3], rt)
    assert torch.equal(M, ref)
    ref64 = _affine_product(w2v.double()[:3], rt.detach().double())
    assert torch.equal(M_lo, (ref64 - ref.detach().double()).float())
    go = torch.randn(M.shape, generator=g).cuda()
    (a,) = torch.autograd.grad(M, rt, go)
    (b,) = torch.autograd.grad(ref, rt, go)
    assert torch.equal(a, b)


def test_render_takes_the_same_rays_for_every_camera_type():
    """Float64 cameras and poses keep the tensor expressions; a camera shared
    by the poses and one per pose give the same image."""
    g = torch.Generator().manual_seed(0)
    sub = nd.Subject.from_volume(torch.rand(20, 24, 28, generator=g).cuda(), (2.0, 2.0, 2.0), convert_to_mu=False)
    k = nd.make_k_inv(400.0, 4.0, 4.0, 0.0, 0.0, 24, 24).cuda()
    s = torch.tensor([400.0], device="cuda")
    rt = nd.make_rt_inv(torch.zeros(2, 3), torch.tensor([[0.0, 200.0, 0.0], [5.0, 210.0, 3.0]])).cuda()
    a = nd.render(sub, k, rt, s, 24, 24, n_samples=50)
    b = nd.render(sub, k.expand(2, 3, 3).contiguous(), rt, s.expand(2).contiguous(), 24, 24, n_samples=50)
    assert torch.equal(a, b)
    kg = k.clone().requires_grad_(True)
    assert torch.equal(nd.render(sub, kg, rt, s, 24, 24, n_samples=50), a)
    c = nd.render(sub, k.double(), rt.double(), s.double(), 24, 24, n_samples=50)
    assert float((c - a).abs().max()) <= 1e-4 * float(a.abs().max())
