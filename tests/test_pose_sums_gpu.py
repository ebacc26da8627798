"""The forward that leaves the pose sums, and the positions-only volume gradient,
against the marching adjoint at their tile shapes, types and windows."""

import pytest
import torch

import nanodrr_gb300 as nd
import nanodrr_gb300.renderer as renderer
from nanodrr_gb300.empty_space import EmptySpace
from nanodrr_gb300.raymarch import quad_volume, raymarch_backward, volume_gradient
from nanodrr_gb300.renderer import _camera_affine, _ray_setup

pytestmark = pytest.mark.gpu


def _scene(shape=(33, 40, 37), dtype=torch.float32, B=2, seed=0):
    g = torch.Generator().manual_seed(seed)
    v = torch.rand(shape, generator=g)
    v[:, :9] = 0.0  # air, for the skip
    sub = nd.Subject.from_volume(v.to(dtype).cuda(), (1.5, 1.3, 1.7), convert_to_mu=False)
    rot = (torch.rand(B, 3, generator=g) - 0.5) * 50.0
    rt = nd.make_rt_inv(rot, torch.tensor([[2.0, 150.0, -3.0]]).expand(B, 3)).cuda()
    return sub, rt, g


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("H,W", [(1, 1), (7, 13), (48, 50)])
@pytest.mark.parametrize("skip", [False, True])
@pytest.mark.parametrize("with_volume", [False, True])
def test_sums_equal_the_marching_adjoint(monkeypatch, dtype, H, W, skip, with_volume):
    sub, rt, g = _scene(dtype=dtype, seed=H)
    if skip:
        sub.empty_space = EmptySpace.occupancy(sub.image[0, 0], cell=3)
    k = nd.make_k_inv(300.0, 120.0 / W, 120.0 / H, 1.0, -1.0, H, W).cuda()
    s = torch.tensor([300.0], device="cuda")
    go = torch.randn(2, 1, H, W, generator=g).to(dtype).cuda()
    got = []
    for limit in (1, 1 << 30):
        monkeypatch.setattr(renderer, "_SUMS_RAYS", limit)
        r = rt.clone().requires_grad_(True)
        sub._image_hu = sub._image_hu.detach().clone().requires_grad_(with_volume)
        img = nd.render(sub, k, r, s, H, W, n_samples=101)
        img.backward(go)
        got.append((img.detach(), r.grad, sub._image_hu.grad))
    (ia, ga, va), (ib, gb, vb) = got
    eps = {torch.float32: 1e-5, torch.float16: 2e-3, torch.bfloat16: 1e-2}[dtype]  # the stored type's rounding
    assert float((ia.double() - ib.double()).abs().max()) <= eps * float(ib.abs().max().clamp(min=1e-3))
    # the same terms in another order: 1e-5 of the gradient's scale
    assert float((ga - gb).abs().max()) <= 1e-4 * float(gb.abs().max().clamp(min=1e-6))
    if with_volume:
        assert float((va.double() - vb.double()).abs().max()) <= eps * float(vb.abs().max().clamp(min=1e-6))


def test_a_render_without_a_backward_or_with_camera_gradients_keeps_its_path(monkeypatch):
    monkeypatch.setattr(renderer, "_SUMS_RAYS", 1)
    sub, rt, _ = _scene()
    k = nd.make_k_inv(300.0, 5.0, 5.0, 0.0, 0.0, 24, 24).cuda().requires_grad_(True)
    s = torch.tensor([300.0], device="cuda")
    r = rt.clone().requires_grad_(True)
    nd.render(sub, k, r, s, 24, 24, n_samples=50).sum().backward()
    assert float(k.grad.abs().max()) > 0 and float(r.grad.abs().max()) > 0
    with torch.no_grad():
        a = nd.render(sub, k, rt, s, 24, 24, n_samples=50)
    sub2, _, _ = _scene()
    torch.use_deterministic_algorithms(True)
    try:
        sub2._image_hu.requires_grad_(True)
        img = nd.render(sub2, k.detach(), r, s, 24, 24, n_samples=50)
        with pytest.raises(RuntimeError, match="nondeterministic"):
            img.sum().backward()
    finally:
        torch.use_deterministic_algorithms(False)
    assert float((img.detach() - a).abs().max()) <= 1e-5 * float(a.abs().max())


@pytest.mark.parametrize("H,W,B", [(5, 3, 1), (96, 100, 7), (257, 260, 1), (1024, 1030, 1)])
def test_volume_gradient_alone(H, W, B):
    """One ray per thread (8 x 4 tiles of small launches), columns of two and of
    four, against the scatter of the marching adjoint."""
    sub, rt, g = _scene(B=B, seed=W)
    vol = sub.image[0, 0].contiguous()
    k = nd.make_k_inv(300.0, 130.0 / W, 130.0 / H, 0.0, 0.0, H, W).cuda()
    S = 40
    src, tgt, step = _ray_setup(k, torch.tensor([300.0], device="cuda"), B, H, W, S, False)
    M, M_lo = _camera_affine(sub.world_to_voxel, rt, True)
    go = torch.randn(B, 1, H * W, generator=g).cuda()
    go[..., ::7] = 0.0
    quad = quad_volume(vol)
    ref = raymarch_backward(go, vol, vol, M, src, tgt, step, S, 1, W, True, False, gvol_mode=1, M_lo=M_lo)[0]
    for slab_mib in (0, 1):
        a = volume_gradient(go, vol, quad, M, src, tgt, step, S, W, M_lo, slab_mib)
        assert float((a - ref).abs().max()) <= 1e-5 * float(ref.abs().max())
