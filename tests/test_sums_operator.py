"""The sums operator called by itself: its backward prepares its inputs as its
forward does (host), and gives the gradients of prepared ones (GPU)."""

import pytest
import torch

import nanodrr_gb300 as nd
from nanodrr_gb300 import _ffi, raymarch
from nanodrr_gb300.raymarch import fused_raymarch_sums, quad_volume, quad_volume_labeled
from nanodrr_gb300.renderer import _camera_affine, _ray_setup

B, N, S = 2, 5, 10


def _unprepared():
    """M, src, tgt, step: float64, expanded and strided views."""
    g = torch.Generator().manual_seed(0)
    return (torch.rand(B, 3, 4, generator=g).double(), torch.rand(B, 1, 3, generator=g).double(),
            torch.rand(1, N, 3, generator=g).expand(B, N, 3), torch.rand(N, B, generator=g).t())


def test_the_backward_launches_on_prepared_inputs(monkeypatch):
    class Library:
        def __getattr__(self, name):
            return lambda *args: 0

    monkeypatch.setattr(_ffi, "load", Library)
    monkeypatch.setattr(raymarch, "_stream_handle", lambda d: 0)
    monkeypatch.setattr(raymarch, "_check_inputs", lambda *a: None)
    seen, base = [], raymarch._base_args
    monkeypatch.setattr(raymarch, "_base_args", lambda *a: (seen.append(a[2:6]), base(*a))[1])
    given = _unprepared()
    vol, quad = torch.rand(4, 5, 6), torch.zeros(8 * 8 * 9 * 16, dtype=torch.uint8)
    raymarch._sums_bwd(torch.rand(B, 1, N), vol, quad, given[0], torch.zeros(0), *given[1:], torch.zeros(6, B, N), S,
                       N, True, 0)
    assert len(seen) == 2  # the pose's launch and the volume's
    for launch in seen:
        for t, want in zip(launch, given):
            assert t.dtype == torch.float32 and t.is_contiguous() and torch.equal(t, want.float())


def test_shapes_of_the_backward(monkeypatch):
    monkeypatch.setattr(raymarch, "_check_inputs", lambda *a: None)
    given = _unprepared()
    vol, quad = torch.rand(4, 5, 6), torch.zeros(8 * 8 * 9 * 16, dtype=torch.uint8)
    for go, sums in ((torch.rand(B, N), torch.zeros(6, B, N)), (torch.rand(B, 1, N), torch.zeros(6, N, B)),
                     (torch.rand(B, 1, N), torch.zeros(6, B, N, dtype=torch.float64))):
        with pytest.raises(ValueError, match="must be"):
            raymarch._sums_bwd(go, vol, quad, given[0], torch.zeros(0), *given[1:], sums, S, N, False, 0)


def _scene(dtype=torch.float32):
    g = torch.Generator().manual_seed(2)
    sub = nd.Subject.from_volume(torch.rand(19, 22, 20, generator=g).to(dtype).cuda(), (2.0, 2.0, 2.0),
                                 convert_to_mu=False)
    rot = torch.tensor([[10.0, 5.0, 0.0], [-20.0, 0.0, 3.0]])
    rt = nd.make_rt_inv(rot, torch.tensor([[0.0, 130.0, 2.0]]).expand(2, 3)).cuda()
    k, s = nd.make_k_inv(260.0, 4.0, 4.0, 1.0, -1.0, 12, 14).cuda(), torch.tensor([260.0], device="cuda")
    src, tgt, step = _ray_setup(k, s, 2, 12, 14, 40, False)
    M, _ = _camera_affine(sub.world_to_voxel, rt, False)
    return sub.image[0, 0].contiguous(), M, src, tgt, step, g


def _call(vol, quad, M, src, tgt, step):
    e = torch.empty(0, device="cuda")
    return fused_raymarch_sums(vol, quad, M, e, src, tgt, step, 40, 14, e.byte(), 0, e.byte(), 0, 0.0, 0)


@pytest.mark.gpu
def test_unprepared_inputs_give_the_gradients_of_prepared_ones():
    vol, M, src, tgt, step, g = _scene()
    quad = quad_volume(vol)
    go = torch.randn(2, 1, 12 * 14, generator=g).cuda()
    results = []
    strided = torch.stack([step, step], -1)[..., 0]
    for m, a, b, c in ((M, src, tgt, step), (M.double(), src.double(), tgt[:1].expand(2, -1, -1), strided)):
        m, v = m.detach().requires_grad_(True), vol.detach().requires_grad_(True)
        out, _ = _call(v, quad, m, a, b, c)
        results.append([out.detach(), *torch.autograd.grad(out, (m, v), go)])
    for a, b in zip(*results):
        # the volume's scattered sums add in no fixed order
        assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())


@pytest.mark.gpu
def test_a_labelled_quad_and_a_gradient_of_the_sums_are_refused():
    vol, M, src, tgt, step, _ = _scene(torch.bfloat16)
    with pytest.raises(ValueError, match="labelled"):
        _call(vol, quad_volume_labeled(vol, torch.zeros(vol.shape, device="cuda"), 2), M, src, tgt, step)
    _, sums = _call(vol, quad_volume(vol), M.requires_grad_(True), src, tgt, step)
    with pytest.raises(RuntimeError, match="no gradient"):
        sums.sum().backward()


@pytest.mark.gpu
def test_no_rays():
    vol, M, src, tgt, step, _ = _scene()
    M = M.requires_grad_(True)
    out, _ = _call(vol, quad_volume(vol), M, src, tgt[:, :0], step[:, :0])
    assert out.shape == (2, 1, 0)
    out.sum().backward()
    assert torch.equal(M.grad, torch.zeros_like(M))
