"""The march's inside test at the box's faces: rays on, just inside and just
outside each face, one- and two-sample rays, and a volume whose axis exceeds
the range of the fast floor, against the float64 restatement."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from nanodrr_gb300.raymarch import quad_volume, raymarch_backward, raymarch_forward
from oracle.numpy_oracle import march_numpy, march_numpy_adjoint

pytestmark = pytest.mark.gpu

SHAPE = (7, 9, 11)  # D, H, W


def _edge_rays(axis, offsets):
    """Rays along each other axis, both ways, at `offsets` from both faces of
    `axis`, running past the box at both ends (identity affine)."""
    dims = np.array(SHAPE[::-1], dtype=np.float64)
    src, tgt = [], []
    for run in range(3):
        if run == axis:
            continue
        for face in (0.0, dims[axis] - 1.0):
            for o in offsets:
                for flip in (False, True):
                    a = dims * 0.5 + 0.137
                    b = a.copy()
                    a[axis] = b[axis] = face + o
                    a[run], b[run] = -3.3, dims[run] + 2.7
                    src.append(b if flip else a)
                    tgt.append(a if flip else b)
    f = lambda v: torch.tensor(np.array(v), dtype=torch.float32, device="cuda")[None].contiguous()  # noqa: E731
    return f(src), f(tgt)


def _identity(B=1):
    return torch.eye(4, device="cuda")[:3][None].repeat(B, 1, 1).contiguous()


@pytest.mark.parametrize("layout", ["plain", "quad"])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("S", [2, 3, 64])
def test_faces(axis, S, layout):
    g = torch.Generator().manual_seed(axis)
    vol = (torch.rand(SHAPE, generator=g) + 0.5).cuda()
    M = _identity()
    step = lambda s, t: ((t - s).norm(dim=-1) / (S - 1)).contiguous()  # noqa: E731
    quad = quad_volume(vol) if layout == "quad" else None
    # on the faces too: the image is continuous there
    src, tgt = _edge_rays(axis, (-1.25, -1.0, -0.999, -0.5, 0.0, 0.25, 0.999, 1.0, 1.001))
    out, _ = raymarch_forward(vol, vol, M, src, tgt, step(src, tgt), S, 1, 0, quad=quad)
    ref = march_numpy(vol.cpu(), None, M.cpu(), src.cpu(), tgt.cpu(), step(src, tgt).cpu(), S)
    # float32 positions up to 13 voxels: 1e-6 voxel each, values up to 1.5
    assert np.abs(out.double().cpu().numpy() - ref).max() <= 1e-5 * max(1.0, np.abs(ref).max())
    # off the faces: the gradient jumps on them
    src, tgt = _edge_rays(axis, (-1.25, -0.97, -0.53, 0.21, 0.47, 0.93, 1.31))
    go = torch.randn(1, 1, src.shape[1], generator=g).cuda()
    got = raymarch_backward(go, vol, vol, M, src, tgt, step(src, tgt), S, 1, 0, True, layout == "plain", quad=quad)
    want = march_numpy_adjoint(go.cpu(), vol.cpu(), None, M.cpu(), src.cpu(), tgt.cpu(), step(src, tgt).cpu(), S)
    for a, b in zip(got, want):
        if a.numel():
            assert np.abs(a.double().cpu().numpy() - b).max() <= 1e-5 * max(1.0, np.abs(b).max())


def test_an_axis_of_four_million_voxels():
    W = (1 << 22) + 9
    vol = torch.zeros(1, 2, W, device="cuda")
    vol[0, :, -6:] = torch.arange(1.0, 7.0, device="cuda")
    x = float(W - 3)  # exact in float32, as the half-voxel positions around it are
    src = torch.tensor([[[x, -3.0, 0.0], [x - 0.5, -3.0, 0.0], [4.0, -3.0, 0.0]]], device="cuda")
    tgt = src + torch.tensor([0.0, 7.0, 0.0], device="cuda")
    step = torch.ones(1, 3, device="cuda")
    ref = march_numpy(vol.cpu(), None, _identity().cpu(), src.cpu(), tgt.cpu(), step.cpu(), 8)
    for quad in (None, quad_volume(vol)):
        out, _ = raymarch_forward(vol, vol, _identity(), src, tgt, step, 8, 1, 0, quad=quad)
        # eight sums of exactly representable values
        assert np.abs(out.double().cpu().numpy() - ref).max() <= 1e-5


def test_a_target_far_outside():
    """A ray whose far end lies 2^29 voxels out keeps the samples inside."""
    vol = torch.rand(SHAPE, generator=torch.Generator().manual_seed(3)).cuda()
    src = torch.tensor([[[5.2, 4.3, 3.1]]], device="cuda")
    tgt = src + torch.tensor([2.0**29, 2.0**28, -(2.0**27)], device="cuda")
    step = torch.ones(1, 1, device="cuda")
    go = torch.ones(1, 1, 1, device="cuda")
    for quad in (None, quad_volume(vol)):
        out, _ = raymarch_forward(vol, vol, _identity(), src, tgt, step, 9, 1, 0, quad=quad)
        ref = march_numpy(vol.cpu(), None, _identity().cpu(), src.cpu(), tgt.cpu(), step.cpu(), 9)
        assert np.abs(out.double().cpu().numpy() - ref).max() <= 1e-5
        gM = raymarch_backward(go, vol, vol, _identity(), src, tgt, step, 9, 1, 0, False, False, quad=quad)[1]
        want = march_numpy_adjoint(go.cpu(), vol.cpu(), None, _identity().cpu(), src.cpu(), tgt.cpu(), step.cpu(), 9)[1]
        assert np.abs(gM.double().cpu().numpy() - want).max() <= 1e-4 * np.abs(want).max()


@pytest.mark.parametrize("C", [1, 3])
@pytest.mark.parametrize("hw", [(1, 1), (3, 5), (2, 16), (5, 17), (33, 31)])
@pytest.mark.parametrize("tile", [(0, 0), (8, 4), (16, 8), (24, 4), (32, 8)])
def test_warp_patches_cover_the_detector(tile, hw, C):
    """Every ray of the volume layout's forward, for each patch width, tile
    remainder and channel count, bitwise the image of one ray a call."""
    H, W = hw
    g = torch.Generator().manual_seed(5)
    vol = (torch.rand(SHAPE, generator=g) + 0.5).cuda()
    lab = torch.randint(0, C, SHAPE, generator=g).float().cuda() if C > 1 else vol
    y, x = torch.meshgrid(torch.linspace(0.3, 8.4, H), torch.linspace(0.2, 10.6, W), indexing="ij")
    tgt = torch.stack([x, y, torch.full_like(x, 8.2)], -1).reshape(1, -1, 3).cuda()
    src = torch.tensor([5.1, 3.9, -6.0], device="cuda").expand_as(tgt).contiguous()
    step = ((tgt - src).norm(dim=-1) / 39).contiguous()
    args = (vol, lab, _identity())
    out, _ = raymarch_forward(*args, src, tgt, step, 40, C, W, tile=(*tile, 2))
    if C == 1:
        ref = march_numpy(vol.cpu(), None, _identity().cpu(), src.cpu(), tgt.cpu(), step.cpu(), 40)
        # float32 positions up to 13 voxels: 1e-6 voxel each, values up to 1.5
        assert np.abs(out.double().cpu().numpy() - ref).max() <= 1e-5 * max(1.0, np.abs(ref).max())
    for n in range(0, H * W, max(1, H * W // 16)):
        one = [t[:, n : n + 1].contiguous() for t in (src, tgt, step)]
        o, _ = raymarch_forward(*args, *one, 40, C, 1, tile=(0, 0, 2))
        assert torch.equal(o[..., 0], out[..., n])
