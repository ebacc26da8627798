"""The source's gradient where the volume is near the detector: 1 - t is small
there, and the sum over (1 - t) must not be formed as a difference of sums."""

import numpy as np
import pytest
import torch

from nanodrr_gb300.raymarch import quad_volume, raymarch_backward
from oracle.numpy_oracle import march_numpy_adjoint

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_ray", [False, True])
@pytest.mark.parametrize("layout", ["quad", "plain"])
def test_source_gradient_near_the_detector(per_ray, layout):
    """A ramp, so that every sample's term has one sign; 4000 samples, some 900
    in the volume at t of 0.75 to 0.98. A running float32 sum of 900 like terms
    is off by about 6e-7 (root mean square, numpy); a difference of two such
    sums by 5e-5 of the small remainder. Five times the first."""
    H, W, S, n = 8, 12, 4000, 20
    x = torch.arange(n, dtype=torch.float32)
    vol = (x[None, None, :] + 0.5 * x[None, :, None] + 0.25 * x[:, None, None] + 1.0).contiguous()
    u, v = torch.meshgrid(torch.arange(W) - 5.3, torch.arange(H) - 3.6, indexing="xy")
    tgt = torch.stack([0.8 * u, 0.9 * v, torch.full_like(u, 92.0)], -1).reshape(1, -1, 3).float()
    src = torch.tensor([[[0.3, -0.2, 0.1]]])
    if per_ray:
        src = src + 0.2 * torch.rand(1, H * W, 3, generator=torch.Generator().manual_seed(1))
    a = 0.1  # the rays run along the volume's z, tilted
    M = torch.tensor([[[np.cos(a), 0.0, -np.sin(a), 18.1], [0.0, 1.0, 0.0, 9.7], [np.sin(a), 0.0, np.cos(a), -70.2]]])
    M = M.float()
    step = (tgt - src).norm(dim=-1) / (S - 1)
    go = torch.rand(1, 1, H * W, generator=torch.Generator().manual_seed(2)) + 0.5
    want = march_numpy_adjoint(go.numpy(), vol.numpy(), None, M.numpy(), src.numpy(), tgt.numpy(), step.numpy(), S)[2]
    d = [t.cuda() for t in (go, vol, vol, M, src, tgt, step)]
    quad = quad_volume(d[1]) if layout == "quad" else None
    got = raymarch_backward(*d, S, 1, W, False, True, tile=(8, 4, 1), quad=quad)[2].cpu().double()
    want = torch.from_numpy(want)
    assert float(want.norm(dim=-1).min()) > 0
    rel = (got - want).norm(dim=-1) / want.norm(dim=-1)
    assert float(rel.square().mean().sqrt()) <= 3e-6
