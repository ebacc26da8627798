"""Volume preparation kernels at the edges of their tiles: HU conversion of odd
lengths and unaligned views, quad copies around the row groups, occupancy and
distance grids of every kind of cell against their definitions."""

import numpy as np
import pytest
import torch

import nanodrr_gb300 as nd
from nanodrr_gb300.empty_space import OccupancyGrid
from nanodrr_gb300.raymarch import quad_volume, quad_volume_labeled
from oracle import empty_space_oracle as eso

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("n,offset", [(1, 0), (3, 0), (8, 0), (1025, 0), (1025, 1), (4096, 3)])
def test_hu_to_mu_lengths_and_alignments(dtype, n, offset):
    g = torch.Generator().manual_seed(n)
    x = (torch.rand(n + offset, generator=g) * 4000 - 1500).to(dtype)
    x[offset] = float("nan") if n > 8 else -1000.0
    got = nd.hu_to_mu(x.cuda()[offset:]).cpu()
    h = x[offset:].double().clamp(min=-1000.0)
    ref = torch.where(h > 0, 0.0192 + h / 1000.0 * (0.0573 - 0.0192), (h / 1000.0 + 1) * 0.0192).clamp(min=0.0)
    # four float32 roundings of values below 0.3, then the storage type's own
    tol = {torch.float32: 1e-7, torch.float16: 1e-4, torch.bfloat16: 1e-3}[dtype]
    assert torch.equal(got.isnan(), ref.isnan())
    assert float((got.double() - ref).nan_to_num().abs().max()) <= tol


def _corner(v, D, H, W):
    """[D + 4, H + 3, W + 3, 4] quads of a volume by padding and shifting."""
    p = np.zeros((D + 4, H + 5, W + 5), v.dtype)
    p[2:D + 2, 2:H + 2, 2:W + 2] = v
    return np.stack([p[:, y:y + H + 3, x:x + W + 3] for y in (0, 1) for x in (0, 1)], -1)


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 13, 5), (2, 14, 126), (4, 29, 131), (2, 45, 257)])
def test_quad_copies(shape):
    g = torch.Generator().manual_seed(shape[1])
    v = torch.rand(shape, generator=g)
    q = quad_volume(v.cuda()).cpu().numpy().view(np.float32).reshape(*(s + d for s, d in zip(shape, (4, 3, 3))), 4)
    assert np.array_equal(q, _corner(v.numpy(), *shape))
    h = v.half()
    raw = h.view(torch.int16).numpy()
    q = quad_volume(h.cuda()).cpu().numpy().view(np.int16).reshape(*(s + d for s, d in zip(shape, (4, 3, 3))), 4)
    assert np.array_equal(q, _corner(raw, *shape))
    lab = torch.randint(-1, 5, shape, generator=g, dtype=torch.int16)
    q = quad_volume_labeled(h.cuda(), lab.cuda(), 4).cpu().numpy().reshape(*(s + d for s, d in zip(shape, (4, 3, 3))), 16)
    cls = lab.numpy().copy()
    cls[(cls < 0) | (cls >= 4)] = 255
    assert np.array_equal(np.ascontiguousarray(q[..., :8]).view(np.int16), _corner(raw, *shape))
    assert np.array_equal(q[..., 8:12], _corner(cls.astype(np.uint8), *shape))
    assert not q[..., 12:].any()


@pytest.mark.parametrize("cell,max_dist", [(2, 3), (3, 255), (4, 16), (7, 5), (64, 1)])
@pytest.mark.parametrize("shape", [(1, 1, 1), (9, 70, 33), (21, 66, 40), (5, 6, 1100)])
def test_occupancy_and_distance(shape, cell, max_dist):
    rng = np.random.default_rng(cell)
    for density in (0.0, 1e-3, 0.05):
        v = np.where(rng.random(shape) < density, 1.0, 0.0).astype(np.float32)
        v[-1, -1, -1] = 1.0 if density == 1e-3 else 0.0
        got = OccupancyGrid.build(torch.from_numpy(v).cuda(), cell=cell, max_dist=max_dist).grid.cpu().numpy()
        assert np.array_equal(got, _grid(v, cell, max_dist, got.shape))


def _grid(v, cell, max_dist, shape):
    """A cap no distance reaches: the oracle relaxes once per unit of the cap,
    so cells it leaves at a cap just past the grid get the real one."""
    near = max(shape) + 1
    if max_dist <= near:
        return eso.occupancy_grid(v, cell, max_dist)
    d = eso.occupancy_grid(v, cell, near).astype(np.int64)
    return np.where(d == near, max_dist, d).astype(np.uint8)


@pytest.mark.parametrize("cell", [5, 8, 9, 16, 17, 33])
@pytest.mark.parametrize("shape", [(13, 35, 40), (37, 18, 131)])
def test_occupancy_around_the_tile_height(shape, cell):
    """Cells that tile the CTA's lines with a remainder, fill them and exceed them."""
    rng = np.random.default_rng(cell + 1)
    for density in (1e-4, 1e-2):
        v = np.where(rng.random(shape) < density, 1.0, 0.0).astype(np.float32)
        got = OccupancyGrid.build(torch.from_numpy(v).cuda(), cell=cell, max_dist=4).grid.cpu().numpy()
        assert np.array_equal(got, _grid(v, cell, 4, got.shape))
