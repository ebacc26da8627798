"""torch's default dtype does not reach the buffers the kernels write: sizes
and types of every one on the host (a half-size buffer would be written past
its end), and on the GPU the same results under a float64 default."""

import ctypes

import pytest
import torch

import nanodrr_gb300 as nd
from nanodrr_gb300 import _ffi, homography, raymarch, registration, renderer
from nanodrr_gb300.empty_space import EmptySpace, ProposalNetwork


class _Library:
    """Accepts every call (a query of a workspace leaves its size at 0)."""

    def __getattr__(self, name):
        return lambda *args: 0


@pytest.fixture
def default_dtype():
    old = torch.get_default_dtype()
    yield torch.set_default_dtype
    torch.set_default_dtype(old)


def _calls():
    k, s, rt = torch.eye(3)[None], torch.ones(1), torch.eye(4).expand(2, 4, 4).contiguous()
    img, vol, x = torch.rand(2, 1, 5, 6), torch.rand(4, 5, 6), torch.rand(2, 3)
    go = torch.rand(2)
    quad = torch.zeros(8 * 8 * 9 * 16, dtype=torch.uint8)
    M, tgt, step = torch.rand(2, 3, 4), torch.rand(2, 6, 3), torch.rand(2, 6)
    src, empty = torch.zeros(2, 1, 3), torch.zeros(0)
    k2, maps = k.expand(2, 3, 3).contiguous(), torch.zeros(2, 1, 5, 3, 4, dtype=torch.float64)
    stats, s2, sums = torch.zeros(2, 1, 8), torch.ones(2), torch.zeros(6, 2, 6)
    net = lambda: ProposalNetwork("cpu")  # noqa: E731
    return {
        "ray_setup": lambda: renderer._ray_setup(k, s, 2, 5, 6, 10, True),
        "ray_setup_bwd": lambda: renderer._ray_setup_bwd(None, None, None, k2, s2, 2, 5, 6, 10, False),
        "camera_affine": lambda: renderer._camera_affine(torch.eye(4), rt, True),
        "camera_affine_bwd": lambda: renderer._camera_affine_bwd(torch.rand(2, 3, 4), torch.eye(4)),
        "resample": lambda: homography._resample_op(img, k2, k),
        "resample_bwd": lambda: homography._resample_bwd(img, img, k2, k2, k2, True, True),
        "homography_bwd": lambda: homography.homography_resample_bwd(img, img, k2, True, True),
        "so3_pose": lambda: registration._so3_pose_op(x, x, rt, rt, rt),
        "so3_pose_bwd": lambda: registration._so3_pose_bwd(rt, x, x, rt, rt, rt),
        "ncc": lambda: registration._ncc_op(img, img, 1e-7),
        "ncc_bwd": lambda: registration._ncc_bwd(go, img, img, stats, True, True),
        "ncc_patch": lambda: registration._ncc_patch_op(img, img, 3, 1e-7)[:1],
        "ncc_patch_bwd": lambda: registration._ncc_patch_bwd(go, img, img, maps, 3, True, True),
        "volume_gradient": lambda: raymarch.volume_gradient(torch.rand(2, 1, 6), vol, quad, M, src, tgt, step, 10, 6),
        "march_bwd": lambda: raymarch.raymarch_backward(torch.rand(2, 1, 6), vol, vol, M, src, tgt, step, 10, 1, 6,
                                                        True, True),
        "sums_bwd": lambda: raymarch._sums_bwd(torch.rand(2, 1, 6), vol, quad, M, empty, src, tgt, step, sums, 10, 6,
                                               False, 0),
        "proposal": lambda: (net().params, net().forward(torch.rand(3, 64)),
                             net().train_step(torch.rand(3, 64), x, torch.zeros(3, dtype=torch.uint8))),
        "proposal_data": lambda: ProposalNetwork.dataset(vol, M, src, tgt, 10, 6, torch.rand(2, 6, 2))[:2],
    }


@pytest.mark.parametrize("dtype", [torch.float64, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("name", sorted(_calls()))
def test_buffers_do_not_follow_it(monkeypatch, default_dtype, name, dtype):
    monkeypatch.setattr(_ffi, "load", lambda *a: _Library())
    monkeypatch.setattr(_ffi, "check", lambda *a: None)
    for m in (_ffi, raymarch):
        monkeypatch.setattr(m, "stream_handle" if m is _ffi else "_stream_handle", lambda d: 0)
    monkeypatch.setattr("nanodrr_gb300.empty_space._stream", lambda d: 0)
    monkeypatch.setattr(raymarch, "_check_inputs", lambda *a: None)
    monkeypatch.setattr(registration, "_ncc_check", lambda *a: None)
    monkeypatch.setattr(ctypes, "c_uint64", lambda v=0: _U64(64))
    call, made = _calls()[name], []
    for f in ("empty", "zeros", "ones"):
        monkeypatch.setattr(torch, f, lambda *a, _f=getattr(torch, f), **kw: made.append(_f(*a, **kw)) or made[-1])
    want, buffers = call(), [(t.shape, t.dtype) for t in made]
    made.clear()
    default_dtype(dtype)
    got = call()
    assert [(t.shape, t.dtype) for t in made] == buffers
    assert [(t.shape, t.dtype) for t in _flat(got)] == [(t.shape, t.dtype) for t in _flat(want)]


_U64 = ctypes.c_uint64


def _flat(out):
    return [out] if isinstance(out, torch.Tensor) else list(out)


@pytest.mark.gpu
def test_results_under_a_float64_default(default_dtype):
    g = torch.Generator().manual_seed(3)
    H, W = 21, 26
    v = torch.rand(23, 26, 29, generator=g)
    v[:, :6] = 0.0
    img = torch.rand(2, 1, 40, 44, generator=g)
    rot, xyz = torch.tensor([[10.0, 5.0, 0.0], [-20.0, 0.0, 3.0]]), torch.tensor([[0.0, 130.0, 2.0]]).expand(2, 3)
    rt0 = nd.make_rt_inv(rot, xyz)
    k0, s0 = nd.make_k_inv(260.0, 3.0, 3.0, 1.0, -1.0, H, W), torch.tensor([260.0])
    iso, params = torch.zeros(3), 0.01 * torch.rand(2, 2, 3, generator=g)

    def results():
        leaf = lambda t: t.clone().cuda().requires_grad_(True)  # noqa: E731
        out = []
        for ortho in (False, True):
            sub = nd.Subject.from_volume(v.cuda(), (1.5, 1.5, 1.5), convert_to_mu=False)
            k, s, rt = leaf(k0), leaf(s0), leaf(rt0)
            im = nd.render(sub, k, rt, s, H, W, n_samples=60, orthographic=ortho)
            out += [im, *torch.autograd.grad(im.square().sum(), (k, s, rt))]
            sub.empty_space = EmptySpace.occupancy(sub.image[0, 0], cell=3)
            out.append(nd.render(sub, k0.cuda(), rt0.cuda(), s0.cuda(), H, W, n_samples=60, orthographic=ortho))
        a, b = leaf(img), leaf(img.flip(0))
        for patch in (None, 5):
            score = registration.NormalizedCrossCorrelation2d(patch_size=patch, eps=1e-5)(a, b)
            out += [score, *torch.autograd.grad(score.sum(), (a, b))]
        k1 = leaf(k0 * 1.05)
        im = nd.resample(a, k, k1)
        out += [im, *torch.autograd.grad(im.square().sum(), (a, k, k1))]
        sub.isocenter = iso.cuda()
        reg = registration.Registration(sub, rt0.cuda(), k0.cuda(), s0.cuda(), H, W, batch=2)
        with torch.no_grad():
            reg._rot.copy_(params[0])
            reg._xyz.copy_(params[1])
        out += [reg.pose, *torch.autograd.grad(reg.pose.square().sum(), list(reg.parameters()))]
        return [t.detach() for t in out]

    want = results()
    default_dtype(torch.float64)
    for i, (a, b) in enumerate(zip(results(), want)):
        # the image gradient of the resample adds in no fixed order
        assert float((a.double() - b.double()).abs().max()) <= 1e-5 * float(b.abs().max()), i
