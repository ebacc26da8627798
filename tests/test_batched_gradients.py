"""Upstream gradients batched by torch.autograd.grad(is_grads_batched=True),
for every adjoint that a plain eager backward calls without its operator."""

import pytest
import torch

import nanodrr_gb300 as nd
import nanodrr_gb300.renderer as renderer
from nanodrr_gb300._eager import plain_eager
from nanodrr_gb300.registration import NormalizedCrossCorrelation2d, Registration


def test_a_batched_gradient_is_not_plain():
    x = torch.rand(3, requires_grad=True)
    seen = []

    class Square(torch.autograd.Function):
        @staticmethod
        def forward(ctx, a):
            ctx.save_for_backward(a)
            return a * a

        @staticmethod
        def backward(ctx, g):
            (a,) = ctx.saved_tensors
            seen.append(plain_eager(g, a))
            return 2 * a * g

    y = Square.apply(x)
    torch.autograd.grad(y, x, torch.eye(3), is_grads_batched=True, retain_graph=True)
    torch.autograd.grad(y.sum(), x)
    assert seen == [False, True]


def _render(sums=False):
    def f(monkeypatch, g):
        monkeypatch.setattr(renderer, "_SUMS_RAYS", 1 if sums else 1 << 30)
        sub = nd.Subject.from_volume(torch.rand(14, 15, 16, generator=g).cuda(), (4.0, 4.0, 4.0), convert_to_mu=False)
        rt = nd.make_rt_inv(torch.tensor([[20.0, 5.0, 0.0]]), torch.tensor([[0.0, 200.0, 0.0]])).cuda()
        k, s = nd.make_k_inv(400.0, 9.0, 9.0, 0.0, 0.0, 8, 9).cuda(), torch.tensor([400.0], device="cuda")
        leaves = [rt] if sums else [rt, k, s]
        for t in leaves:
            t.requires_grad_(True)
        sub._image_hu = sub._image_hu.detach().clone().requires_grad_(True)
        return nd.render(sub, k, rt, s, 8, 9, n_samples=40), [*leaves, sub._image_hu]

    return f


def _pose(monkeypatch, g):
    sub = nd.Subject.from_volume(torch.rand(6, 6, 6, generator=g).cuda(), (4.0, 4.0, 4.0), convert_to_mu=False)
    rt = nd.make_rt_inv(torch.tensor([[20.0, 5.0, 0.0]]), torch.tensor([[0.0, 200.0, 0.0]])).cuda()
    k, s = nd.make_k_inv(400.0, 9.0, 9.0, 0.0, 0.0, 8, 8).cuda(), torch.tensor([400.0], device="cuda")
    reg = Registration(sub, rt, k, s, 8, 8)
    return reg.pose, list(reg.parameters())


def _ncc(patch):
    def f(monkeypatch, g):
        a, b = (torch.rand(3, 1, 11, 12, generator=g).cuda().requires_grad_(True) for _ in range(2))
        return NormalizedCrossCorrelation2d(patch_size=patch, eps=1e-4)(a, b), [a, b]

    return f


def _resample(monkeypatch, g):
    a = torch.rand(2, 1, 9, 11, generator=g).cuda().requires_grad_(True)
    k = [nd.make_k_inv(400.0, p, p, 0.0, 0.0, 9, 11).cuda().requires_grad_(True) for p in (1.0, 1.1)]
    return nd.resample(a, *k), [a, *k]


@pytest.mark.gpu
@pytest.mark.parametrize("make", [_render(), _render(sums=True), _pose, _ncc(None), _ncc(4), _resample],
                         ids=["camera", "sums", "pose", "ncc", "ncc_patch", "resample"])
def test_batched_gradients_equal_single_ones(monkeypatch, make):
    g = torch.Generator().manual_seed(5)
    out, leaves = make(monkeypatch, g)
    ups = torch.randn(3, *out.shape, generator=g).cuda()
    got = torch.autograd.grad(out, leaves, ups, is_grads_batched=True, retain_graph=True)
    for j, up in enumerate(ups):
        for a, b in zip(got, torch.autograd.grad(out, leaves, up, retain_graph=True)):
            # the same launches; scattered sums add in no fixed order
            assert float((a[j] - b).abs().max()) <= 1e-5 * float(b.abs().max().clamp(min=1e-6))
