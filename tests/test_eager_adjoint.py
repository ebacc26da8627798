"""When an adjoint may skip its operator (host-only), and what a double
backward does on the GPU."""

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from nanodrr_gb300._eager import plain_eager


class _Mode(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


def test_plain_eager_conditions():
    t = torch.ones(3)
    assert not plain_eager(t)  # a gradient may be recorded
    with torch.no_grad():
        assert plain_eager(t, None, torch.nn.Parameter(t))
        assert not plain_eager(torch.Tensor._make_subclass(type("Sub", (torch.Tensor,), {}), t))
        with _Mode():
            assert not plain_eager(t)
        seen = []
        torch.func.vmap(lambda x: (seen.append(plain_eager(x)), x)[1])(t)
        assert seen == [False]
        with torch._subclasses.FakeTensorMode() as m:
            f = m.from_tensor(t)
            assert not plain_eager(f)
        assert not plain_eager(f)


@pytest.mark.gpu
def test_a_double_backward_is_refused():
    import nanodrr_gb300 as nd

    sub = nd.Subject.from_volume(torch.rand(12, 12, 12).cuda(), (4.0, 4.0, 4.0), convert_to_mu=False)
    k = nd.make_k_inv(400.0, 8.0, 8.0, 0.0, 0.0, 8, 8).cuda()
    s = torch.tensor([400.0], device="cuda")
    rt = nd.make_rt_inv(torch.zeros(1, 3), torch.tensor([[0.0, 200.0, 0.0]])).cuda().requires_grad_(True)
    (g,) = torch.autograd.grad(nd.render(sub, k, rt, s, 8, 8, n_samples=20).square().sum(), rt, create_graph=True)
    with pytest.raises(RuntimeError):
        torch.autograd.grad(g.square().sum(), rt)
