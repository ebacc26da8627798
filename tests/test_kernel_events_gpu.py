"""The kernel timing hook brackets the march kernel of every march entry
point, on its stream, within the call."""

import ctypes

import pytest
import torch

import nanodrr_gb300 as nd
from nanodrr_gb300 import _ffi
from nanodrr_gb300.raymarch import fused_raymarch_sums, quad_volume, raymarch_backward, raymarch_forward, volume_gradient
from nanodrr_gb300.renderer import _camera_affine, _ray_setup

pytestmark = pytest.mark.gpu
H, W, S = 64, 66, 120


def _calls():
    g = torch.Generator().manual_seed(0)
    sub = nd.Subject.from_volume(torch.rand(40, 44, 48, generator=g).cuda(), (2.0, 2.0, 2.0), convert_to_mu=False)
    rt = nd.make_rt_inv(torch.zeros(1, 3), torch.tensor([[0.0, 150.0, 0.0]])).cuda()
    k, s = nd.make_k_inv(300.0, 2.5, 2.5, 0.0, 0.0, H, W).cuda(), torch.tensor([300.0], device="cuda")
    rays = _ray_setup(k, s, 1, H, W, S, False)
    M, lo = _camera_affine(sub.world_to_voxel, rt, True)
    vol = sub.image[0, 0].contiguous()
    quad, go, e = quad_volume(vol), torch.ones(1, 1, H * W, device="cuda"), torch.empty(0, device="cuda").byte()
    return {
        "forward": lambda: raymarch_forward(vol, vol, M, *rays, S, 1, W, quad=quad),
        "forward_sums": lambda: fused_raymarch_sums(vol, quad, M, lo, *rays, S, W, e, 0, e, 0, 0.0, 0),
        "adjoint": lambda: raymarch_backward(go, vol, vol, M, *rays, S, 1, W, False, False, quad=quad, M_lo=lo),
        "slab_adjoint": lambda: raymarch_backward(go, vol, vol, M, *rays, S, 1, W, True, False, quad=quad, M_lo=lo),
        "volume_gradient": lambda: volume_gradient(go, vol, quad, M, *rays, S, W, lo),
    }


@pytest.mark.parametrize("name", ["forward", "forward_sums", "adjoint", "slab_adjoint", "volume_gradient"])
def test_the_march_is_bracketed(name):
    call, lib = _calls()[name], _ffi.load()
    call()
    start, stop, before, after = (torch.cuda.Event(enable_timing=True) for _ in range(4))
    start.record()
    stop.record()  # creates both
    torch.cuda.synchronize()
    before.record()
    _ffi.check(lib.ndrr_set_kernel_events(ctypes.c_void_p(start.cuda_event), ctypes.c_void_p(stop.cuda_event)), "set")
    try:
        call()
    finally:
        lib.ndrr_set_kernel_events(None, None)
    after.record()
    torch.cuda.synchronize()
    assert before.elapsed_time(start) >= 0 and start.elapsed_time(stop) > 0 and stop.elapsed_time(after) >= 0
