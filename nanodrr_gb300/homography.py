"""Intrinsics resample: `resample(img, k_inv_old, k_inv_new)`.

Same call and result as the reference's `resample` (nanodrr
src/nanodrr/camera/homography.py:6-58): each destination pixel p' maps to the
source pixel p = K_old K_new^-1 p' and is sampled bilinearly (align_corners,
zero padding). The homography, the warp and the adjoint to the image and both
inverse intrinsics run in the library (`ndrr_resample_{fwd,bwd}`);
`homography_resample` is the warp by a given homography
(`ndrr_homography_resample{,_bwd}`). Differentiable in the image and both
intrinsics. Float32 images on CUDA.
"""

from __future__ import annotations

import ctypes

import torch

from . import _ffi
from ._eager import plain_eager
from .geometry import mm_small


def _inv3(A: torch.Tensor) -> torch.Tensor:
    """Inverse of [..., 3, 3] matrices by cofactors (differentiable)."""
    a, b, c = A[..., 0, 0], A[..., 0, 1], A[..., 0, 2]
    d, e, f = A[..., 1, 0], A[..., 1, 1], A[..., 1, 2]
    g, h, i = A[..., 2, 0], A[..., 2, 1], A[..., 2, 2]
    co = torch.stack([
        e * i - f * h, c * h - b * i, b * f - c * e,
        f * g - d * i, a * i - c * g, c * d - a * f,
        d * h - e * g, b * g - a * h, a * e - b * d,
    ], dim=-1).reshape(A.shape)
    det = a * co[..., 0, 0] + b * co[..., 1, 0] + c * co[..., 2, 0]
    return co / det[..., None, None]


def _stream(dev) -> int:
    return _ffi.stream_handle(dev)


def _check(img: torch.Tensor, hom: torch.Tensor):
    if not img.is_cuda:
        raise RuntimeError("nanodrr_gb300 resamples on CUDA devices only (got an image on %s)" % img.device)
    if img.dim() != 4:
        raise ValueError(f"img must be [B, C, H, W], got {tuple(img.shape)}")
    if img.dtype != torch.float32:
        raise ValueError(f"img dtype {img.dtype} unsupported; the CUDA resample takes float32")
    B = img.shape[0]
    if hom.shape != (B, 3, 3):
        raise ValueError(f"homography must be [B, 3, 3] = [{B}, 3, 3], got {tuple(hom.shape)}")


@torch.library.custom_op("nanodrr_gb300::homography_resample", mutates_args=())
def homography_resample(img: torch.Tensor, hom: torch.Tensor) -> torch.Tensor:
    """[B, C, H, W] warp of `img` by the destination -> source homography."""
    _check(img, hom)
    img = img.contiguous()
    hom = hom.float().contiguous()
    B, C, H, W = img.shape
    out = torch.empty_like(img)
    lib = _ffi.load()
    _ffi.check(lib.ndrr_homography_resample(img.data_ptr(), hom.data_ptr(), B, C, H, W, out.data_ptr(),
                                            _stream(img.device)), "ndrr_homography_resample")
    return out


@homography_resample.register_fake
def _(img, hom):
    return torch.empty_like(img)


@torch.library.custom_op("nanodrr_gb300::homography_resample_bwd", mutates_args=())
def homography_resample_bwd(go: torch.Tensor, img: torch.Tensor, hom: torch.Tensor, need_gimg: bool,
                            need_ghom: bool) -> tuple[torch.Tensor, torch.Tensor]:
    img = img.contiguous()
    hom = hom.float().contiguous()
    go = go.float().contiguous()
    B, C, H, W = img.shape
    gimg = torch.zeros_like(img) if need_gimg else img.new_empty(0)
    ghom = torch.empty(B, 3, 3, device=img.device, dtype=torch.float32) if need_ghom else img.new_empty(0)
    lib = _ffi.load()
    nb = ctypes.c_uint64(0)
    _ffi.check(lib.ndrr_homography_resample_bwd_workspace_bytes(B, H, W, ctypes.byref(nb)), "workspace")
    ws = torch.empty(max(int(nb.value), 16), device=img.device, dtype=torch.uint8)
    _ffi.check(lib.ndrr_homography_resample_bwd(
        go.data_ptr(), img.data_ptr(), hom.data_ptr(), B, C, H, W,
        gimg.data_ptr() if need_gimg else None, ghom.data_ptr() if need_ghom else None,
        ws.data_ptr(), ws.numel(), _stream(img.device)), "ndrr_homography_resample_bwd")
    return gimg, ghom


@homography_resample_bwd.register_fake
def _(go, img, hom, need_gimg, need_ghom):
    B = img.shape[0]
    return (torch.empty_like(img) if need_gimg else img.new_empty(0),
            img.new_empty(B, 3, 3) if need_ghom else img.new_empty(0))


def _setup(ctx, inputs, output):
    img, hom = inputs
    ctx.save_for_backward(img, hom)


def _backward(ctx, go):
    img, hom = ctx.saved_tensors
    need_gimg, need_ghom = ctx.needs_input_grad[0], ctx.needs_input_grad[1]
    gimg, ghom = homography_resample_bwd(go, img, hom, need_gimg, need_ghom)
    return (gimg if need_gimg else None, ghom.to(hom.dtype) if need_ghom else None)


torch.library.register_autograd("nanodrr_gb300::homography_resample", _backward, setup_context=_setup)


# ------------------------------------------------- resample from intrinsics
# The homography and its chain to the two inverse intrinsics inside the
# library's launches: the tensor expressions of both (kept for the inputs
# below that the op does not take) were 190 launches per call and adjoint,
# 2.5 ms of host time against 0.07 ms of kernels for 8 x 512^2.
@torch.library.custom_op("nanodrr_gb300::resample", mutates_args=())
def _resample_op(img: torch.Tensor, k_old: torch.Tensor, k_new: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
    """(warped images, homography [B, 3, 3]); k_old, k_new [1 or B, 3, 3]."""
    img = img.contiguous()
    a, b = k_old.float().contiguous(), k_new.float().contiguous()
    B, C, H, W = img.shape
    hom = torch.empty(B, 3, 3, device=img.device, dtype=torch.float32)
    out = torch.empty_like(img)
    _ffi.check(_ffi.load().ndrr_resample_fwd(img.data_ptr(), a.data_ptr(), a.shape[0], b.data_ptr(), b.shape[0], B, C,
                                             H, W, hom.data_ptr(), out.data_ptr(), _stream(img.device)),
               "ndrr_resample_fwd")
    return out, hom


@_resample_op.register_fake
def _(img, k_old, k_new):
    return torch.empty(img.shape, device=img.device, dtype=img.dtype), img.new_empty(img.shape[0], 3, 3)


def _resample_bwd(go: torch.Tensor, img: torch.Tensor, hom: torch.Tensor, k_old: torch.Tensor, k_new: torch.Tensor,
                  need_gimg: bool, need_gk: bool) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    img = img.contiguous()
    go = go.float().contiguous()
    a, b = k_old.float().contiguous(), k_new.float().contiguous()
    B, C, H, W = img.shape
    gimg = torch.zeros_like(img) if need_gimg else img.new_empty(0)
    g_old, g_new = (torch.empty(B if need_gk else 0, 3, 3, device=img.device, dtype=torch.float32) for _ in range(2))
    lib = _ffi.load()
    nb = ctypes.c_uint64(0)
    _ffi.check(lib.ndrr_homography_resample_bwd_workspace_bytes(B, H, W, ctypes.byref(nb)), "workspace")
    ws = torch.empty(max(int(nb.value) if need_gk else 0, 16), device=img.device, dtype=torch.uint8)
    _ffi.check(lib.ndrr_resample_bwd(
        go.data_ptr(), img.data_ptr(), hom.data_ptr(), a.data_ptr(), a.shape[0], b.data_ptr(), b.shape[0], B, C, H, W,
        gimg.data_ptr() if need_gimg else None, g_old.data_ptr() if need_gk else None,
        g_new.data_ptr() if need_gk else None, ws.data_ptr(), ws.numel(), _stream(img.device)), "ndrr_resample_bwd")
    if need_gk and B > 1:  # one camera shared by the batch: sum over it
        g_old = g_old.sum(0, keepdim=True) if a.shape[0] == 1 else g_old
        g_new = g_new.sum(0, keepdim=True) if b.shape[0] == 1 else g_new
    return gimg, g_old, g_new


_resample_bwd_op = torch.library.custom_op("nanodrr_gb300::resample_bwd", mutates_args=())(_resample_bwd)


@_resample_bwd_op.register_fake
def _(go, img, hom, k_old, k_new, need_gimg, need_gk):
    f = lambda t, on: t.new_empty(t.shape if on else (0,) + t.shape[1:], dtype=torch.float32)  # noqa: E731
    gimg = torch.empty(img.shape, device=img.device, dtype=torch.float32) if need_gimg else img.new_empty(0)
    return gimg, f(k_old, need_gk), f(k_new, need_gk)


def _resample_setup(ctx, inputs, output):
    ctx.save_for_backward(*inputs, output[1])


def _resample_backward(ctx, go, _g_hom):
    img, k_old, k_new, hom = ctx.saved_tensors
    need_gimg, need_old, need_new = ctx.needs_input_grad
    bwd = _resample_bwd if plain_eager(go, img, hom, k_old, k_new) else _resample_bwd_op
    gimg, g_old, g_new = bwd(go, img, hom, k_old, k_new, need_gimg, need_old or need_new)
    return (gimg if need_gimg else None, g_old.to(k_old.dtype) if need_old else None,
            g_new.to(k_new.dtype) if need_new else None)


torch.library.register_autograd("nanodrr_gb300::resample", _resample_backward, setup_context=_resample_setup)


def _resample_takes(img: torch.Tensor, *cameras: torch.Tensor) -> bool:
    """Float32 CUDA images with float cameras [1 or B, 3, 3] on their device;
    other inputs (and the ones that raise) go through the tensor expression."""
    return img.is_cuda and img.dim() == 4 and img.shape[0] > 0 and img.dtype == torch.float32 and all(
        k.device == img.device and k.is_floating_point() and k.dim() == 3 and tuple(k.shape[1:]) == (3, 3)
        and k.shape[0] in (1, img.shape[0]) for k in cameras)


def resample(img: torch.Tensor, k_inv_old: torch.Tensor, k_inv_new: torch.Tensor) -> torch.Tensor:
    """Resample images from one camera's inverse intrinsics to another's
    (reference homography.py:6-58): H = K_old K_new^-1 = inv(k_inv_old) @
    k_inv_new, applied to destination pixel coordinates."""
    if _resample_takes(img, k_inv_old, k_inv_new):
        return _resample_op(img, k_inv_old, k_inv_new)[0]
    hom = mm_small(_inv3(k_inv_old.float()), k_inv_new.float())
    if hom.shape[0] != img.shape[0]:
        hom = hom.expand(img.shape[0], 3, 3)
    return homography_resample(img, hom.contiguous())
