"""`render`: the user-facing call, a drop-in for the reference's fused backend.

Mirrors nanodrr's `render` (src/nanodrr/drr/renderer.py:21-98) and the
adapter `render_fused` (src/nanodrr/drr/backends.py:72-117): same arguments,
same ray construction (`_make_tgt`/`_make_src`, renderer.py:101-132), same
camera-space step size (renderer.py:82) and the same camera -> voxel affine
`M = (world_to_voxel @ rt_inv)[:, :3]` in float32 (backends.py:96). There is
one backend, the sm_103a CUDA kernels: `backend` accepts "auto", "cuda" and
"triton" (the reference's name for its fused backend, kept so existing calls
switch unchanged); any other value raises, and CPU tensors raise rather than
falling back to a CPU path.
"""

from __future__ import annotations

import ctypes
import weakref

import torch

from . import _ffi
from ._eager import plain_eager, plain_tensors
from .raymarch import (
    _SkipArgs,
    fused_raymarch_ex,
    fused_raymarch_sums,
    march_direct,
    quad_volume,
    quad_volume_labeled,
)
from .subject import Subject

_BACKENDS = ("auto", "cuda", "triton")

# Ray set-ups (src, tgt, step expanded to the batch) of recent render calls,
# keyed by the intrinsics and sdd tensor objects: a repeated render with the
# same camera reuses them instead of rebuilding N rays with a dozen small
# launches. An entry is valid while both tensors are alive (weak references)
# and unmodified (version counters).
_RAY_CACHE: dict = {}
_RAY_CACHE_SIZE = 4

# Rays (of all poses together) from which a one-channel render that needs a
# pose gradient takes the forward that leaves the pose sums
# (`fused_raymarch_sums`). Kernels of a pose step, with sums / with two marches,
# us, and of its forward alone (500 samples of 512 x 512 x 400, float32):
#   1 x 200^2   143 /  190   forward 126 /   95
#   4 x 128^2   174 /  419           158 /  203
#   8 x 200^2   399 /  690           380 /  321
#  32 x 120^2  1506 / 3018          1491 / 1536
#  16 x 200^2   768 / 1493           751 /  741
#   4 x 512^2   802 / 1306           781 /  528
# (250 of 128^3: 1 x 200^2 30 / 32 and 18 / 16, 16 x 200^2 79 / 104 and 63 / 46.)
# The step gains at every size measured, so the line is not where the sums start
# to pay. It keeps them out of small renders, where sums in another order would
# move the ill-conditioned rotation gradient of a single pose at the 1e-5 level,
# and where the gain is little of a step of 0.6 ms or more of host time; a batch
# of small renders below it (32 x 120^2) would gain too. A forward whose
# backward never runs pays for the sums, up to 1.6 times: evaluations of the loss
# alone belong under torch.no_grad.
_SUMS_RAYS = 1 << 19

# Camera -> voxel affines of recent calls without a gradient, keyed by the
# world_to_voxel and rt_inv tensor objects: a repeated render of the same
# pose reuses M instead of two tensor launches (~25 us of host time per call).
# Valid while both tensors are alive and unmodified, as for the ray cache.
_M_CACHE: dict = {}
_M_CACHE_SIZE = 4


def fused_supported(subject: Subject, B: int, n_pixels: int) -> bool:
    """Limits of the CUDA kernels: one volume, int32 voxel and ray indexing
    (reference backends.py:66-69)."""
    return _within_limits(subject.image, subject.n_classes, B * n_pixels)


def _within_limits(img: torch.Tensor, n_classes: int, n_rays: int) -> bool:
    return img.shape[0] == 1 and max(img.numel(), n_classes * n_rays, 3 * n_rays) < 2**31


def _make_tgt(k_inv, sdd, height, width, device, dtype) -> torch.Tensor:
    """Detector pixel centres (u + 0.5, v + 0.5, 1) mapped by sdd * K^-1."""
    N = height * width
    v, u = torch.meshgrid(
        torch.arange(height, device=device, dtype=dtype) + 0.5,
        torch.arange(width, device=device, dtype=dtype) + 0.5,
        indexing="ij",
    )
    uv1 = torch.stack([u, v, torch.ones_like(u)], dim=-1).reshape(N, 3)
    # K^-1 @ uv1 as three broadcast multiply-adds: no library GEMM for a 3x3
    # product, so the call also runs under torch's deterministic mode.
    k = k_inv[:, None]  # [B, 1, 3, 3]
    rays = k[..., 0] * uv1[None, :, 0:1] + k[..., 1] * uv1[None, :, 1:2] + k[..., 2] * uv1[None, :, 2:3]
    return sdd[:, None, None] * rays


def _make_src(orthographic: bool, tgt: torch.Tensor, sdd: torch.Tensor) -> torch.Tensor:
    """Point source at the camera origin, or parallel rays for orthographic."""
    if orthographic:
        src = tgt.clone()
        src[..., 2] -= sdd[:, None]
        return src
    B = tgt.shape[0]
    return torch.zeros(B, 1, 3, device=tgt.device, dtype=tgt.dtype)


def _camera_rays(k_inv, sdd, height, width, orthographic, device, dtype) -> tuple[torch.Tensor, torch.Tensor]:
    """(src, tgt) of the detector. Float32 CUDA cameras that need no gradient
    take one `ndrr_camera_rays` launch, which rounds every product and sum as
    `_make_tgt`/`_make_src` do, so the rays are bitwise the same; other
    cameras (a differentiable K^-1 or sdd, float64, traced calls) use the
    tensor expressions."""
    compiling = hasattr(torch, "compiler") and torch.compiler.is_compiling()
    want = torch.device(device)
    if (
        not compiling
        and dtype == torch.float32
        and k_inv.dtype == torch.float32
        and sdd.dtype == torch.float32
        and k_inv.is_cuda
        and k_inv.device == sdd.device
        and want.type == "cuda"
        and (want.index is None or want == k_inv.device)
        and k_inv.dim() == 3
        and tuple(k_inv.shape[1:]) == (3, 3)
        and sdd.dim() == 1
        and not (torch.is_grad_enabled() and (k_inv.requires_grad or sdd.requires_grad))
    ):
        n_k, n_s = k_inv.shape[0], sdd.shape[0]
        B = max(n_k, n_s)
        if n_k in (1, B) and n_s in (1, B):
            k = k_inv.detach().contiguous()
            s = sdd.detach().contiguous()
            N = height * width
            tgt = torch.empty(B, N, 3, device=k.device, dtype=torch.float32)
            src = torch.empty(B, N if orthographic else 1, 3, device=k.device, dtype=torch.float32)
            lib = _ffi.load()
            _ffi.check(
                lib.ndrr_camera_rays(k.data_ptr(), n_k, s.data_ptr(), n_s, B, height, width, int(bool(orthographic)),
                                     src.data_ptr(), tgt.data_ptr(), _ffi.stream_handle(k.device)),
                "ndrr_camera_rays",
            )
            return src, tgt
    tgt = _make_tgt(k_inv, sdd, height, width, device, dtype)
    return _make_src(orthographic, tgt, sdd), tgt


# ------------------------------------------------------------- ray set-up
# Rays and sample spacing of a call in one launch, and their adjoint to K^-1
# and sdd in two: as tensor expressions a differentiable camera was 40 launches
# per step, most of the host time of a small calibration step.
def _ray_setup_takes(k_inv, sdd, height, width, rt_inv) -> bool:
    """Float32 CUDA cameras and poses of one device, K^-1 [1 or B, 3, 3] and
    sdd [1 or B] for B poses; other inputs, and traced calls, use
    `_camera_rays` and tensor operations."""
    if hasattr(torch, "compiler") and torch.compiler.is_compiling():
        return False
    if not (rt_inv.dtype == k_inv.dtype == sdd.dtype == torch.float32):
        return False
    if not (rt_inv.is_cuda and rt_inv.device == k_inv.device == sdd.device):
        return False
    if k_inv.dim() != 3 or tuple(k_inv.shape[1:]) != (3, 3) or sdd.dim() != 1 or rt_inv.dim() != 3:
        return False
    B = max(rt_inv.shape[0], k_inv.shape[0], sdd.shape[0])
    return (min(rt_inv.shape[0], height, width) >= 1 and k_inv.shape[0] in (1, B) and sdd.shape[0] in (1, B)
            and B <= 65535 and 3 * B * height * width < 2**31)


def _ray_setup(k_inv, sdd, batch, height, width, n_samples, orthographic):
    """(src, tgt, step) of `batch` poses, expanded and contiguous."""
    k, s = k_inv.detach().contiguous(), sdd.detach().contiguous()
    N = height * width
    tgt = torch.empty(batch, N, 3, device=k.device, dtype=torch.float32)
    src = torch.empty(batch, N if orthographic else 1, 3, device=k.device, dtype=torch.float32)
    step = torch.empty(batch, N, device=k.device, dtype=torch.float32)
    _ffi.check(
        _ffi.load().ndrr_ray_setup(k.data_ptr(), k.shape[0], s.data_ptr(), s.shape[0], batch, height, width,
                                   int(orthographic), n_samples, src.data_ptr(), tgt.data_ptr(), step.data_ptr(),
                                   _ffi.stream_handle(k.device)),
        "ndrr_ray_setup",
    )
    return src, tgt, step


@torch.library.custom_op("nanodrr_gb300::ray_setup", mutates_args=())
def _ray_setup_op(k_inv: torch.Tensor, sdd: torch.Tensor, batch: int, height: int, width: int, n_samples: int,
                  orthographic: bool) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    return _ray_setup(k_inv, sdd, batch, height, width, n_samples, orthographic)


@_ray_setup_op.register_fake
def _(k_inv, sdd, batch, height, width, n_samples, orthographic):
    N = height * width
    return (k_inv.new_empty(batch, N if orthographic else 1, 3), k_inv.new_empty(batch, N, 3),
            k_inv.new_empty(batch, N))


def _ray_setup_bwd(gsrc: torch.Tensor | None, gtgt: torch.Tensor | None, gstep: torch.Tensor | None,
                   k_inv: torch.Tensor, sdd: torch.Tensor, batch: int, height: int, width: int, n_samples: int,
                   orthographic: bool) -> tuple[torch.Tensor, torch.Tensor]:
    k, s = k_inv.contiguous(), sdd.contiguous()
    grads = [None if g is None else g.float().contiguous() for g in (gsrc if orthographic else None, gtgt, gstep)]
    g_k = torch.empty(batch, 3, 3, device=k.device, dtype=torch.float32)
    g_s = torch.empty(batch, device=k.device, dtype=torch.float32)
    lib = _ffi.load()
    nb = ctypes.c_uint64(0)
    _ffi.check(lib.ndrr_ray_setup_bwd_workspace_bytes(batch, height, width, ctypes.byref(nb)), "workspace query")
    ws = torch.empty(int(nb.value), device=k.device, dtype=torch.uint8)
    _ffi.check(
        lib.ndrr_ray_setup_bwd(k.data_ptr(), k.shape[0], s.data_ptr(), s.shape[0], batch, height, width,
                               int(orthographic), n_samples, *(None if g is None else g.data_ptr() for g in grads),
                               g_k.data_ptr(), g_s.data_ptr(), ws.data_ptr(), ws.numel(),
                               _ffi.stream_handle(k.device)),
        "ndrr_ray_setup_bwd",
    )
    if batch > 1:  # one camera shared by the poses: sum over them
        g_k = g_k.sum(0, keepdim=True) if k.shape[0] == 1 else g_k
        g_s = g_s.sum(0, keepdim=True) if s.shape[0] == 1 else g_s
    return g_k, g_s


_ray_setup_bwd_op = torch.library.custom_op("nanodrr_gb300::ray_setup_bwd", mutates_args=())(_ray_setup_bwd)


@_ray_setup_bwd_op.register_fake
def _(gsrc, gtgt, gstep, k_inv, sdd, batch, height, width, n_samples, orthographic):
    return torch.empty_like(k_inv), torch.empty_like(sdd)


def _ray_setup_context(ctx, inputs, output):
    ctx.save_for_backward(inputs[0], inputs[1])
    ctx.args = inputs[2:]
    ctx.set_materialize_grads(False)


def _ray_setup_backward(ctx, gsrc, gtgt, gstep):
    k_inv, sdd = ctx.saved_tensors
    bwd = _ray_setup_bwd if plain_eager(gsrc, gtgt, gstep, k_inv, sdd) else _ray_setup_bwd_op
    g_k, g_s = bwd(gsrc, gtgt, gstep, k_inv, sdd, *ctx.args)
    return (g_k if ctx.needs_input_grad[0] else None, g_s if ctx.needs_input_grad[1] else None, *[None] * 5)


torch.library.register_autograd("nanodrr_gb300::ray_setup", _ray_setup_backward, setup_context=_ray_setup_context)


# --------------------------------------------------------- camera -> voxel
def _affine_takes(w2v: torch.Tensor, rt_inv: torch.Tensor) -> bool:
    """Float32 affine and poses on one CUDA device, the affine without a
    gradient, outside tracing and transforms (poses batched by vmap or fake
    have no pointer to launch with); others use `_affine_product`."""
    return (rt_inv.is_cuda and w2v.device == rt_inv.device and w2v.dtype == rt_inv.dtype == torch.float32
            and tuple(w2v.shape) == (4, 4) and rt_inv.dim() == 3 and rt_inv.shape[0] >= 1
            and tuple(rt_inv.shape[1:]) == (4, 4) and not w2v.requires_grad and plain_tensors(w2v, rt_inv))


def _camera_affine(w2v: torch.Tensor, rt_inv: torch.Tensor, low: bool) -> tuple[torch.Tensor, torch.Tensor]:
    w, rt = w2v.detach().contiguous(), rt_inv.detach().contiguous()
    B = rt.shape[0]
    M = torch.empty(B, 3, 4, device=rt.device, dtype=torch.float32)
    M_lo = torch.empty_like(M) if low else M.new_empty(0)
    _ffi.check(_ffi.load().ndrr_camera_affine(w.data_ptr(), rt.data_ptr(), B, M.data_ptr(),
                                              M_lo.data_ptr() if low else None,
                                              _ffi.stream_handle(rt.device)), "ndrr_camera_affine")
    return M, M_lo


@torch.library.custom_op("nanodrr_gb300::camera_affine", mutates_args=())
def _camera_affine_op(w2v: torch.Tensor, rt_inv: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
    """M = (world_to_voxel @ rt_inv)[:, :3] in float32 and its low parts."""
    return _camera_affine(w2v, rt_inv, True)


@_camera_affine_op.register_fake
def _(w2v, rt_inv):
    return rt_inv.new_empty(rt_inv.shape[0], 3, 4), rt_inv.new_empty(rt_inv.shape[0], 3, 4)


def _camera_affine_bwd(gM: torch.Tensor, w2v: torch.Tensor) -> torch.Tensor:
    g, w = gM.contiguous(), w2v.contiguous()
    out = torch.empty(g.shape[0], 4, 4, device=g.device, dtype=torch.float32)
    _ffi.check(_ffi.load().ndrr_camera_affine_bwd(w.data_ptr(), g.data_ptr(), g.shape[0], out.data_ptr(),
                                                  _ffi.stream_handle(g.device)),
               "ndrr_camera_affine_bwd")
    return out


_camera_affine_bwd_op = torch.library.custom_op("nanodrr_gb300::camera_affine_bwd",
                                                mutates_args=())(_camera_affine_bwd)


@_camera_affine_bwd_op.register_fake
def _(gM, w2v):
    return gM.new_empty(gM.shape[0], 4, 4)


def _camera_affine_context(ctx, inputs, output):
    ctx.save_for_backward(inputs[0])
    ctx.set_materialize_grads(False)


def _camera_affine_backward(ctx, gM, _g_lo):
    # M_lo is a rounding correction of M, not differentiated
    if gM is None:
        return None, None
    w2v = ctx.saved_tensors[0]
    return None, (_camera_affine_bwd if plain_eager(gM, w2v) else _camera_affine_bwd_op)(gM, w2v)


torch.library.register_autograd("nanodrr_gb300::camera_affine", _camera_affine_backward,
                                setup_context=_camera_affine_context)


def _affine_product(A3: torch.Tensor, rt: torch.Tensor) -> torch.Tensor:
    """(A @ rt)[:, :3, :] for A3 = A[:3] ([3, 4]) and rt [B, 4, 4], written as a
    broadcast sum (camera -> voxel affine of the reference, backends.py:96)."""
    return (A3[None, :, :, None] * rt[:, None, :, :]).sum(dim=2)


def _call_affine(w2v: torch.Tensor, rt_inv: torch.Tensor, grad: bool) -> torch.Tensor:
    """M = (world_to_voxel @ rt_inv)[:, :3] in float32 (`_affine_product`),
    from the affine cache when no gradient is recorded and nothing is traced
    or captured into a CUDA graph (a graph must read rt_inv on every replay)."""
    def product():
        if not grad and _affine_takes(w2v, rt_inv):
            return _camera_affine(w2v, rt_inv, False)[0]
        return _affine_product(w2v.float()[:3], rt_inv.float())

    if (grad or (hasattr(torch, "compiler") and torch.compiler.is_compiling())
            or rt_inv.device.type != "cuda" or torch.cuda.is_current_stream_capturing()):
        return product()
    stream = _ffi.stream_handle(rt_inv.device)
    key = (id(w2v), id(rt_inv))
    hit = _M_CACHE.get(key)
    if hit is not None:
        wref, wver, rref, rver, M, made_on = hit
        if wref() is w2v and rref() is rt_inv and wver == w2v._version and rver == rt_inv._version:
            if stream != made_on:  # keep the allocator from reusing it under this stream's kernels
                M.record_stream(torch.cuda.current_stream(rt_inv.device))
            return M
    M = product()
    for k in [k for k, v in _M_CACHE.items() if v[0]() is None or v[2]() is None]:
        del _M_CACHE[k]  # entries whose tensors are gone
    while len(_M_CACHE) >= _M_CACHE_SIZE:
        _M_CACHE.pop(next(iter(_M_CACHE)))
    _M_CACHE[key] = (weakref.ref(w2v), w2v._version, weakref.ref(rt_inv), rt_inv._version, M, stream)
    return M


def compact_label(subject: Subject) -> torch.Tensor:
    """Label map for the kernels: float labels with n_classes <= 255 are packed
    to uint8 once per label tensor version (trunc(label) if it is a class in
    [0, C), else 255, which the kernels drop), saving 3 of 4 bytes per label
    read with identical routing. Other label maps pass through unchanged."""
    lab = subject.label[0, 0]
    C = subject.n_classes
    if not lab.is_floating_point() or C > 255:
        return lab.contiguous()
    key = (lab.data_ptr(), lab._version, lab.dtype, tuple(lab.shape), C, lab.device)
    cache = getattr(subject, "_ndrr_label_cache", None)
    if cache is not None and cache[0] == key:
        return cache[1]
    t = torch.trunc(lab.float())
    packed = torch.where((t >= 0) & (t < C), t, torch.full_like(t, 255.0)).to(torch.uint8).contiguous()
    object.__setattr__(subject, "_ndrr_label_cache", (key, packed))
    return packed


def _batched(t: torch.Tensor, B: int, dim: int) -> torch.Tensor:
    """`t` expanded to B poses (a leading batch added where it has one dimension
    less than `dim`), float32 and contiguous (itself when it is)."""
    if t.dim() == dim and t.shape[0] == B and t.dtype == torch.float32 and t.is_contiguous():
        return t
    return t.expand(B, *[-1] * (dim - 1)).float().contiguous()


def render_cuda(subject, rt_inv, src, tgt, step_size, n_samples, height, width) -> torch.Tensor:
    """Adapter from the render call to the `nanodrr_gb300::fused_raymarch_ex` op (the
    reference's `fused_raymarch` contract plus the layout, skip and the
    affine's low parts)."""
    C = subject.n_classes
    img = subject.image
    # A reshape of the [1, 1, D, H, W] image back-propagates as a view; an
    # index ([0, 0]) would allocate and zero a volume-sized gradient per level.
    vol = (img.reshape(img.shape[-3:]) if img.shape[:2] == (1, 1) else img[0, 0]).contiguous()
    lab = compact_label(subject) if C > 1 else vol
    # With a gradient recorded, the adjoint forms sample positions from M +
    # M_lo in float-float and carries them in fixed point
    # (ndrr_raymarch_args.M_lo): M_lo is the float32 product's error against
    # the float64 affine of the same inputs. The forward reads float32 M only,
    # so a call without a gradient skips the float64 product.
    grad = torch.is_grad_enabled() and any(t.requires_grad for t in (vol, rt_inv, src, tgt, step_size))
    if grad and _affine_takes(subject.world_to_voxel, rt_inv):
        if rt_inv.requires_grad:
            M, M_lo = _camera_affine_op(subject.world_to_voxel, rt_inv)
            M_lo = M_lo.detach()
        else:
            M, M_lo = _camera_affine(subject.world_to_voxel, rt_inv, True)
    elif not grad:
        M = _call_affine(subject.world_to_voxel, rt_inv, grad)
        M_lo = M.new_empty(0)
    else:
        M = _call_affine(subject.world_to_voxel, rt_inv, grad)
        M64 = _affine_product(subject.world_to_voxel.detach().double()[:3], rt_inv.detach().double())
        M_lo = (M64 - M.detach().double()).float()
    B = max(M.shape[0], tgt.shape[0])
    if M.shape[0] != B:
        M = M.expand(B, -1, -1)
        if grad:
            M_lo = M_lo.expand(B, -1, -1)
    if not _within_limits(img, C, B * height * width):
        raise ValueError("inputs exceed the CUDA kernel's limits (int32 indexing)")
    args = (
        vol,
        lab,
        M.contiguous(),
        _batched(src, B, 3),
        _batched(tgt, B, 3),
        _batched(step_size, B, 2),
        n_samples,
        C,
        width,
    )
    skip = getattr(subject, "empty_space", None)
    # The quad copy is cached by the volume's address and version, which a
    # traced graph cannot read: under torch.compile the plain layout is used.
    compiling = hasattr(torch, "compiler") and torch.compiler.is_compiling()
    if skip is not None and not compiling:
        skip.grid.refresh(vol)  # the grid must describe the volume rendered
    # The quad copy (4x the volume's bytes) pays when many poses reuse it
    # through L2; one pose streams it once, and a one-pose forward read 408 MB
    # from DRAM in 73.6 us (82 % of HBM) where the plain volume took 52 us
    # (512 x 512 x 400 f32, 200^2 x 500 samples). A forward of one pose with no
    # gradient recorded therefore reads the plain volume; same image either way.
    default = "plain" if (not grad and B == 1) else "quad"
    layout = "plain" if compiling else (getattr(subject, "layout", None) or default)
    # Without a recorded gradient the forward is called directly, skipping
    # the custom op's dispatch (tens of microseconds of host time per call).
    direct = not compiling and not grad
    quad = cached_quad(subject, vol, lab, C) if layout == "quad" else None
    if direct:
        sk = None
        if skip is not None and int(skip.mode) != _ffi.NDRR_SKIP_NONE:
            sk = _SkipArgs(skip.grid.grid, skip.grid.cell, skip.packed, int(skip.mode), float(skip.margin), vol.shape,
                           getattr(skip, "fused", True))
        return march_direct(vol, quad, *args[1:], skip=sk).reshape(B, C, height, width)
    empty = vol.new_empty(0, dtype=torch.uint8)
    if quad is None:
        quad = empty
    if skip is not None:
        # With a gradient recorded the skip always goes through sample windows
        # computed ahead of the march (not the in-kernel walk of a fused
        # occupancy skip): the adjoint reuses them, and with a volume gradient
        # they spare the loads of zero-corner samples (every sample is still
        # scattered).
        sk = (skip.grid.grid, skip.grid.cell, skip.packed, int(skip.mode), float(skip.margin),
              (not getattr(skip, "fused", True)) or grad)
    else:
        sk = (empty, 0, empty, 0, 0.0, False)
    slab_mib = int(getattr(subject, "slab_mib", 0))
    if (C == 1 and layout == "quad" and M.requires_grad and B * tgt.shape[1] >= _SUMS_RAYS
            and max(vol.shape) < 1 << 22 and not any(t.requires_grad for t in (src, tgt, step_size))):
        out = fused_raymarch_sums(vol, quad, args[2], M_lo.contiguous(), *args[3:7], width, *sk[:5], slab_mib)[0]
        return out.reshape(B, C, height, width)
    out = fused_raymarch_ex(args[0], quad, args[1], args[2], M_lo.contiguous(), *args[3:], *sk, slab_mib)[0]
    return out.reshape(B, C, height, width)


def labeled_quad_applies(vol: torch.Tensor, n_classes: int) -> bool:
    """Per-label renders of 16-bit volumes read the labelled quad layout:
    the class of a sample rides in the loads of its corners."""
    return vol.dtype in (torch.float16, torch.bfloat16) and 2 <= n_classes <= 255


def quad_cache_key(vol: torch.Tensor, lab: torch.Tensor | None, n_classes: int) -> tuple:
    key = (vol.data_ptr(), vol._version, vol.dtype, tuple(vol.shape), vol.device)
    if lab is not None and labeled_quad_applies(vol, n_classes):
        key += (lab.data_ptr(), lab._version, lab.dtype, n_classes)
    return key


def build_quad(vol: torch.Tensor, lab: torch.Tensor | None, n_classes: int, out: torch.Tensor | None = None):
    if lab is not None and labeled_quad_applies(vol, n_classes):
        return quad_volume_labeled(vol.detach(), lab, n_classes, out=out)
    return quad_volume(vol.detach(), out=out)


def cached_quad(subject, vol: torch.Tensor, lab: torch.Tensor | None = None, n_classes: int = 1) -> torch.Tensor:
    """The volume's quad-layout copy (labelled with `lab`'s classes for a
    per-label render of a 16-bit volume), rebuilt whenever the volume or
    label tensor or their contents (version counters) change."""
    key = quad_cache_key(vol, lab, n_classes)
    cache = getattr(subject, "_ndrr_quad_cache", None)
    if cache is not None and cache[0] == key:
        return cache[1]
    q = build_quad(vol, lab, n_classes)
    object.__setattr__(subject, "_ndrr_quad_cache", (key, q, lab, n_classes))
    return q


def render(
    subject: Subject,
    k_inv: torch.Tensor,
    rt_inv: torch.Tensor,
    sdd: torch.Tensor,
    height: int,
    width: int,
    n_samples: int = 500,
    orthographic: bool = False,
    src: torch.Tensor | None = None,
    tgt: torch.Tensor | None = None,
    backend: str = "auto",
) -> torch.Tensor:
    """Differentiable DRR: [B, C, H, W] line integrals of `subject.image`
    (per label channel when the subject has a multi-class label map).

    Args mirror the reference: `k_inv` [B|1, 3, 3], `rt_inv` [B, 4, 4]
    (camera -> world), `sdd` [B|1]; optional precomputed camera-space ray
    endpoints `src` [B, 1|N, 3] and `tgt` [B, N, 3]. Gradients flow to the
    pose, the intrinsics, the ray endpoints and the volume."""
    if n_samples < 2:
        raise ValueError("n_samples must be at least 2")
    if backend not in _BACKENDS:
        raise ValueError(f"Unknown backend {backend!r}; expected 'auto', 'cuda', or 'triton'")
    if not rt_inv.is_cuda or not subject.image.is_cuda:
        raise RuntimeError("nanodrr_gb300 renders on CUDA devices only; move the subject and poses to a GPU")
    device, dtype = rt_inv.device, rt_inv.dtype
    if tgt is None and src is None:
        rays = _cached_rays(k_inv, sdd, height, width, n_samples, orthographic, rt_inv)
        if rays is not None:
            return render_cuda(subject, rt_inv, *rays, n_samples, height, width)
        if _ray_setup_takes(k_inv, sdd, height, width, rt_inv):
            B = max(rt_inv.shape[0], k_inv.shape[0], sdd.shape[0])
            args = (k_inv, sdd, B, height, width, n_samples, bool(orthographic))
            live = torch.is_grad_enabled() and (k_inv.requires_grad or sdd.requires_grad)
            rays = (_ray_setup_op if live else _ray_setup)(*args)
            return render_cuda(subject, rt_inv, *rays, n_samples, height, width)
    if tgt is None and src is None:
        src, tgt = _camera_rays(k_inv, sdd, height, width, orthographic, device, dtype)
    if tgt is None:
        tgt = _make_tgt(k_inv, sdd, height, width, device, dtype)
    if src is None:
        src = _make_src(orthographic, tgt, sdd)
    step_size = (tgt - src).norm(dim=-1) / float(n_samples - 1)
    return render_cuda(subject, rt_inv, src, tgt, step_size, n_samples, height, width)


def _cached_rays(k_inv, sdd, height, width, n_samples, orthographic, rt_inv):
    """(src, tgt, step) of the render call, float32, expanded to the batch and
    contiguous, from the ray cache or built and stored there; None when the
    call differentiates the camera (k_inv or sdd requires a gradient), is
    traced, or is captured into a CUDA graph (a graph must own its rays: a
    cache entry may be evicted and freed while the graph still replays)."""
    if k_inv.requires_grad or sdd.requires_grad:
        return None
    if hasattr(torch, "compiler") and torch.compiler.is_compiling():
        return None
    device, dtype = rt_inv.device, rt_inv.dtype
    if device.type != "cuda" or torch.cuda.is_current_stream_capturing():
        return None
    stream = _ffi.stream_handle(device)
    B = max(rt_inv.shape[0], k_inv.shape[0], sdd.shape[0])
    key = (id(k_inv), id(sdd), height, width, n_samples, bool(orthographic), B, dtype, device)
    hit = _RAY_CACHE.get(key)
    if hit is not None:
        kref, kver, sref, sver, rays, made_on = hit
        if kref() is k_inv and sref() is sdd and kver == k_inv._version and sver == sdd._version:
            if stream != made_on:  # keep the allocator from reusing them under this stream's kernels
                for t in rays:
                    t.record_stream(torch.cuda.current_stream(device))
            return rays
    if _ray_setup_takes(k_inv, sdd, height, width, rt_inv):
        rays = _ray_setup(k_inv, sdd, B, height, width, n_samples, bool(orthographic))
    else:
        src, tgt = _camera_rays(k_inv, sdd, height, width, orthographic, device, dtype)
        step = (tgt - src).norm(dim=-1) / float(n_samples - 1)
        rays = (src.expand(B, -1, -1).float().contiguous(), tgt.expand(B, -1, -1).float().contiguous(),
                step.expand(B, -1).float().contiguous())
    for k in [k for k, v in _RAY_CACHE.items() if v[0]() is None or v[2]() is None]:
        del _RAY_CACHE[k]  # entries whose camera tensors are gone
    while len(_RAY_CACHE) >= _RAY_CACHE_SIZE:
        _RAY_CACHE.pop(next(iter(_RAY_CACHE)))
    _RAY_CACHE[key] = (weakref.ref(k_inv), k_inv._version, weakref.ref(sdd), sdd._version, rays, stream)
    return rays
