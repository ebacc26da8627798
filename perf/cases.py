"""Workloads of the renderer, through its public entry points.

A case is a dict of plain values; `prepare` makes the inputs of one (seeded,
on the GPU) and whatever a user's program keeps between calls, `run` is one
pass and `exact` the same results in 64 bits from torch's own operators.
Volumes are body-in-air phantoms (soft tissue, a few bone ellipsoids, noise),
poses +-30 degrees and +-50 mm about an AP view, the source 600 mm from the
isocenter and the detector 1020 mm from the source.
"""

from __future__ import annotations

import math

import torch
import torch.nn.functional as F

import nanodrr_gb300 as nd
from nanodrr_gb300.batched import BatchedRenderer, RenderRequest
from nanodrr_gb300.empty_space import EmptySpace
from nanodrr_gb300.registration import GraphedStep, NormalizedCrossCorrelation2d, Registration

SOD, SDD = 600.0, 1020.0
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


def _case(name, kind, shape, spacing, **more):
    D, H, W = shape
    sx, sy, sz = spacing
    return {"name": name, "kind": kind, "D": D, "H": H, "W": W, "sx": sx, "sy": sy, "sz": sz, **more}


def listed():
    return [
        # One frame for display or for a derivative-free search: one AP pose,
        # no gradient, the call of the published single-frame benchmark.
        _case("frame_200", "frame", (400, 512, 512), (0.8, 0.8, 1.0), dtype="f32", B=1, height=200, width=200,
              pixel=2.0, samples=500, orthographic=False),
        # The smallest step in use: one pose of a small scan at the coarse
        # level of a registration, replayed from a CUDA graph (latency).
        _case("pose_step_coarse", "pose", (128, 128, 128), (1.0, 1.0, 1.0), dtype="f32", B=1, height=100, width=100,
              pixel=2.8, samples=250, graph=True),
        # The ordinary registration: a batch of poses of one scan, NCC loss,
        # gradients to the pose parameters, eager autograd.
        _case("pose_step_16", "pose", (400, 512, 512), (0.8, 0.8, 1.0), dtype="f32", B=16, height=200, width=200,
              pixel=1.5, samples=500, graph=False),
        # The benchmark's registration step: poses and volume both learned.
        _case("volume_step_32", "volume", (512, 512, 512), (0.8, 0.8, 1.0), dtype="f32", B=32, height=256, width=256,
              pixel=1.2, samples=800, graph=True),
        # Tomographic reconstruction: fixed views, a volume that the
        # optimiser changed since the last pass; ragged sizes.
        _case("reconstruct_9", "reconstruct", (277, 250, 301), (1.1, 1.3, 1.2), dtype="f32", B=9, height=211,
              width=187, pixel=1.9, samples=383),
        # Per-label projections of a segmented scan held in 16 bits.
        _case("labels_32", "labels", (400, 512, 512), (0.8, 0.8, 1.0), dtype="bf16", B=32, height=256, width=256,
              pixel=1.2, samples=800, classes=8, grad=False),
        # Large detector with empty-space skipping, gradients to the pose
        # (the largest case by rays and samples).
        _case("skip_1024", "skip", (400, 512, 512), (0.8, 0.8, 1.0), dtype="f32", B=8, height=1024, width=1024,
              pixel=0.3, samples=1000),
        # A serving batch: requests of uneven volumes, detectors and sample
        # counts in one launch, forward and pose gradients.
        _case("batch_uneven", "batch", (300, 512, 512), (0.8, 0.8, 0.8), dtype="f32", requests=32, most_side=512,
              least_samples=300, most_samples=1000),
        # Calibration: gradients to intrinsics and pose of a half-precision
        # scan, odd sizes.
        _case("calibrate_f16", "camera", (193, 211, 257), (1.4, 1.3, 1.1), dtype="f16", B=3, height=133, width=211,
              pixel=1.7, samples=333, orthographic=False),
        # Local (patch-wise) NCC of a multi-start registration, both ways.
        {"name": "local_ncc", "kind": "ncc", "B": 8, "height": 200, "width": 200, "patch": 13},
        # Undoing a detector's intrinsics on a stack of radiographs, both ways.
        {"name": "resample_512", "kind": "resample", "B": 8, "C": 1, "height": 512, "width": 512},
        # A new patient: HU to attenuation, occupancy grid, first images.
        _case("new_subject", "subject", (400, 512, 512), (0.8, 0.8, 1.0), dtype="f32", B=4, height=200, width=200,
              pixel=1.5, samples=500),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _scan(rng, lo, hi):
    """Sizes and spacings of a scan 220 to 410 mm across."""
    shape = [_log(rng, lo, hi) for _ in range(3)]
    D, H, W = shape
    return {"D": D, "H": H, "W": W, **{k: round(rng.uniform(220.0, 410.0) / n, 3) for k, n in
                                       (("sx", W), ("sy", H), ("sz", D))}}


def _detector(rng, lo, hi):
    h, w = _log(rng, lo, hi), _log(rng, lo, hi)
    return {"height": h, "width": w, "pixel": round(rng.uniform(250.0, 420.0) / max(h, w), 3)}


def draw(rng):
    kind = rng.choice(["frame", "pose", "pose", "volume", "reconstruct", "labels", "skip", "batch", "camera", "ncc",
                       "resample", "subject"])
    any_type = rng.choice(["f32", "f32", "f16", "bf16"])
    if kind == "frame":
        return {"kind": kind, **_scan(rng, 96, 512), "dtype": any_type, "B": rng.choice([1, 1, 2, 4]),
                **_detector(rng, 64, 512), "samples": _log(rng, 150, 1000), "orthographic": rng.random() < 0.25}
    if kind == "pose":
        return {"kind": kind, **_scan(rng, 96, 512), "dtype": any_type, "B": _log(rng, 1, 32),
                **_detector(rng, 80, 280), "samples": _log(rng, 150, 800), "graph": rng.random() < 0.5}
    if kind == "volume":
        return {"kind": kind, **_scan(rng, 128, 512), "dtype": "f32", "B": _log(rng, 2, 32),
                **_detector(rng, 80, 256), "samples": _log(rng, 200, 800), "graph": rng.random() < 0.5}
    if kind == "reconstruct":
        return {"kind": kind, **_scan(rng, 96, 400), "dtype": "f32", "B": _log(rng, 2, 16),
                **_detector(rng, 80, 256), "samples": _log(rng, 200, 600)}
    if kind == "labels":
        return {"kind": kind, **_scan(rng, 96, 512), "dtype": any_type, "B": _log(rng, 1, 32),
                **_detector(rng, 64, 256), "samples": _log(rng, 150, 800), "classes": rng.randint(2, 12),
                "grad": rng.random() < 0.3}
    if kind == "skip":
        return {"kind": kind, **_scan(rng, 128, 512), "dtype": any_type, "B": _log(rng, 1, 8),
                **_detector(rng, 200, 1000), "samples": _log(rng, 300, 1000)}
    if kind == "batch":
        return {"kind": kind, **_scan(rng, 128, 400), "dtype": any_type, "requests": _log(rng, 4, 32),
                "most_side": _log(rng, 128, 512), "least_samples": 200, "most_samples": _log(rng, 400, 1000)}
    if kind == "camera":
        return {"kind": kind, **_scan(rng, 96, 320), "dtype": any_type, "B": _log(rng, 1, 8),
                **_detector(rng, 64, 256), "samples": _log(rng, 150, 600), "orthographic": rng.random() < 0.25}
    if kind == "ncc":
        return {"kind": kind, "B": _log(rng, 1, 8), "height": _log(rng, 64, 200), "width": _log(rng, 64, 200),
                "patch": rng.choice([0, 7, 9, 13])}
    if kind == "resample":
        return {"kind": kind, "B": _log(rng, 1, 8), "C": rng.choice([1, 1, 3]), "height": _log(rng, 64, 512),
                "width": _log(rng, 64, 512)}
    return {"kind": kind, **_scan(rng, 128, 450), "dtype": any_type, "B": rng.choice([1, 2, 4]),
            **_detector(rng, 100, 200), "samples": _log(rng, 200, 500)}


# ------------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _phantom(case, seed, classes=0):
    """HU volume [D, H, W] float32 (air -1000 outside the body) and, with
    `classes`, its label map (0 air, 1 tissue, 2.. the bones)."""
    D, H, W = case["D"], case["H"], case["W"]
    host = torch.Generator().manual_seed(int(seed) + 17)
    z, y, x = (torch.linspace(-1.0, 1.0, n, device="cuda").reshape([-1 if i == k else 1 for i in range(3)])
               for k, n in enumerate((D, H, W)))
    u = torch.rand(3, generator=host)
    body = (x / (0.88 + 0.08 * u[0].item())) ** 2 + (y / (0.66 + 0.1 * u[1].item())) ** 2 \
        + (z / (0.88 + 0.08 * u[2].item())) ** 2 <= 1.0
    hu = torch.randn(D, H, W, device="cuda", generator=_generator(seed)).mul_(10.0).add_(40.0)
    label = body.to(torch.float32) if classes else None
    for i in range(max(6, classes - 2)):
        c = (torch.rand(3, generator=host) - 0.5) * 0.9
        r = 0.08 + 0.16 * torch.rand(3, generator=host)
        value = 400.0 + 1100.0 * torch.rand((), generator=host).item()
        cx, cy, cz = (c * torch.tensor([0.88, 0.66, 0.88])).tolist()
        rx, ry, rz = r.tolist()
        bone = ((x - cx) / rx) ** 2 + ((y - cy) / ry) ** 2 + ((z - cz) / rz) ** 2 <= 1.0
        hu.masked_fill_(bone, value)
        if classes and 2 + i < classes:
            label.masked_fill_(bone & body, float(2 + i))
    hu.masked_fill_(~body, -1000.0)
    return hu, label


def _mu(hu):
    return (hu / 1000.0 + 1.0).mul_(0.02).clamp_(min=0.0)


def _rotations(angles):
    """Intrinsic ZXY rotations [n, 3, 3] from degrees [n, 3]."""
    a = angles.double() * (math.pi / 180.0)
    c, s = torch.cos(a), torch.sin(a)
    n = angles.shape[0]
    Rz, Rx, Ry = (torch.eye(3, dtype=torch.float64).repeat(n, 1, 1) for _ in range(3))
    Rz[:, 0, 0], Rz[:, 0, 1], Rz[:, 1, 0], Rz[:, 1, 1] = c[:, 0], -s[:, 0], s[:, 0], c[:, 0]
    Rx[:, 1, 1], Rx[:, 1, 2], Rx[:, 2, 1], Rx[:, 2, 2] = c[:, 1], -s[:, 1], s[:, 1], c[:, 1]
    Ry[:, 0, 0], Ry[:, 0, 2], Ry[:, 2, 0], Ry[:, 2, 2] = c[:, 2], s[:, 2], -s[:, 2], c[:, 2]
    return Rz @ Rx @ Ry


def _poses(n, seed):
    """Camera-to-world poses [n, 4, 4], float32."""
    g = torch.Generator().manual_seed(int(seed) + 29)
    R = _rotations((torch.rand(n, 3, generator=g) * 2 - 1) * 30.0)
    t = torch.tensor([0.0, SOD, 0.0], dtype=torch.float64) + (torch.rand(n, 3, generator=g).double() * 2 - 1) * 50.0
    ap = torch.tensor([[-1.0, 0, 0], [0, 0, -1.0], [0, -1.0, 0]], dtype=torch.float64)
    rt = torch.eye(4, dtype=torch.float64).repeat(n, 1, 1)
    rt[:, :3, :3] = R @ ap
    rt[:, :3, 3] = (R @ t[..., None])[..., 0]
    return rt.float().cuda()


def _camera(height, width, pixel):
    f = SDD / pixel
    k_inv = torch.tensor([[[1 / f, 0.0, -width / 2 / f], [0.0, 1 / f, -height / 2 / f], [0.0, 0.0, 1.0]]])
    return k_inv.cuda(), torch.tensor([SDD], device="cuda")


def _nudges(n, seed):
    """Offsets of a registration's start: 0.05 rad and 5 mm at most."""
    g = torch.Generator().manual_seed(int(seed) + 43)
    return ((torch.rand(n, 3, generator=g) * 2 - 1) * 0.05).cuda(), ((torch.rand(n, 3, generator=g) * 2 - 1) * 5.0).cuda()


def _spacing(case):
    return case["sx"], case["sy"], case["sz"]


def _subject(case, seed):
    classes = case.get("classes", 0)
    hu, label = _phantom(case, seed, classes)
    vol = _mu(hu).to(DTYPES[case["dtype"]])
    return nd.Subject.from_volume(vol, _spacing(case), label=label, max_label=max(classes - 1, 0), convert_to_mu=False)


def _requests(case):
    """(scan, height, width, pixel, samples) of a batch's requests; three scans."""
    g = torch.Generator().manual_seed(case["requests"] * 1009 + case["most_side"])
    scans = [case, {**case, **{k: max(32, case[k] * 4 // 5) for k in "DHW"}},
             {**case, **{k: max(32, case[k] // 2) for k in "DHW"}, **{k: case[k] * 2 for k in ("sx", "sy", "sz")}}]
    sides = [max(16, int(case["most_side"] * f)) for f in (0.25, 0.39, 0.5, 0.75, 1.0)]
    out = []
    for i in range(case["requests"]):
        h, w, v = (int(torch.randint(0, n, (), generator=g)) for n in (5, 5, 3))
        s = int(torch.randint(case["least_samples"], case["most_samples"] + 1, (), generator=g))
        out.append((v, sides[h], sides[w], 330.0 / max(sides[h], sides[w]), s))
    return scans, out


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "ncc":
        g = _generator(seed)
        a = torch.rand(case["B"], 1, case["height"], case["width"], device="cuda", generator=g)
        b = torch.rand(a.shape, device="cuda", generator=g)
        smooth = F.avg_pool2d(F.pad(a, (4, 4, 4, 4), mode="replicate"), 9, stride=1)
        st["moving"] = (smooth * 4.0 + 0.05 * b).requires_grad_(True)
        st["fixed"] = torch.roll(smooth, (1, 2), (2, 3)) * 4.0 + 0.05 * a
        st["metric"] = NormalizedCrossCorrelation2d(patch_size=case["patch"] or None)
        return st
    if kind == "resample":
        g = _generator(seed)
        st["img"] = torch.rand(case["B"], case["C"], case["height"], case["width"], device="cuda",
                               generator=g).requires_grad_(True)
        st["go"] = torch.randn(st["img"].shape, device="cuda", generator=g)
        st["old"], st["new"] = (k.requires_grad_(True) for k in _resample_cameras(case, seed))
        return st
    if kind == "batch":
        scans, reqs = _requests(case)
        subs = [_subject(s, seed + i) for i, s in enumerate(scans)]
        todo = []
        for v, h, w, px, s in reqs:
            k_inv, sdd = _camera(h, w, px)
            todo.append(RenderRequest(subs[v], k_inv, sdd, h, w, s))
        st["renderer"] = BatchedRenderer(todo)
        st["poses"] = _poses(len(todo), seed)
        st["go"] = torch.randn(st["renderer"].go_flat.shape, device="cuda",
                               generator=_generator(seed + 5)).to(st["renderer"].go_flat.dtype)
        return st
    k_inv, sdd = _camera(case["height"], case["width"], case["pixel"])
    rt = _poses(case["B"], seed)
    st |= {"k_inv": k_inv, "sdd": sdd, "rt": rt}
    if kind == "subject":
        st["hu"] = _phantom(case, seed)[0].to(DTYPES[case["dtype"]])
        return st
    sub = st["subject"] = _subject(case, seed)
    size = (case["height"], case["width"])
    if kind in ("pose", "volume", "skip"):
        st["target"] = nd.render(sub, k_inv, rt, sdd, *size, n_samples=case["samples"])
        ncc = NormalizedCrossCorrelation2d()
        st["loss"] = lambda img, target: -ncc(img, target).mean()
        if kind == "skip":
            sub.empty_space = EmptySpace.occupancy(sub.image[0, 0])
        if kind == "volume":
            sub._image_hu = sub._image_hu.requires_grad_(True)
        reg = st["reg"] = Registration(sub, rt, k_inv, sdd, *size, batch=case["B"])
        with torch.no_grad():
            for p, v in zip((reg._rot, reg._xyz), _nudges(case["B"], seed)):
                p.copy_(v)
        if case.get("graph"):
            st["step"] = GraphedStep(reg, st["loss"], st["target"], n_samples=case["samples"])
    elif kind == "reconstruct":
        st["views"] = nd.render(sub, k_inv, rt, sdd, *size, n_samples=case["samples"])
        st["update"] = sub._image_hu * (1 + 0.2 * torch.rand(sub._image_hu.shape, device="cuda",
                                                              generator=_generator(seed + 7)))
        sub._image_hu = torch.zeros_like(sub._image_hu).requires_grad_(True)
    elif kind == "camera" or case.get("grad"):
        st["go"] = torch.randn(case["B"], case.get("classes", 1), *size, device="cuda",
                               generator=_generator(seed + 5)).to(DTYPES[case["dtype"]])
        rt.requires_grad_(True)
        if kind == "camera":
            k_inv.requires_grad_(True)
    return st


def _resample_cameras(case, seed):
    """Inverse intrinsics [B, 3, 3] before and after, some pixels apart."""
    h, w, B = case["height"], case["width"], case["B"]
    g = torch.Generator().manual_seed(int(seed) + 61)
    got = []
    for scale in (0.0, 0.1):
        f = 2.0 * max(h, w) * (1 + scale * (torch.rand(B, 2, generator=g).double() - 0.5))
        c = torch.tensor([w / 2, h / 2]).double() * (1 + scale * (torch.rand(B, 2, generator=g).double() - 0.5))
        k = torch.eye(3, dtype=torch.float64).repeat(B, 1, 1)
        k[:, 0, 0], k[:, 1, 1], k[:, 0, 2], k[:, 1, 2] = 1 / f[:, 0], 1 / f[:, 1], -c[:, 0] / f[:, 0], -c[:, 1] / f[:, 1]
        got.append(k.float().cuda())
    return got


# ---------------------------------------------------------------- one pass
def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "ncc":
        st["moving"].grad = None
        score = st["metric"](st["moving"], st["fixed"])
        (-score.mean()).backward()
        return {"score": score.detach(), "moving": st["moving"].grad}
    if kind == "resample":
        for k in ("img", "old", "new"):
            st[k].grad = None
        out = nd.resample(st["img"], st["old"], st["new"])
        out.backward(st["go"])
        return {"out": out.detach(), "img": st["img"].grad, "old": st["old"].grad, "new": st["new"].grad}
    if kind == "batch":
        r = st["renderer"]
        r.set_poses(st["poses"])
        r.forward()
        r.go_flat.copy_(st["go"])
        r.backward()
        return {"images": r.out_flat, "poses": r.pose_grad()}
    size, S = (case["height"], case["width"]), case["samples"]
    if kind == "subject":
        sub = nd.Subject.from_volume(st["hu"], _spacing(case), max_label=0)
        mu = sub.image
        sub.empty_space = EmptySpace.occupancy(mu[0, 0])
        img = nd.render(sub, st["k_inv"], st["rt"], st["sdd"], *size, n_samples=S)
        return {"mu": mu, "grid": sub.empty_space.grid.grid, "image": img}
    sub = st["subject"]
    if kind in ("pose", "volume", "skip"):
        reg = st["reg"]
        if "step" in st:
            loss = st["step"].replay()
            return {"loss": loss, "grads": list(st["step"].grads)}
        params = [reg._rot, reg._xyz] + ([sub._image_hu] if kind == "volume" else [])
        for p in params:
            p.grad = None
        loss = st["loss"](reg(n_samples=S), st["target"])
        loss.backward()
        return {"loss": loss.detach(), "grads": [p.grad for p in params]}
    if kind == "reconstruct":
        vol = sub._image_hu
        with torch.no_grad():
            vol.copy_(st["update"])  # what the optimiser's step leaves behind
        vol.grad = None
        img = nd.render(sub, st["k_inv"], st["rt"], st["sdd"], *size, n_samples=S)
        loss = (img - st["views"]).square().mean()
        loss.backward()
        return {"image": img.detach(), "loss": loss.detach(), "volume": vol.grad}
    if kind == "camera" or case.get("grad"):
        st["rt"].grad = st["k_inv"].grad = None
        img = nd.render(sub, st["k_inv"], st["rt"], st["sdd"], *size, n_samples=S,
                        orthographic=case.get("orthographic", False))
        img.backward(st["go"])
        return {"image": img.detach(), "poses": st["rt"].grad, "intrinsics": st["k_inv"].grad}
    return nd.render(sub, st["k_inv"], st["rt"], st["sdd"], *size, n_samples=S,
                     orthographic=case.get("orthographic", False))


# ------------------------------------------------- what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "ncc":
        p = case["patch"] or 1
        pixels = case["B"] * case["height"] * case["width"]
        return {"bytes": 12.0 * pixels, "flops": 30.0 * pixels * p * p}
    if kind == "resample":
        pixels = case["B"] * case["C"] * case["height"] * case["width"]
        return {"bytes": 16.0 * pixels, "flops": 60.0 * pixels}
    es = 4 if case["dtype"] == "f32" else 2
    voxels = case["D"] * case["H"] * case["W"]
    depth = 0.5 * (case["H"] * case["sy"]) / SDD + 0.5 * min(case["H"] * case["sy"], case["D"] * case["sz"]) / SDD
    if kind == "batch":
        rays = sum(h * w for _, h, w, _, _ in _requests(case)[1])
        taps = sum(h * w * s for _, h, w, _, s in _requests(case)[1]) * depth
        voxels = voxels * 1.63
    else:
        rays = case["B"] * case["height"] * case["width"]
        taps = rays * case["samples"] * depth
    out = rays * es * max(1, case.get("classes", 1))
    volume = min(voxels, 8 * taps) * es
    forward, adjoint, scatter = 30.0 * taps, 60.0 * taps, 24.0 * taps
    if kind in ("frame", "subject") or (kind == "labels" and not case["grad"]):
        extra = 2 * voxels * es if kind == "subject" else volume if kind == "labels" else 0
        return {"bytes": volume + out + extra, "flops": forward}
    if kind in ("volume", "reconstruct"):
        return {"bytes": volume + voxels * 4 + 3 * out, "flops": forward + adjoint + scatter}
    return {"bytes": volume + 3 * out, "flops": forward + adjoint}


# --------------------------------------------------------- the same in 64 bits
CHUNK = 24_000_000  # samples at a time


def _world_to_voxel(case):
    D, H, W = case["D"], case["H"], case["W"]
    step = torch.tensor(_spacing(case), dtype=torch.float64)
    m = torch.eye(4, dtype=torch.float64)
    m[:3, :3] = torch.diag(1 / step)
    m[:3, 3] = 0.5 * torch.tensor([W - 1, H - 1, D - 1], dtype=torch.float64)
    return m.float().double().cuda()  # a scan's affine is kept in 32 bits


def _rays64(k_inv, sdd, height, width, orthographic):
    v, u = torch.meshgrid(torch.arange(height, device="cuda", dtype=torch.float64) + 0.5,
                          torch.arange(width, device="cuda", dtype=torch.float64) + 0.5, indexing="ij")
    uv1 = torch.stack([u, v, torch.ones_like(u)], -1).reshape(-1, 3)
    tgt = sdd[:, None, None] * (uv1 @ k_inv.transpose(1, 2))
    if orthographic:
        src = tgt - sdd[:, None, None] * torch.tensor([0.0, 0, 1.0], device="cuda", dtype=torch.float64)
    else:
        src = torch.zeros_like(tgt)
    return src, tgt


def _march64(vol, label, classes, M, src, tgt, samples):
    """[classes, n] line integrals of n rays of one pose."""
    p, q = (x @ M[:3, :3].T + M[:3, 3] for x in (src, tgt))
    t = torch.linspace(0, 1, samples, dtype=torch.float64, device="cuda")[:, None, None]
    D, H, W = vol.shape
    size = torch.tensor([W, H, D], dtype=torch.float64, device="cuda")
    at = ((2 * (p + t * (q - p)) + 1) / size - 1)[None, None]
    got = F.grid_sample(vol[None, None], at, mode="bilinear", align_corners=False)[0, 0, 0]
    step = (tgt - src).norm(dim=-1) / (samples - 1)
    if classes <= 1:
        return (got.sum(0) * step)[None]
    which = F.grid_sample(label[None, None], at.detach(), mode="nearest", align_corners=False)[0, 0, 0].long()
    return torch.zeros(classes, p.shape[0], dtype=torch.float64, device="cuda").scatter_add(0, which, got) * step


def _render64(case, vol, label, rt, k_inv, sdd, go=None, w2v=None):
    """[B, classes, height, width], and with `go` (the gradient of it) the
    gradients accumulated in the leaves among vol, rt and k_inv."""
    B, S, classes = rt.shape[0], case["samples"], max(1, case.get("classes", 1))
    n = case["height"] * case["width"]
    w2v = _world_to_voxel(case) if w2v is None else w2v
    rows = max(1, CHUNK // S)
    out = torch.zeros(B, classes, n, dtype=torch.float64, device="cuda")
    for b in range(B):
        for i in range(0, n, rows):
            with torch.set_grad_enabled(go is not None):
                src, tgt = _rays64(k_inv, sdd, case["height"], case["width"], case.get("orthographic", False))
                got = _march64(vol, label, classes, w2v @ rt[b], src[0, i:i + rows], tgt[0, i:i + rows], S)
            out[b, :, i:i + rows] = got.detach()
            if go is not None:
                got.backward(go.reshape(B, classes, n)[b, :, i:i + rows])
    return out.reshape(B, classes, case["height"], case["width"])


def _ncc64(a, b, eps=1e-7):
    a, b = (x - x.mean((-1, -2), keepdim=True) for x in (a, b))
    a, b = (x / (x.square().mean((-1, -2), keepdim=True) + eps).sqrt() for x in (a, b))
    return (a * b).mean((1, 2, 3))


def _registration_poses64(rt, rot, xyz):
    """rt P T P^-1 with P the translation to the isocenter in the camera and
    T = [R(rot) | R(rot) xyz]."""
    x, y, z = rot.unbind(-1)
    o = torch.zeros_like(x)
    R = torch.linalg.matrix_exp(torch.stack([o, -z, y, z, o, -x, -y, x, o], -1).reshape(-1, 3, 3))
    c = torch.linalg.inv(rt)[:, :3, 3:]
    t = R @ xyz[..., None] + c - R @ c
    last = torch.tensor([0.0, 0, 0, 1.0], dtype=torch.float64, device="cuda").expand(rt.shape[0], 1, 4)
    return rt @ torch.cat([torch.cat([R, t], -1), last], 1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "ncc":
        st = prepare(case, seed)
        a, b, p = st["moving"].detach().double().requires_grad_(True), st["fixed"].double(), case["patch"]
        if p:
            score = _ncc64(*(x.unfold(2, p, 1).unfold(3, p, 1).reshape(x.shape[0], -1, p, p) for x in (a, b)))
        else:
            score = _ncc64(a, b)
        (-score.mean()).backward()
        return {"score": score.detach(), "moving": a.grad}
    if kind == "resample":
        st = prepare(case, seed)
        img, old, new = (st[k].detach().double().requires_grad_(True) for k in ("img", "old", "new"))
        h, w = img.shape[-2:]
        y, x = torch.meshgrid(*(torch.arange(n, device="cuda", dtype=torch.float64) for n in (h, w)), indexing="ij")
        p = torch.stack([x, y, torch.ones_like(x)], -1).reshape(-1, 3) @ (torch.linalg.inv(old) @ new).transpose(1, 2)
        at = p[..., :2] / p[..., 2:] * (2 / torch.tensor([w - 1, h - 1], device="cuda", dtype=torch.float64)) - 1
        out = F.grid_sample(img, at.reshape(-1, h, w, 2), mode="bilinear", align_corners=True)
        out.backward(st["go"].double())
        return {"out": out.detach(), "img": img.grad, "old": old.grad, "new": new.grad}
    if kind == "batch":
        scans, reqs = _requests(case)
        dt = DTYPES[case["dtype"]]
        vols = [_mu(_phantom(s, seed + i)[0]).to(dt).double() for i, s in enumerate(scans)]
        poses = _poses(len(reqs), seed).double().requires_grad_(True)
        go = torch.randn(sum(h * w for _, h, w, _, _ in reqs), device="cuda",
                         generator=_generator(seed + 5)).to(dt).double()
        images, at = [], 0
        for i, (v, h, w, px, s) in enumerate(reqs):
            k_inv, sdd = (x.double() for x in _camera(h, w, px))
            one = {"height": h, "width": w, "samples": s}
            images.append(_render64(one, vols[v], None, poses[i:i + 1], k_inv, sdd, go=go[at:at + h * w],
                                    w2v=_world_to_voxel(scans[v])).reshape(-1))
            at += h * w
        return {"images": torch.cat(images), "poses": poses.grad}
    k_inv, sdd = (x.double() for x in _camera(case["height"], case["width"], case["pixel"]))
    rt = _poses(case["B"], seed).double()
    classes = case.get("classes", 0)
    hu, label = _phantom(case, seed, classes)
    dt = DTYPES[case["dtype"]]
    if kind == "subject":
        h = hu.to(dt).double().clamp(min=-1000.0)
        mu = torch.where(h > 0, 0.0192 + h / 1000.0 * (0.0573 - 0.0192), (h / 1000.0 + 1) * 0.0192).clamp(min=0.0)
        return {"mu": mu[None, None], "grid": None,
                "image": _render64(case, mu.to(dt).double(), None, rt, k_inv, sdd)}
    vol = _mu(hu).to(dt).double()
    del hu
    label = label.double() if label is not None else None
    if kind in ("pose", "volume", "skip"):
        target = _render64(case, vol, label, rt, k_inv, sdd)
        rot, xyz = (x.double().requires_grad_(True) for x in _nudges(case["B"], seed))
        pose = _registration_poses64(rt, rot, xyz)
        at = pose.detach().requires_grad_(True)
        img = _render64(case, vol, label, at, k_inv, sdd).requires_grad_(True)
        loss = -_ncc64(img, target).mean()
        loss.backward()
        vol.requires_grad_(kind == "volume")
        _render64(case, vol, label, at, k_inv, sdd, go=img.grad)
        pose.backward(at.grad)
        grads = [rot.grad, xyz.grad] + ([vol.grad[None, None]] if kind == "volume" else [])
        return {"loss": loss.detach(), "grads": grads}
    if kind == "reconstruct":
        views = _render64(case, vol, label, rt, k_inv, sdd)
        gain = torch.rand((1, 1) + tuple(vol.shape), device="cuda", generator=_generator(seed + 7))
        vol = (vol.float() * (1 + 0.2 * gain)[0, 0]).double()
        img = _render64(case, vol, label, rt, k_inv, sdd)
        go = 2 * (img - views) / img.numel()
        vol.requires_grad_(True)
        _render64(case, vol, label, rt, k_inv, sdd, go=go)
        return {"image": img, "loss": (img - views).square().mean(), "volume": vol.grad[None, None]}
    if kind == "camera" or case.get("grad"):
        go = torch.randn(case["B"], max(1, classes), case["height"], case["width"], device="cuda",
                         generator=_generator(seed + 5)).to(dt).double()
        rt.requires_grad_(True)
        k_inv.requires_grad_(kind == "camera")
        img = _render64(case, vol, label, rt, k_inv, sdd, go=go)
        return {"image": img, "poses": rt.grad, "intrinsics": k_inv.grad}
    return _render64(case, vol, label, rt, k_inv, sdd)
