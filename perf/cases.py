"""Performance cases of the reconstruction path: what a scan's host program has the library do.

A scan runs, in this order: image preparation (camera frames to gray images and thumbnails), the
PatchMatch solve of every view, the geometric pass and the consistency filter, then either TSDF
integration and surface extraction or the dense point cloud, and optionally gradient polishing of
planes, poses and depths.  Every case is one of these stages through its public entry point, over
sizes from a phone preview (160x120) to the largest volume of the benchmark (512^3).  Images are
rendered from the sphere-on-plane scene along the benchmark's helix with its pose and pixel noise;
depth maps are that scene's true depths with 0.2 % noise, holes and matching costs.
"""
from __future__ import annotations

import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "luvas.io-3d_b200"))

from luvas3d import (DTYPE_F16, DTYPE_F32, DTYPE_U8, FORM_EXACT, FORM_FAST, FORM_PLAIN,  # noqa: E402
                     DenseStereo, IntegrationView, SolveOptions, StereoOptions, TsdfVolume, _lib)
from luvas3d import scenes  # noqa: E402
from luvas3d.cloud import FusionView, fuse_depth_maps  # noqa: E402
from luvas3d.grad import integrate_depth, ncc_value_and_grad  # noqa: E402
from luvas3d.image import downsample_rgb, rgba_to_gray, upsample_depth  # noqa: E402
from luvas3d.mesh import extract_surface  # noqa: E402

FORMS = {"plain": FORM_PLAIN, "fast": FORM_FAST, "exact": FORM_EXACT}
STORAGES = {"f32": DTYPE_F32, "f16": DTYPE_F16, "u8": DTYPE_U8}
NEAR, FAR = 0.15, 4.0


def listed():
    return [
        # one keyframe of the preview resolution with the handle's default form: launch latency
        dict(name="solve preview plain", op="solve", form="plain", storage="f32", gather=False,
             views=5, refs=1, width=160, height=120, sources=4, iterations=3, mixed=False,
             geometric=False),
        # one keyframe at scan resolution, solved as the scanner's host solves them: view by view
        dict(name="solve view plain", op="solve", form="plain", storage="f32", gather=False,
             views=9, refs=1, width=640, height=480, sources=8, iterations=5, mixed=False,
             geometric=False),
        # a third of the benchmark's scan in the headline form, all reference views in one batch
        dict(name="solve batch fast f16", op="solve", form="fast", storage="f16", gather=False,
             views=16, refs=16, width=640, height=480, sources=8, iterations=5, mixed=False,
             geometric=False),
        # frames of different cameras, odd sizes, exact bilinear weights (the FP64-accurate form)
        dict(name="solve mixed fast gather", op="solve", form="fast", storage="f32", gather=True,
             views=10, refs=10, width=481, height=359, sources=6, iterations=3, mixed=True,
             geometric=False),
        # photometric solve, geometric pass and consistency filter, bit-exact form
        dict(name="geometric exact", op="solve", form="exact", storage="f32", gather=False,
             views=8, refs=8, width=320, height=240, sources=4, iterations=3, mixed=False,
             geometric=True),
        # fusing filtered maps into the dense cloud, view by view, read back to the host
        dict(name="fuse cloud", op="cloud", views=16, width=640, height=480, sources=8),
        # the benchmark's volume: filtered maps of a scan swept into 512^3
        dict(name="tsdf sweep 512", op="sweep", views=24, width=640, height=480, dim=512, q8=True,
             pool=False, confidence=0.0, one_by_one=False),
        # the reference's own form: f32 weights in a brick pool, one view per call
        dict(name="tsdf views pool", op="sweep", views=8, width=320, height=240, dim=152, q8=False,
             pool=True, confidence=1.2, one_by_one=True),
        # mesh of an integrated volume without its small components, read back to the host
        dict(name="surface 384", op="surface", views=12, width=640, height=480, dim=384, q8=True),
        # one polishing step's gradients: planes and poses of a few reference views
        dict(name="ncc gradients", op="ncc", storage="f32", views=9, refs=3, width=640, height=480,
             sources=4),
        # one depth-polishing step: integrate a view from FP32 depths, gradients back to them
        dict(name="tsdf gradients", op="tsdfgrad", width=640, height=480, dim=256, q8=False),
        # camera frames to gray images, thumbnails and depth priors
        dict(name="frames", op="frames", frames=8, width=1280, height=960, target=640),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["solve", "solve", "solve", "solve", "cloud", "sweep", "sweep", "surface",
                     "ncc", "tsdfgrad", "frames"])
    w = _log(rng, 160, 640)
    h = max(90, int(w * rng.uniform(0.56, 0.78)))
    if op == "solve":
        form = rng.choice(["plain", "fast", "fast", "exact"])
        storage = rng.choice(["f32", "f16", "u8"]) if form == "fast" else "f32"
        # plain and exact cost several times the fast form per pixel, and the geometric pass
        # doubles a solve: fewer views keep every draw under the largest listed case
        most = {"plain": 2, "exact": 4, "fast": 8}[form]
        refs = rng.randint(1, most)
        return dict(op=op, form=form, storage=storage, gather=form == "fast" and rng.random() < 0.5,
                    views=9, refs=refs, width=w, height=h, sources=rng.randint(2, 8),
                    iterations=rng.randint(1, 4), mixed=rng.random() < 0.3,
                    geometric=rng.random() < 0.3)
    if op == "cloud":
        return dict(op=op, views=rng.randint(2, 14), width=w, height=h, sources=rng.randint(2, 8))
    if op == "sweep":
        one = rng.random() < 0.4
        return dict(op=op, views=rng.randint(1, 10 if one else 24), width=w, height=h,
                    dim=_log(rng, 64, 448), q8=rng.random() < 0.5, pool=rng.random() < 0.3,
                    confidence=rng.choice([0.0, 1.2]), one_by_one=one)
    if op == "surface":
        return dict(op=op, views=rng.randint(4, 12), width=w, height=h, dim=_log(rng, 64, 380),
                    q8=rng.random() < 0.5)
    if op == "ncc":
        return dict(op=op, storage=rng.choice(["f32", "f16", "u8"]), views=9, refs=rng.randint(1, 3),
                    width=w, height=h, sources=rng.randint(1, 8))
    if op == "tsdfgrad":
        return dict(op=op, width=w, height=h, dim=_log(rng, 64, 250), q8=rng.random() < 0.5)
    return dict(op=op, frames=rng.randint(1, 8), width=_log(rng, 320, 1920),
                height=_log(rng, 240, 1080), target=rng.randint(100, 300))


# ---- inputs -------------------------------------------------------------------------------------

def _stream():
    """The one stream every handle and torch op of a case runs on."""
    global _the_stream
    try:
        return _the_stream
    except NameError:
        _the_stream = torch.cuda.Stream()
        return _the_stream


def _sizes(c):
    if not c.get("mixed"):
        return [(c["width"], c["height"])] * c["views"]
    # cameras of 1, 3/4, 4/3 and 1/2 of the nominal resolution, in turn
    scale = (1.0, 0.75, 4.0 / 3.0, 0.5)
    return [(max(40, int(c["width"] * scale[i % 4])), max(30, int(c["height"] * scale[i % 4])))
            for i in range(c["views"])]


def _cameras(c, seed, noise=True):
    """(views rendered, views handed to the solver, sizes): consecutive views of the helix."""
    sizes = _sizes(c)
    first = 12 + seed % 8  # from view 12 on the cameras keep 0.4 m or more from the sphere
    true = []
    for i, (w, h) in enumerate(sizes):
        true.append(scenes.helix_views(48, w, h, 560.0 * w / 640.0, turns=1.0)[first + i])
    return true, scenes.perturb(true, seed + 1000, 0.002, 0.1) if noise else true, sizes


def _packed_maps(views, truth, seed):
    """Packed depth maps (int32 torch tensors) of true depths: 0.2 % noise, 3 % holes, normals of
    the sphere or the plane, costs mostly low."""
    gen = torch.Generator(device="cuda").manual_seed(seed + 77)
    out = []
    for v, t in zip(views, truth):
        d = torch.as_tensor(t, device="cuda", dtype=torch.float64)
        h, w = d.shape
        k = v.intrinsics
        y, x = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float64),
                              torch.arange(w, device="cuda", dtype=torch.float64), indexing="ij")
        cam = torch.stack([(x - k.cx) / k.fx * d, (y - k.cy) / k.fy * d, d], -1)
        R = torch.as_tensor(np.asarray(v.pose.R), device="cuda", dtype=torch.float64)
        p = (cam - torch.as_tensor(np.asarray(v.pose.t), device="cuda")) @ R
        n = torch.where((p.norm(dim=-1, keepdim=True) - 1.0).abs() < 0.02, p,
                        torch.tensor([0.0, 1.0, 0.0], device="cuda", dtype=torch.float64))
        n = n @ R.T
        n = n / n.abs().sum(-1, keepdim=True).clamp_min(1e-9)
        ex, ey = n[..., 0], n[..., 1]
        fold = n[..., 2] < 0
        sx, sy = torch.where(ex >= 0, 1.0, -1.0), torch.where(ey >= 0, 1.0, -1.0)
        ex, ey = torch.where(fold, (1 - ey.abs()) * sx, ex), torch.where(fold, (1 - ex.abs()) * sy, ey)
        qx = ((ex * 0.5 + 0.5).clamp(0, 1) * 63 + 0.5).to(torch.int64)
        qy = ((ey * 0.5 + 0.5).clamp(0, 1) * 63 + 0.5).to(torch.int64)
        r = torch.rand((3, h, w), generator=gen, device="cuda")
        noisy = (d * (1 + 0.002 * (r[0] + r[1] - 1))).to(torch.float16).view(torch.int16)
        cost = (r[2] ** 3 * 10).to(torch.int64)
        word = (noisy.to(torch.int64) & 0xffff) | (qx << 16) | (qy << 22) | (cost << 28)
        word = torch.where((d > 0) & (r[1] > 0.03), word, torch.zeros_like(word))
        word = torch.where(word >= 1 << 31, word - (1 << 32), word)
        out.append(word.to(torch.int32).contiguous())
    return out


class _DeviceArray:
    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner  # the handle whose memory it is lives as long as its views
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr=typestr, data=(int(ptr), False),
                                             version=3, strides=None)


def _view(owner, ptr, shape, typestr):
    """A torch tensor over device memory of a library handle (no copy)."""
    return torch.as_tensor(_DeviceArray(owner, ptr, shape, typestr), device="cuda")


def _volume_buffers(volume):
    t, w = C.c_void_p(), C.c_void_p()
    _lib.check(_lib.load().l3d_tsdf_device_buffers(volume._h(), C.byref(t), C.byref(w)))
    n = volume.voxels
    return _view(volume, t.value, (n,), "<f4"), _view(volume, w.value, (n,), "<i2" if volume.weight_q8 else "<f4")


def _filtered_stereo(views, maps, sizes, stream):
    """A stereo handle whose packed and filtered maps are the given ones."""
    w, h = sizes[0]
    s = DenseStereo(w, h, views, StereoOptions(stream=stream), sizes=sizes)
    s.filter_all([0], [[0]], [0])  # allocates the filtered maps
    b = s.buffers()
    flat = torch.cat([m.reshape(-1) for m in maps])
    s.synchronize()
    _view(s, b.depths, (flat.numel(),), "<i4").copy_(flat)
    _view(s, b.filtered_all, (flat.numel(),), "<i4").copy_(flat)
    return s


def _pool_layout(dim, voxel, origin):
    """Brick coordinates of the bricks within the truncation band of the scene's sphere and floor
    (BrickGrid.build's layout)."""
    nb = (dim + 7) // 8
    side, band = voxel * 8, 5 * voxel
    bz, by, bx = np.meshgrid(*[np.arange(nb)] * 3, indexing="ij")
    at = np.stack([bx, by, bz], -1).reshape(-1, 3)
    centre = (at + 0.5) * side + np.asarray(origin)
    reach = band + side * 0.87
    near = (np.abs(np.linalg.norm(centre, axis=-1) - 1.0) < reach) | (np.abs(centre[:, 1] + 1.0) < reach)
    coords = np.zeros((int(near.sum()), 4), dtype=np.int32)
    coords[:, :3] = at[near]
    return coords, None, int(coords.shape[0])


def _volume(c, stream):
    """The benchmark's volume: 2.048 m around the origin, truncation 5 voxels."""
    dim = c["dim"]
    voxel = 2.048 / dim
    origin = (-1.024, -1.024, -1.024)
    if c.get("pool"):
        return TsdfVolume(c["width"], c["height"], voxel, origin, truncation=5 * voxel, weight_q8=c["q8"],
                          layout=_pool_layout(dim, voxel, origin), stream=stream)
    return TsdfVolume(c["width"], c["height"], voxel, origin, truncation=5 * voxel, weight_q8=c["q8"],
                      dense=(dim, dim, dim), stream=stream)


def prepare(c, seed):
    op, stream = c["op"], _stream()
    with torch.cuda.stream(stream):
        s = globals()["_prepare_" + op](c, seed, stream.cuda_stream)
        torch.cuda.current_stream().synchronize()
    s["op"], s["case"] = op, c
    return s


def run(s):
    with torch.cuda.stream(_stream()):
        return globals()["_run_" + s["op"]](s)


# ---- solve ------------------------------------------------------------------------------------

def _images(true, sizes, seed, storage):
    images, _ = scenes.render_sphere(true, sizes, seed, sigma=0.01)
    if storage == "u8":
        return [np.clip(np.rint(im * 255.0), 0, 255).astype(np.uint8) for im in images]
    return images


def _prepare_solve(c, seed, stream):
    true, views, sizes = _cameras(c, seed)
    stereo = DenseStereo(c["width"], c["height"], views,
                         StereoOptions(form=FORMS[c["form"]], storage=STORAGES[c["storage"]], stream=stream),
                         sizes=sizes)
    if c["gather"]:
        stereo.variant = 14 | 16 | 32
    for i, im in enumerate(_images(true, sizes, seed, c["storage"])):
        stereo.set_image(i, im)
    stereo.synchronize()
    src = scenes.neighbour_sources(c["views"], c["sources"], circular=False)
    middle = (c["views"] - c["refs"]) // 2
    refs = list(range(middle, middle + c["refs"]))
    opts = [SolveOptions(src[r], NEAR, FAR, iterations=c["iterations"]) for r in refs]
    geo = [SolveOptions(src[r], NEAR, FAR, iterations=1, geometric=True) for r in refs]
    return dict(stereo=stereo, refs=refs, opts=opts, geo=geo, checks=[src[r] for r in refs])


def _run_solve(s):
    st, refs, c = s["stereo"], s["refs"], s["case"]
    if c["refs"] == 1 and not c["geometric"]:
        st.solve(refs[0], s["opts"][0])
        b = st.buffers()
        h, w = st.shape(refs[0])
        n = sum(x * y for x, y in st.sizes)
        return dict(hyp=_view(st, b.hyp, (h, w, 4), "<f4"), cost=_view(st, b.cost, (h, w), "<f4"),
                    depths=_view(st, b.depths, (n,), "<i4"))
    st.solve_all(refs, s["opts"])
    if c["geometric"]:
        st.solve_all(refs, s["geo"])
        st.filter_all(refs, s["checks"], [1] * len(refs))
    b = st.buffers()
    first = sum(x * y for x, y in st.sizes[:refs[0]])
    n = sum(st.sizes[r][0] * st.sizes[r][1] for r in refs)
    out = dict(hyp=_view(st, b.hyp_all + 16 * first, (n, 4), "<f4"),
               cost=_view(st, b.cost_all + 4 * first, (n,), "<f4"),
               depths=_view(st, b.depths + 4 * first, (n,), "<i4"))
    if c["geometric"]:
        out["filtered"] = _view(st, b.filtered_all + 4 * first, (n,), "<i4")
    return out


def _work_solve(c):
    sizes = _sizes(c)
    middle = (c["views"] - c["refs"]) // 2
    px = sum(w * h for w, h in sizes[middle:middle + c["refs"]])
    texel = {"f32": 4, "f16": 2, "u8": 1}[c["storage"]]
    its = c["iterations"] + (1 if c["geometric"] else 0)
    # a candidate plane: homography, 36 warped bilinear samples and NCC sums per source
    flops = px * (its * 14 + 1) * c["sources"] * (18 + 36 * 37 + 15)
    return dict(bytes=sum(w * h for w, h in sizes) * texel + px * 24 * (2 if c["geometric"] else 1), flops=flops)


# ---- dense cloud --------------------------------------------------------------------------------

def _prepare_cloud(c, seed, stream):
    # the depths are the same for every seed, so that every seed's cloud has as many points; the
    # normals and the colours are the seed's
    true, views, sizes = _cameras(c, 0, noise=False)
    _, truth = scenes.render_sphere(true, sizes, 0)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    maps = [m ^ torch.where(m != 0, torch.randint(0, 16, m.shape, generator=gen, device="cuda",
                                                  dtype=torch.int32) * (1 << 18), torch.zeros_like(m))
            for m in _packed_maps(views, truth, 0)]
    st = _filtered_stereo(views, maps, sizes, stream)
    rng = np.random.default_rng(seed)
    src = scenes.neighbour_sources(c["views"], min(c["sources"], c["views"] - 1), circular=False)
    fv = [FusionView(v, src[i], min(2, len(src[i])), rng.integers(0, 256, (120, 160, 3), dtype=np.uint8))
          for i, v in enumerate(views)]
    return dict(stereo=st, views=fv)


def _run_cloud(s):
    # a budget that most scans stay under: the cell keeps its 4 mm
    cloud, cell = fuse_depth_maps(s["stereo"], s["views"], 0.004, 500000)
    return dict(positions=cloud.positions, normals=cloud.normals, colors=cloud.colors,
                support=cloud.support, cells=cloud.cells, cell=cell)


def _work_cloud(c):
    px = c["views"] * c["width"] * c["height"]
    # maps in (own and each checked source's), nine sums per sample, half a point per pixel out
    return dict(bytes=px * 4 * 2 + px // 8 * 41, flops=px * (60 * c["sources"] + 60))


# ---- TSDF ---------------------------------------------------------------------------------------

def _prepare_sweep(c, seed, stream):
    true, views, sizes = _cameras(c, seed, noise=False)
    _, truth = scenes.render_sphere(true, sizes, seed)
    maps = _packed_maps(views, truth, seed)
    st = _filtered_stereo(views, maps, sizes, stream)
    vol = _volume(c, stream)
    iv = [IntegrationView(v.intrinsics, v.pose, FAR, None, c["confidence"]) for v in views]
    return dict(stereo=st, volume=vol, views=iv)


def _run_sweep(s):
    vol, views = s["volume"], s["views"]
    vol.reset()
    if s["case"]["one_by_one"]:
        for i, v in enumerate(views):
            vol.integrate_layer(v, s["stereo"], i)
    else:
        vol.integrate_many(views, stereo=s["stereo"], layers=list(range(len(views))))
    t, w = _volume_buffers(vol)
    return dict(tsdf=t, weight=w)


def _shell(c):
    """Voxels within the truncation band of the scene's surfaces (sphere and floor)."""
    v = c["dim"] / 2.048
    return min(c["dim"] ** 3, int((4 * math.pi * 0.5 + 2.0) * v * v * 10))


def _work_sweep(c):
    n = c["dim"] ** 3 if not c["pool"] else min(c["dim"] ** 3, 2 * _shell(c))
    per = 6 if c["q8"] else 8
    return dict(bytes=n * per + c["views"] * c["width"] * c["height"] * 4, flops=_shell(c) * c["views"] * 50)


# ---- surface ------------------------------------------------------------------------------------

def _prepare_surface(c, seed, stream):
    # the signs and weights are the same for every seed, so that every seed's mesh has as many
    # triangles; the distances are the seed's
    s = _prepare_sweep(dict(c, pool=False, confidence=0.0), 0, stream)
    s["volume"].integrate_many(s["views"], stereo=s["stereo"], layers=list(range(len(s["views"]))))
    s["volume"].synchronize()
    t, _ = _volume_buffers(s["volume"])
    gen = torch.Generator(device="cuda").manual_seed(seed)
    t.mul_(1 - 0.3 * torch.rand(t.shape, generator=gen, device="cuda"))
    return dict(volume=s["volume"])


def _run_surface(s):
    m = extract_surface(s["volume"], 1.0, components=(0.01, 200))
    return dict(positions=m.positions, normals=m.normals, indices=m.indices)


def _work_surface(c):
    faces = int((4 * math.pi * 0.5 + 2.0) * (c["dim"] / 2.048) ** 2 * 2)
    return dict(bytes=c["dim"] ** 3 * (6 if c["q8"] else 8) + faces * 24, flops=faces * 300)


# ---- gradients ----------------------------------------------------------------------------------

def _prepare_ncc(c, seed, stream):
    true, views, sizes = _cameras(c, seed)
    images, truth = scenes.render_sphere(true, sizes, seed, sigma=0.01)
    if c["storage"] == "u8":
        images = [np.clip(np.rint(im * 255.0), 0, 255).astype(np.uint8) for im in images]
    form = FORM_PLAIN if c["storage"] == "f32" else FORM_FAST
    st = DenseStereo(c["width"], c["height"], views,
                     StereoOptions(form=form, storage=STORAGES[c["storage"]], stream=stream))
    for i, im in enumerate(images):
        st.set_image(i, im)
    st.synchronize()
    src = scenes.neighbour_sources(c["views"], c["sources"], circular=False)
    middle = (c["views"] - c["refs"]) // 2
    refs = list(range(middle, middle + c["refs"]))
    gen = torch.Generator(device="cuda").manual_seed(seed + 5)
    h, w = c["height"], c["width"]
    planes = []
    for r in refs:  # planes near the surface: noisy depths, normals within 20 degrees of the view axis
        d = torch.as_tensor(truth[r], device="cuda")
        d = torch.where(d > 0, d, torch.full_like(d, 2.0))
        n = torch.randn((h, w, 3), generator=gen, device="cuda")
        planes.append(torch.stack([d * (1 + 0.003 * n[..., 0]), 0.2 * n[..., 1], 0.2 * n[..., 2]], -1).contiguous())
    weights = [torch.rand((h, w), generator=gen, device="cuda") for _ in refs]
    deltas = torch.randn((c["views"], 6), generator=gen, device="cuda") * 1e-3
    stored = [im if c["storage"] != "f16" else im.astype(np.float16) for im in images]
    return dict(stereo=st, refs=refs, sources=[src[r] for r in refs], planes=planes, weights=weights,
                deltas=deltas, images=stored, views=views)


def _run_ncc(s):
    gd = torch.zeros((s["case"]["views"], 6), dtype=torch.float64, device="cuda")
    costs, grads = [], []
    for r, src, p, w in zip(s["refs"], s["sources"], s["planes"], s["weights"]):
        cost, gp = ncc_value_and_grad(s["stereo"], r, src, p, s["deltas"], w, gd)
        costs.append(cost)
        grads.append(gp)
    # the planes' three parameters have units of their own; the optimiser takes f32 pose gradients
    g = gd.to(torch.float32)
    return dict(cost=costs, depth=[p[..., 0] for p in grads], angles=[p[..., 1:] for p in grads],
                trans=g[:, :3], rot=g[:, 3:])


def _work_ncc(c):
    px = c["refs"] * c["width"] * c["height"]
    texel = {"f32": 4, "f16": 2, "u8": 1}[c["storage"]]
    return dict(bytes=c["views"] * c["width"] * c["height"] * texel + px * 32,
                flops=px * c["sources"] * 36 * 75)


def _exact_ncc(s):
    """The NCC objective in 64 bits, differentiated by autograd, source by source."""
    c = s["case"]
    f64 = dict(device="cuda", dtype=torch.float64)
    h, w = c["height"], c["width"]
    images = [torch.as_tensor(np.asarray(im), device="cuda").to(torch.float64) / (255.0 if im.dtype == np.uint8 else 1.0)
              for im in s["images"]]
    off = torch.arange(-5, 6, 2, **f64)
    oy, ox = [t.reshape(-1) for t in torch.meshgrid(off, off, indexing="ij")]
    y, x = torch.meshgrid(torch.arange(h, **f64), torch.arange(w, **f64), indexing="ij")
    x, y = x.reshape(-1, 1), y.reshape(-1, 1)

    def pose(i, d):
        v = s["views"][i].pose
        wx, wy, wz = d[i, 3], d[i, 4], d[i, 5]
        z = torch.zeros((), **f64)
        E = torch.matrix_exp(torch.stack([z, -wz, wy, wz, z, -wx, -wy, wx, z]).reshape(3, 3))
        return E @ torch.as_tensor(np.asarray(v.R), **f64), E @ torch.as_tensor(np.asarray(v.t), **f64) + d[i, :3]

    def kmat(i):
        k = s["views"][i].intrinsics
        return torch.tensor([[k.fx, 0, k.cx], [0, k.fy, k.cy], [0, 0, 1]], **f64)

    total = torch.zeros((c["views"], 6), **f64)
    costs, depth, angles = [], [], []
    for r, src, planes, weights in zip(s["refs"], s["sources"], s["planes"], s["weights"]):
        img = images[r]
        vals = img[(y + oy).clamp(0, h - 1).long(), (x + ox).clamp(0, w - 1).long()]
        dc = vals - img.reshape(-1, 1)
        wt = torch.exp(-dc * dc / (2 * 0.06 ** 2) - (ox * ox + oy * oy) / 50.0)
        W = wt.sum(-1)
        rm = (wt * vals).sum(-1) / W
        rv = (wt * (vals - rm[:, None]) ** 2).sum(-1) / W
        cost = torch.zeros(h * w, **f64)
        gp = torch.zeros((h * w, 3), **f64)
        for q in src:
            p = planes.reshape(-1, 3).double().requires_grad_(True)
            d = s["deltas"].double().requires_grad_(True)
            n = torch.stack([torch.sin(p[:, 1]) * torch.cos(p[:, 2]), torch.sin(p[:, 2]),
                             -torch.cos(p[:, 1]) * torch.cos(p[:, 2])], -1)
            m = n @ torch.linalg.inv(kmat(r))
            mu = m[:, 0] * x[:, 0] + m[:, 1] * y[:, 0] + m[:, 2]
            u = m / (p[:, :1] * mu[:, None])
            (Ra, ta), (Rb, tb) = pose(r, d), pose(q, d)
            R = Rb @ Ra.T
            B, kt = kmat(q) @ R @ torch.linalg.inv(kmat(r)), kmat(q) @ (tb - R @ ta)
            H = B + kt[:, None] * u[:, None, :]
            X, Y = x + ox, y + oy
            Q = [H[:, i, 0:1] * X + H[:, i, 1:2] * Y + H[:, i, 2:3] for i in range(3)]
            U, V = Q[0] / Q[2], Q[1] / Q[2]
            ok = ((Q[2] > 1e-6) & (U >= 0) & (V >= 0) & (U <= w - 1) & (V <= h - 1)).all(-1) & \
                (mu < -1e-3) & (p[:, 0] > 0)
            x0, y0 = U.detach().floor().clamp(0, w - 1), V.detach().floor().clamp(0, h - 1)
            fx, fy = U - x0, V - y0
            i0, j0 = x0.long(), y0.long()
            i1, j1 = (i0 + 1).clamp(max=w - 1), (j0 + 1).clamp(max=h - 1)
            im = images[q]
            S = (im[j0, i0] * (1 - fx) + im[j0, i1] * fx) * (1 - fy) + (im[j1, i0] * (1 - fx) + im[j1, i1] * fx) * fy
            S = torch.where(ok[:, None], S, vals)
            sm = (wt * S).sum(-1) / W
            sv = (wt * (S - sm[:, None]) ** 2).sum(-1) / W
            den = torch.sqrt((rv * sv).clamp_min(1e-30))
            cov = (wt * (vals - rm[:, None]) * (S - sm[:, None])).sum(-1) / W
            k = torch.where(den < 1e-5, torch.ones_like(den), (1 - cov / den).clamp(0, 2))
            k = torch.where(ok, k, torch.full_like(k, 2.0))
            g = torch.autograd.grad((weights.reshape(-1).double() * k).sum(), [p, d])
            cost += k.detach()
            gp += g[0]
            total += g[1]
        costs.append(cost.reshape(h, w))
        depth.append(gp[:, 0].reshape(h, w))
        angles.append(gp[:, 1:].reshape(h, w, 2))
    return dict(cost=costs, depth=depth, angles=angles, trans=total[:, :3], rot=total[:, 3:])


def _prepare_tsdfgrad(c, seed, stream):
    cc = dict(c, views=3, pool=False)
    true, views, sizes = _cameras(cc, seed, noise=False)
    _, truth = scenes.render_sphere(true, sizes, seed)
    maps = _packed_maps(views, truth, seed)
    st = _filtered_stereo(views, maps, sizes, stream)
    vol = _volume(cc, stream)
    iv = [IntegrationView(v.intrinsics, v.pose, FAR) for v in views]
    vol.integrate_many(iv[:2], stereo=st, layers=[0, 1])  # the state the third view updates
    vol.synchronize()
    t, w = _volume_buffers(vol)
    depth = (maps[2] & 0xffff).to(torch.int16).view(torch.float16).float().contiguous()
    gen = torch.Generator(device="cuda").manual_seed(seed + 9)
    target = t + 0.1 * torch.randn(t.shape, generator=gen, device="cuda")
    return dict(volume=vol, view=iv[2], packed=maps[2], depth=depth, tsdf=t.clone(), weight=w.clone(),
                target=target)


def _run_tsdfgrad(s):
    d = s["depth"].detach().requires_grad_(True)
    t = s["tsdf"].detach().requires_grad_(True)
    t1, w1 = integrate_depth(s["volume"], s["view"], s["packed"], d, t, s["weight"])
    # the loss gradient a mean-squared residual to a target volume sends back
    gd, gt = torch.autograd.grad(t1, [d, t], grad_outputs=(t1.detach() - s["target"]))
    return dict(tsdf=t1.detach(), weight=w1, depth=gd, state=gt)


def _work_tsdfgrad(c):
    n = c["dim"] ** 3
    w = 2 if c["q8"] else 4
    # forward: state in and out; residual: three; backward: state, gradient in and out
    return dict(bytes=n * ((8 + 2 * w) + 12 + (8 + w + 4)) + c["width"] * c["height"] * 20, flops=n * 40)


# ---- TSDF in 64 bits ----------------------------------------------------------------------------

def _observe(v, packed, z0, z1, c, confidence):
    """One view's observation of the voxel layers [z0, z1): (valid, sdf, weight, pixel), 64 bits."""
    f64 = dict(device="cuda", dtype=torch.float64)
    dim = c["dim"]
    vox = 2.048 / dim
    g = (torch.arange(dim, **f64) + 0.5) * vox - 1.024
    gz = (torch.arange(z0, z1, **f64) + 0.5) * vox - 1.024
    R, t = np.asarray(v.pose.R, dtype=np.float64), np.asarray(v.pose.t, dtype=np.float64)
    cam = [R[i, 0] * g[None, None, :] + R[i, 1] * g[None, :, None] + R[i, 2] * gz[:, None, None] + t[i]
           for i in range(3)]
    k = v.intrinsics
    h, w = packed.shape
    z = cam[2].clamp_min(0.01)
    px, py = torch.round(k.fx * cam[0] / z + k.cx), torch.round(k.fy * cam[1] / z + k.cy)
    ok = (cam[2] > 0.01) & (px >= 0) & (py >= 0) & (px < w) & (py < h)
    pix = torch.where(ok, py * w + px, torch.zeros_like(px)).long()
    word = packed.reshape(-1)[pix]
    d = (word & 0xffff).to(torch.int16).view(torch.float16).double()
    code = (word >> 16) & 4095
    ex, ey = (code & 63).double() / 63 * 2 - 1, (code >> 6).double() / 63 * 2 - 1
    nz = 1 - ex.abs() - ey.abs()
    fold = nz < 0
    nx = torch.where(fold, (1 - ey.abs()) * torch.where(ex >= 0, 1.0, -1.0), ex)
    ny = torch.where(fold, (1 - ex.abs()) * torch.where(ey >= 0, 1.0, -1.0), ey)
    dot = (nx * cam[0] + ny * cam[1] + nz * cam[2]).abs()
    dot = dot / torch.sqrt((nx * nx + ny * ny + nz * nz) * (cam[0] ** 2 + cam[1] ** 2 + cam[2] ** 2))
    wt = dot.clamp_min(0.2)
    if confidence > 0:
        q = 1 - ((word >> 28) & 15).double() / 8
        wt = wt * (q * q).clamp_min(0.15) * (confidence / d.clamp_min(1e-9)).clamp(0.5, 2.0) ** 2
    sdf = d - cam[2]
    return ok & (d > 0) & (sdf >= -5 * vox), sdf, wt, pix


def _step(t, w, ok, sdf, wt, c):
    if c["q8"]:
        wt = torch.round(wt * 256) / 256
    obs = (sdf / (5 * 2.048 / c["dim"])).clamp(max=1.0)
    ok = ok & (wt > 0)
    return (torch.where(ok, (t * w + obs * wt) / (w + wt), t),
            torch.where(ok, (w + wt).clamp(max=96.0), w))


def _exact_sweep(c, seed):
    true, views, sizes = _cameras(c, seed, noise=False)
    _, truth = scenes.render_sphere(true, sizes, seed)
    maps = _packed_maps(views, truth, seed)
    dim = c["dim"]
    ts, ws = [], []
    for z0 in range(0, dim, 64):
        z1 = min(dim, z0 + 64)
        t = torch.ones((z1 - z0, dim, dim), device="cuda", dtype=torch.float64)
        w = torch.zeros_like(t)
        for v, m in zip(views, maps):
            ok, sdf, wt, _ = _observe(v, m, z0, z1, c, c["confidence"])
            t, w = _step(t, w, ok, sdf, wt, c)
        ts.append(t)
        ws.append(w)
    t, w = torch.cat(ts), torch.cat(ws)
    if c["pool"]:  # dense voxels -> brick * 512 + x + 8 y + 64 z
        coords = _pool_layout(dim, 2.048 / dim, (-1.024,) * 3)[0]
        pad = (-dim) % 8
        grow = lambda a: torch.nn.functional.pad(a, (0, pad, 0, pad, 0, pad))  # noqa: E731
        b = torch.as_tensor(coords, device="cuda").long()
        n = (dim + pad) // 8
        cut = lambda a: grow(a).reshape(n, 8, n, 8, n, 8).permute(0, 2, 4, 1, 3, 5)[b[:, 2], b[:, 1], b[:, 0]]  # noqa: E731
        t, w = cut(t), cut(w)
    return dict(tsdf=t.reshape(-1), weight=None if c["q8"] else w.reshape(-1))


def _exact_tsdfgrad(s):
    c = s["case"]
    dim, mu = c["dim"], 5 * 2.048 / c["dim"]
    t = s["tsdf"].double().reshape(dim, dim, dim)
    w = s["weight"].double().reshape(dim, dim, dim) / (256.0 if c["q8"] else 1.0)
    target = s["target"].double().reshape(dim, dim, dim)
    t1, gt = torch.empty_like(t), torch.empty_like(t)
    gd = torch.zeros(s["depth"].numel(), device="cuda", dtype=torch.float64)
    w1 = torch.empty_like(w)
    for z0 in range(0, dim, 64):
        z1 = min(dim, z0 + 64)
        ok, sdf, wt, pix = _observe(s["view"], s["packed"], z0, z1, c, 0.0)
        a, b = _step(t[z0:z1], w[z0:z1], ok, sdf, wt, c)
        t1[z0:z1], w1[z0:z1] = a, b
        if c["q8"]:
            wt = torch.round(wt * 256) / 256
        g = a - target[z0:z1]
        den = torch.where(ok, w[z0:z1] + wt, torch.ones_like(wt))
        gt[z0:z1] = torch.where(ok, g * w[z0:z1] / den, g)
        part = torch.where(ok & (sdf / mu <= 1), g * wt / den / mu, torch.zeros_like(g))
        gd.index_add_(0, pix.reshape(-1), part.reshape(-1))
    return dict(tsdf=t1.reshape(-1), weight=None if c["q8"] else w1.reshape(-1),
                depth=gd.reshape(s["depth"].shape), state=gt.reshape(-1))


# ---- frames -------------------------------------------------------------------------------------

def _prepare_frames(c, seed, stream):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    frames = [torch.randint(0, 256, (c["height"], c["width"], 4), generator=gen, device="cuda",
                            dtype=torch.uint8) for _ in range(c["frames"])]
    grids = []
    for _ in range(c["frames"]):  # a phone's depth grid, a fifth of it empty
        g = torch.rand((90, 160), generator=gen, device="cuda") * 3 + 0.3
        grids.append(torch.where(torch.rand((90, 160), generator=gen, device="cuda") < 0.2,
                                 torch.zeros_like(g), g))
    return dict(frames=frames, grids=grids)


def _run_frames(s):
    c = s["case"]
    w = c["target"]
    h = max(1, round(w * c["height"] / c["width"]))
    out = []
    for f, g in zip(s["frames"], s["grids"]):
        out.append((rgba_to_gray(f, w, h), rgba_to_gray(f, w * 15 // 16, h * 15 // 16),
                    downsample_rgb(f, 160, 120), upsample_depth(g, w, h)))
    return out


def _work_frames(c):
    h = max(1, round(c["target"] * c["height"] / c["width"]))
    px = c["target"] * h
    return dict(bytes=c["frames"] * (c["width"] * c["height"] * 4 + px * 6 + 57600 * 2),
                flops=c["frames"] * c["width"] * c["height"] * 20)


def _exact_frames(s):
    """Bilinear upsampling of the grids that ignores empty cells, in 64 bits (the bytes have no
    other value than their own)."""
    c = s["case"]
    f64 = dict(device="cuda", dtype=torch.float64)
    w = c["target"]
    h = max(1, round(w * c["height"] / c["width"]))
    out = []
    for grid in s["grids"]:
        g = grid.double()
        gh, gw = g.shape
        gy = ((torch.arange(h, **f64) + 0.5) / h * gh - 0.5).clamp(0, gh - 1)
        gx = ((torch.arange(w, **f64) + 0.5) / w * gw - 0.5).clamp(0, gw - 1)
        y0, x0 = gy.floor().long(), gx.floor().long()
        y1, x1 = (y0 + 1).clamp(max=gh - 1), (x0 + 1).clamp(max=gw - 1)
        wy, wx = (gy - y0)[:, None], (gx - x0)[None, :]
        total, weight = torch.zeros((h, w), **f64), torch.zeros((h, w), **f64)
        for yy, a in ((y0, 1 - wy), (y1, wy)):
            for xx, b in ((x0, 1 - wx), (x1, wx)):
                d = g[yy[:, None], xx[None, :]]
                k = torch.where(d > 0, a * b, torch.zeros_like(d))
                total += k * d
                weight += k
        out.append((None, None, None, torch.where(weight > 0.5, total / weight.clamp_min(1e-30), torch.zeros_like(total))))
    return out


# ---- -------------------------------------------------------------------------------------------

def work(c):
    return globals()["_work_" + c["op"]](c)


def exact(c, seed):
    """64-bit values of the outputs that have one.  A PatchMatch solve is a random search that
    every change of rounding sends another way, and the cloud and the mesh are lists whose length
    and order follow from thresholds: those have none."""
    if c["op"] == "sweep":
        return _exact_sweep(c, seed)
    if c["op"] in ("ncc", "tsdfgrad", "frames"):
        return globals()["_exact_" + c["op"]](prepare(c, seed))
    return None
