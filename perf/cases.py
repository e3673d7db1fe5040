"""The work a user of the library has it do, as cases that can be timed.

Seven kinds of pass, each through the public Python classes over the C ABI:

  gs_step     one step of the 3D Gaussian trainer as `train.fit` runs it (set_views, then one train_step:
              forward over all views, loss, backward, Adam), replayed as one CUDA graph (mode "graph") or
              run eagerly one view at a time (mode "per_view", the plain trainer)
  gs_render   the trainer's forward alone into images, as the PSNR evaluation and a viewer run it
  splat       one dispatch of the reference-semantics splat optimiser (backward, Adam, every 25th ADC)
  bezier      one dispatch of the reference-semantics Bezier optimiser, as one of the viewer's three layers
  path_trace  frames of path-traced targets, with the resolved image
  targets     a viewer frame's target side: mesh pass (colour and depth), depth edges, depth-aware blur,
              separable sRGB blur

Sizes are the repository's own configurations (gradient check, single-view fit, 200k benchmark, 1M / 1080p
scene, the viewer's 512 splats and 256 curves, the 50k-curve fit, the path-tracer and mesh benchmarks) and
odd sizes between them.  Inputs are seeded; optimiser targets come from a seeded teacher of the same kind
(Gaussians, curves) or from smooth seeded images (the viewer's splats).
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from nprush_b200 import _lib, camera, meshes, targets
from nprush_b200.bezier import GpuBezierOptimizerManager
from nprush_b200.gaussians import SH_C0, GaussianTrainer
from nprush_b200.mesh_render import MeshRenderer
from nprush_b200.path_trace import PathTracer
from nprush_b200.splat import GpuSplatOptimizerManager

DEV = "cuda:0"


def _gs(name, n, w, h, views, sh, log_scale, loss="l1_dssim", mode="graph", tuned=False):
    return dict(name=name, kind="gs_step", n=n, w=w, h=h, views=views, sh=sh, log_scale=log_scale, loss=loss,
                mode=mode, tuned=tuned)


def listed():
    return [
        # the smallest fit: the gradient-check scene, one small view, where launches and latency count
        _gs("gs_step_1k_64", 1024, 64, 64, 1, 3, -3.0, loss="l2"),
        # the plain trainer on the single-view-fit scene: eager, one view per launch sequence
        _gs("gs_per_view_16k_256", 16384, 256, 256, 2, 1, -3.5, loss="l1", mode="per_view"),
        # an ordinary small scene, everything odd: count, ragged image, views, SH degree 2, untuned raster
        _gs("gs_step_57k_517x389", 57001, 517, 389, 3, 2, -3.7),
        # the benchmark's training step (200k, SH3, 800 x 800, 8 views) with the raster the autotuner picks for it
        _gs("gs_step_200k_800", 200_000, 800, 800, 8, 3, -4.0, tuned=True),
        # the large scene: 1M Gaussians at 1080p
        _gs("gs_step_1m_1080p", 1_000_000, 1920, 1080, 8, 3, -4.5, tuned=True),
        # images of a trained-size scene, odd size (evaluation, viewer)
        dict(name="gs_render_200k_1237x701", kind="gs_render", n=200_000, w=1237, h=701, views=4, sh=3,
             log_scale=-4.0),
        # the viewer's splat layer: 512 splats of the reference's initial scene, one 512 x 512 view a dispatch
        dict(name="splat_512_512", kind="splat", n=512, w=512, h=512, views=1, scene="viewer"),
        # the reference arm's scene of the benchmark: 200k small splats, 8 views a dispatch
        dict(name="splat_200k_800", kind="splat", n=200_000, w=800, h=800, views=8, scene="cloud"),
        # the viewer's fine colour layer: 256 curves, one view
        dict(name="bezier_256_512", kind="bezier", n=256, w=512, h=512, views=1, layer="color"),
        # the curve fit: 50k random-walk curves, 4 views a dispatch
        dict(name="bezier_50k_512", kind="bezier", n=50_000, w=512, h=512, views=4, layer="fit"),
        # one frame of the path-traced target (12k triangles, 30% mirrors)
        dict(name="path_trace_1024x768", kind="path_trace", w=1024, h=768, objects=16, detail=20, frames=1),
        # the target side of a frame at the mesh benchmark's size (~80k triangles)
        dict(name="targets_1024x768", kind="targets", w=1024, h=768, objects=40, detail=32, radius=4, blur=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gs_step", "gs_step", "gs_step", "gs_render", "splat", "bezier", "path_trace", "targets"])
    if kind in ("gs_step", "gs_render"):
        n = _log_int(rng, 1000, 600_000)
        side = _log_int(rng, 64, 1100)
        w, h = side, max(48, int(side * rng.uniform(0.55, 1.1)))
        views = rng.randint(1, 8)
        sh = rng.choice([0, 1, 2, 3, 3])
        # larger scenes have smaller Gaussians, as in the listed ones
        ls = round(-3.0 - 1.4 * math.log(n / 1000.0) / math.log(1000.0) + rng.uniform(-0.15, 0.15), 3)
        if kind == "gs_render":
            return dict(kind=kind, n=n, w=w, h=h, views=views, sh=sh, log_scale=ls)
        loss = rng.choice(["l1_dssim", "l1_dssim", "l1", "l2"])
        mode = rng.choice(["graph", "graph", "graph", "per_view"])
        return dict(kind=kind, n=n, w=w, h=h, views=views, sh=sh, log_scale=ls, loss=loss, mode=mode,
                    tuned=rng.random() < 0.5)
    if kind == "splat":
        if rng.random() < 0.5:
            side = _log_int(rng, 128, 1024)
            return dict(kind=kind, n=_log_int(rng, 256, 2048), w=side, h=max(64, int(side * rng.uniform(0.5, 1.1))),
                        views=1, scene="viewer")
        side = _log_int(rng, 128, 800)
        return dict(kind=kind, n=_log_int(rng, 4000, 150_000), w=side, h=max(64, int(side * rng.uniform(0.5, 1.0))),
                    views=rng.randint(1, 6), scene="cloud")
    if kind == "bezier":
        side = _log_int(rng, 128, 768)
        h = max(64, int(side * rng.uniform(0.6, 1.0)))
        if rng.random() < 0.5:
            return dict(kind=kind, n=_log_int(rng, 64, 1024), w=side, h=h, views=1,
                        layer=rng.choice(["edge", "base", "color"]))
        return dict(kind=kind, n=_log_int(rng, 2000, 60_000), w=side, h=h, views=rng.randint(1, 4), layer="fit")
    side = _log_int(rng, 160, 1400)
    h = max(96, int(side * rng.uniform(0.5, 1.0)))
    if kind == "path_trace":
        return dict(kind=kind, w=side, h=h, objects=rng.randint(3, 24), detail=rng.randint(6, 24),
                    frames=rng.choice([1, 1, 2, 4]))
    return dict(kind=kind, w=side, h=h, objects=rng.randint(4, 40), detail=rng.randint(8, 32),
                radius=rng.choice([2, 3, 4, 6]), blur=rng.choice([3, 5, 8, 12]))


# ------------------------------------------------------------------ inputs
def _gen(seed, stream):
    g = torch.Generator(device=DEV)
    g.manual_seed(1_000_003 * int(seed) + stream)
    return g


def _gaussians(n, sh, log_scale, g):
    """The repository's random scene (gaussians.random_gaussians' distributions) made on the GPU."""
    p = torch.zeros((n, 64), device=DEV)
    p[:, 0:3] = torch.rand((n, 3), generator=g, device=DEV) * 2 - 1
    p[:, 3:6] = log_scale + 0.5 * torch.randn((n, 3), generator=g, device=DEV)
    q = torch.randn((n, 4), generator=g, device=DEV)
    p[:, 6:10] = q / q.norm(dim=1, keepdim=True)
    p[:, 10] = torch.randn(n, generator=g, device=DEV)
    p[:, 12:15] = (torch.rand((n, 3), generator=g, device=DEV) - 0.5) / SH_C0
    nb = (sh + 1) ** 2
    if nb > 1:
        p[:, 15:12 + 3 * nb] = 0.1 * torch.randn((n, 3 * (nb - 1)), generator=g, device=DEV)
    return p


def _gs_inputs(case, seed):
    """(parameters, targets [V, H, W, 4], vp, vp_inv): a student, and a teacher's images as its targets."""
    w, h, v = case["w"], case["h"], case["views"]
    params = _gaussians(case["n"], case["sh"], case["log_scale"], _gen(seed, 1))
    vp, vpi = camera.sphere_cameras(32, 4.0, math.radians(50.0), w / h)
    pick = np.sort(np.random.default_rng(int(seed)).permutation(32)[:v])
    vp, vpi = vp[pick], vpi[pick]
    tg = None
    if case["kind"] == "gs_step":
        nt = min(case["n"] + case["n"] // 4, 250_000)
        teacher = GaussianTrainer(nt, sh_degree=case["sh"], params=_gaussians(nt, case["sh"], case["log_scale"],
                                                                             _gen(seed, 2)))
        teacher.set_image_size(w, h)
        teacher.set_views(vp, vpi)
        tg = torch.zeros((v, h, w, 4), device=DEV)
        teacher.forward(out=tg)
        teacher.close()
        tg[..., 3] = 1.0
    return params, tg, vp, vpi


def _smooth(g, v, h, w, ch):
    """Seeded smooth images in [0, 1] with some fine detail, [V, H, W, ch]."""
    low = torch.rand((v, ch, max(2, h // 48), max(2, w // 48)), generator=g, device=DEV)
    mid = torch.rand((v, ch, max(2, h // 6), max(2, w // 6)), generator=g, device=DEV)
    up = torch.nn.functional.interpolate
    x = 0.75 * up(low, size=(h, w), mode="bicubic", align_corners=False) + \
        0.25 * up(mid, size=(h, w), mode="bilinear", align_corners=False)
    return x.clamp(0, 1).permute(0, 2, 3, 1).contiguous()


def _viewer_images(g, v, h, w):
    """(rgba, depth, background, background depth, normals): a foreground blob of reciprocal depth before an
    empty background, as the viewer's mesh pass gives them."""
    rgba = torch.ones((v, h, w, 4), device=DEV)
    rgba[..., :3] = _smooth(g, v, h, w, 3)
    mask = _smooth(g, v, h, w, 1)[..., 0] > 0.45
    depth = torch.where(mask, 0.9 + 0.06 * _smooth(g, v, h, w, 1)[..., 0], torch.ones((), device=DEV))
    bg = torch.ones((v, h, w, 4), device=DEV)
    bg[..., :3] = _smooth(g, v, h, w, 3)
    normal = torch.ones((v, h, w, 4), device=DEV)
    normal[..., :3] = _smooth(g, v, h, w, 3)
    return rgba, depth.contiguous(), bg, (0.9 + 0.1 * _smooth(g, v, h, w, 1)[..., 0]).contiguous(), normal


def _splats(case, seed):
    n, g = case["n"], _gen(seed, 1)
    s = torch.zeros((n, 16), device=DEV)
    u = lambda *sh: torch.rand(sh, generator=g, device=DEV)  # noqa: E731
    if case["scene"] == "viewer":  # splat.reference_init's distributions: 512 live splats near the origin
        s[:, 0:3] = (u(n, 3) * 2 - 1) * 0.3
        s[:, 3], s[:, 12], s[:, 15] = 0.1 + 0.15 * u(n), 0.1 + 0.15 * u(n), 0.1 + 0.15 * u(n)
        s[:, 4:7] = u(n, 3)
        live = min(n, 512)
        s[:live, 7] = 0.3 + 0.4 * u(live)
        s[:, 8] = 1.0
    else:  # the benchmark's cloud of small splats
        s[:, 0:3] = u(n, 3) * 2 - 1
        sc = torch.exp(-4.0 + 0.5 * torch.randn((n, 3), generator=g, device=DEV))
        s[:, 3], s[:, 12], s[:, 15] = sc[:, 0], sc[:, 1], sc[:, 2]
        s[:, 4:7] = u(n, 3)
        s[:, 7] = torch.sigmoid(torch.randn(n, generator=g, device=DEV)).clamp(0.06, 0.99)
        q = torch.randn((n, 4), generator=g, device=DEV)
        s[:, 8:12] = q / q.norm(dim=1, keepdim=True)
    s[:, 13], s[:, 14] = 2.0, 0.5
    return s


def _curves(n, layer, h, g):
    b = torch.zeros((n, 20), device=DEV)
    u = lambda *sh: torch.rand(sh, generator=g, device=DEV)  # noqa: E731
    if layer == "fit":  # bezier_fit.random_walk_curves' distributions
        p = u(n, 3) * 2 - 1
        for k in range(4):
            if k:
                p = p + 0.05 * torch.randn((n, 3), generator=g, device=DEV)
            b[:, 4 * k:4 * k + 3] = p
        b[:, 3] = 2.0 * torch.exp(u(n) * math.log(3.0)) / h
        b[:, 7] = 0.5 * b[:, 3]
        b[:, 19] = 0.3 + 0.7 * u(n)
    else:  # bezier.reference_init's: short squiggles near the origin
        c = u(n, 2) * 2 - 1
        ln, ang = 0.2 + 0.2 * u(n), u(n) * 2 * math.pi
        d = torch.stack([torch.cos(ang) * ln, torch.sin(ang) * ln], 1)
        for k, f in enumerate((-0.5, -0.15, 0.15, 0.5)):
            b[:, 4 * k:4 * k + 2] = c + f * d
            if k in (1, 2):
                b[:, 4 * k:4 * k + 2] += (u(n, 2) - 0.5) * 0.08
            b[:, 4 * k + 2] = (u(n) * 2 - 1) * 0.3
        b[:, 3], b[:, 7], b[:, 19] = 0.02, 0.005, 0.5
    b[:, 16:19] = u(n, 3)
    return b


def _sphere_views(seed, v, w, h, radius, fov):
    vp, vpi = camera.sphere_cameras(32, radius, fov, w / h)
    pick = np.sort(np.random.default_rng(int(seed)).permutation(32)[:v])
    return vp[pick], vpi[pick]


class _Buffer:
    """A float32 device buffer of `owner` as a CUDA array interface; a tensor made from it keeps the owner alive."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False), "version": 3}


def _alias(owner, ptr, *shape):
    return torch.as_tensor(_Buffer(owner, ptr, shape), device=DEV)


class State:
    """The handle and buffers a user's program keeps (the handle frees the library's side when it goes)."""

    def __init__(self, case):
        self.case = case
        self.owner = None


def prepare(case, seed):
    s = State(case)
    kind, w, h = case["kind"], case["w"], case["h"]
    if kind in ("gs_step", "gs_render"):
        params, tg, s.vp, s.vpi = _gs_inputs(case, seed)
        n, v = case["n"], case["views"]
        s.owner = t = GaussianTrainer(n, sh_degree=case["sh"], params=params)
        if kind == "gs_render":
            t.set_image_size(w, h)
            s.out = torch.zeros((v, h, w, 4), device=DEV)
        else:
            t.set_targets(tg, borrow=True)
            t.set_loss(case["loss"])
            if case["tuned"]:  # what the autotuner picks (and caches) for such steps
                t.set_raster(fwd=(2, 2, 128), bwd=(2, 2, 128))
            t.set_graph(case["mode"] == "graph")
            b = t.buffers()
            s.grads = _alias(t, b["grads"], n, 64)
            s.params = _alias(t, b["params"], n, 64)
        s.ids = np.arange(v)
    elif kind == "splat":
        n, v = case["n"], case["views"]
        rgba, depth, _, _, _ = _viewer_images(_gen(seed, 3), v, h, w)
        s.owner = m = GpuSplatOptimizerManager(n, init=_splats(case, seed))
        if case["scene"] == "viewer":
            ang = np.random.default_rng(int(seed)).uniform(0, 2 * math.pi)
            vp, vpi = camera.view_proj((1.6 * math.sin(ang), 0.4, 1.6 * math.cos(ang)), (0.0, 0.0, 0.0), math.pi / 3,
                                       w / h)
        else:
            vp, vpi = _sphere_views(seed, v, w, h, 4.0, math.radians(50.0))
        m.write_splat_vp_matrix(vp, vpi)
        m.set_backward_target(rgba, depth, w, h, borrow=True)
        b = m.buffers()
        s.buf = [_alias(m, b[k], n, 16) for k in ("splats", "adam_m", "adam_v")]
    elif kind == "bezier":
        n, v, layer = case["n"], case["views"], case["layer"]
        s.owner = m = GpuBezierOptimizerManager(n, init=_curves(n, layer, h, _gen(seed, 1)))
        if layer == "fit":
            vp, vpi = _sphere_views(seed, v, w, h, 4.0, math.radians(50.0))
            nt = n + n // 5
            teacher = GpuBezierOptimizerManager(nt, init=_curves(nt, layer, h, _gen(seed, 2)))
            s.rgba = torch.zeros((v, h, w, 4), device=DEV)
            for k in range(v):
                teacher.render(vp[k], w, h, s.rgba[k])
            teacher.close()
            s.depth = torch.ones((v, h, w), device=DEV)
            s.bg = s.normal = torch.zeros((v, h, w, 4), device=DEV)
            s.bg_depth = s.depth
            m.write_mode(1.0)
        else:
            vp, vpi = camera.view_proj((0.3, 0.4, 1.6), (0.0, 0.0, 0.0), math.pi / 3, w / h)
            s.rgba, s.depth, s.bg, s.bg_depth, s.normal = _viewer_images(_gen(seed, 3), v, h, w)
            if layer == "edge":
                m.write_mode(0.0)
            else:  # layers.LayeredFit's settings
                m.write_mode(1.0)
                m.write_no_kill(True)
                m.write_kill_thresholds(0.0001, 0.0001)
                if layer == "color":
                    m.write_max_width(0.012)
                else:
                    m.set_adc_period(150)
        m.write_vp(vp, vpi)
        ptrs = [ctypes.c_void_p() for _ in range(7)]
        _lib.call("nps_bezier_opt_buffers", m._h, *[ctypes.byref(p) for p in ptrs])
        s.buf = [_alias(m, ptrs[k].value, n, c) for k, c in ((0, 20), (2, 18), (3, 18))]
    else:
        # another seed is another scene: other objects, other places and colours
        mirrors = 0.3 if kind == "path_trace" else 0.0
        scene = meshes.demo_scene(case["objects"], seed=int(seed), mirror_fraction=mirrors,
                                  sphere_detail=case["detail"])
        env = meshes.sky_env(256, 128)
        eye, at, up = (4.0, -3.5, 2.6), (0.0, 0.0, 0.3), (0.0, 0.0, 1.0)
        vp, inv = camera.view_proj(eye, at, 0.9, w / h, up=up)
        if kind == "path_trace":
            s.owner = pt = PathTracer(env_texture=env)
            pt.set_meshes(scene)
            pt.set_output_size(w, h)
            pt.write_inv_view_proj_mat(inv)
        else:
            s.owner = r = MeshRenderer(scene, matcap=env, env=env)
            r.write_view_proj_mat(vp)
            r.write_view_mat(camera.col_major(camera.look_at(eye, at, up)))
            r.write_inv_view_proj_mat(inv)
            r.write_shading_mode("shaded")
            new = lambda: torch.zeros((h, w, 4), device=DEV)  # noqa: E731
            s.images = {k: new() for k in ("color", "depth", "edge", "bilateral", "temp", "blurred")}
            s.blur = targets.GpuBlurPipelineManager()
            s.bilateral = targets.GpuDepthAwareBlurPipelineManager()
    torch.cuda.synchronize()
    return s


def run(s):
    case = s.case
    kind, w, h = case["kind"], case["w"], case["h"]
    if kind == "gs_step":
        if case["mode"] == "graph":
            s.owner.set_views(s.vp, s.vpi, s.ids)
            s.owner.train_step()
        else:
            s.owner.train_step_per_view(s.vp, s.vpi, s.ids)
        return {"grads": s.grads, "params": s.params}
    if kind == "gs_render":
        s.owner.set_views(s.vp, s.vpi)
        s.owner.forward(out=s.out)
        return {"image": s.out}
    if kind == "splat":
        s.owner.dispatch()
        return {"splats": s.buf[0], "adam_m": s.buf[1], "adam_v": s.buf[2]}
    if kind == "bezier":
        m = s.owner
        m.set_backward_target(s.rgba, s.depth, s.bg, s.bg_depth, s.normal, w, h, borrow=True)
        m.dispatch()
        return {"beziers": s.buf[0], "adam_m": s.buf[1], "adam_v": s.buf[2]}
    if kind == "path_trace":
        s.owner.dispatch(frames=case["frames"])
        return {"accum": s.owner.accum, "image": s.owner.output}
    im = s.images
    s.owner.render(w, h, out=(im["color"], im["depth"]))
    targets.splat_edge(im["depth"], im["edge"], quantize=True)
    s.bilateral.blur(im["color"], im["depth"], im["bilateral"], w, h, case["radius"])
    s.blur.blur(im["color"], im["blurred"], im["temp"], w, h, case["blur"], 4.0, is_srgb=True)
    return {k: im[k] for k in ("color", "depth", "edge", "bilateral", "blurred")}


# ------------------------------------------------------------------ least work
def work(case):
    """Bytes: inputs read once, outputs written once.  Flops: what the method itself needs on the sizes, with the
    scene's typical coverage (a pixel of an opaque scene meets some tens of primitives before it saturates)."""
    kind, px = case["kind"], case["w"] * case["h"]
    if kind in ("gs_step", "gs_render"):
        n, v = case["n"], case["views"]
        nb = 11 + 3 * (case["sh"] + 1) ** 2
        sigma = math.exp(case["log_scale"] + 0.25) * case["h"] / (2 * math.tan(math.radians(25.0))) / 4.0
        per_px = min(n * math.pi * 8.0 * (sigma * sigma + 0.3) / px, 60.0)
        if kind == "gs_render":
            return {"bytes": 4.0 * n * nb + 16.0 * v * px, "flops": v * (px * per_px * 25.0 + n * 300.0)}
        return {"bytes": 4.0 * n * nb * 7 + 16.0 * v * px, "flops": v * (px * (per_px * 75.0 + 900.0) + n * 1200.0)}
    if kind == "splat":
        n, v = case["n"], case["views"]
        per_px = 150.0 if case["scene"] == "cloud" else 300.0
        return {"bytes": 64.0 * n * 6 + 20.0 * v * px, "flops": v * px * min(n, per_px) * 250.0}
    if kind == "bezier":
        n, v = case["n"], case["views"]
        per_px = min(n, 8.0 if case["layer"] != "fit" else 12.0)
        return {"bytes": 76.0 * n * 6 + 56.0 * v * px, "flops": v * px * per_px * 500.0}
    if kind == "path_trace":
        tris = case["objects"] * (2 * case["detail"] ** 2 + 6)
        rays = 2.5 * px * case["frames"]
        return {"bytes": 48.0 * px + 150.0 * tris, "flops": rays * (25.0 * 2 * math.log2(tris + 2) + 4 * 60.0 + 100.0)}
    tris = case["objects"] * (2 * case["detail"] ** 2 + 6)
    return {"bytes": 16.0 * px * 10 + 60.0 * tris,
            "flops": px * (100.0 + (2 * case["radius"] + 1) ** 2 * 20.0 + 2 * (2 * case["blur"] + 1) * 8.0)}


# ------------------------------------------------------------------ 64-bit values
_BLOCK = 32  # pixels; a block's Gaussians are composited densely


def _sh_basis(deg, d):
    x, y, z = d[:, 0], d[:, 1], d[:, 2]
    f = math.sqrt
    pi = math.pi
    b = [torch.full_like(x, 0.5 / f(pi))]
    if deg >= 1:
        c = f(3 / (4 * pi))
        b += [-c * y, c * z, -c * x]
    if deg >= 2:
        c = f(15 / pi) / 2
        b += [c * x * y, -c * y * z, f(5 / pi) / 4 * (2 * z * z - x * x - y * y), -c * x * z, c / 2 * (x * x - y * y)]
    if deg >= 3:
        c3, c2, c1, c0 = f(35 / (2 * pi)) / 4, f(105 / pi) / 2, f(21 / (2 * pi)) / 4, f(7 / pi) / 4
        b += [-c3 * y * (3 * x * x - y * y), c2 * x * y * z, -c1 * y * (4 * z * z - x * x - y * y),
              c0 * z * (2 * z * z - 3 * x * x - 3 * y * y), -c1 * x * (4 * z * z - x * x - y * y),
              c2 / 2 * z * (x * x - y * y), -c3 * x * (x * x - 3 * y * y)]
    return torch.stack(b, 1)


def _project(p, vp, centre, w, h, deg):
    """(u, v, conic a, b, c, opacity, r, g, b) per Gaussian, its box half-extents, depth and whether it shows."""
    m = torch.tensor(np.asarray(vp, np.float64).reshape(4, 4).T.copy(), device=DEV)  # row-major
    mean = p[:, 0:3]
    cx, cy, cw = (mean @ m[r, :3] + m[r, 3] for r in (0, 1, 3))
    u, v = (cx / cw + 1) * (0.5 * w) - 0.5, (1 - cy / cw) * (0.5 * h) - 0.5
    j0 = 0.5 * w * (m[0, :3] * cw[:, None] - cx[:, None] * m[3, :3]) / (cw * cw)[:, None]
    j1 = -0.5 * h * (m[1, :3] * cw[:, None] - cy[:, None] * m[3, :3]) / (cw * cw)[:, None]
    q = p[:, 6:10] / p[:, 6:10].norm(dim=1, keepdim=True)
    qw, x, y, z = q.unbind(1)
    rot = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - qw * z), 2 * (x * z + qw * y),
                       2 * (x * y + qw * z), 1 - 2 * (x * x + z * z), 2 * (y * z - qw * x),
                       2 * (x * z - qw * y), 2 * (y * z + qw * x), 1 - 2 * (x * x + y * y)], 1).view(-1, 3, 3)
    ms = rot * torch.exp(p[:, 3:6])[:, None, :]
    a0, a1 = (j0[:, :, None] * ms).sum(1), (j1[:, :, None] * ms).sum(1)
    A, B, C = (a0 * a0).sum(1) + 0.3, (a0 * a1).sum(1), (a1 * a1).sum(1) + 0.3
    det = A * C - B * B
    op = torch.sigmoid(p[:, 10])
    d = mean - centre
    basis = _sh_basis(deg, d / d.norm(dim=1, keepdim=True))
    nb = (deg + 1) ** 2
    col = (0.5 + (basis[:, :, None] * p[:, 12:12 + 3 * nb].view(-1, nb, 3)).sum(1)).clamp(min=0)
    rec = torch.stack([u, v, C / det, -B / det, A / det, op, col[:, 0], col[:, 1], col[:, 2]], 1)
    with torch.no_grad():
        show = (cw > 0.2) & (det > 0) & (op * 255 > 1)
        t2 = 2 * torch.log((255 * op).clamp(min=1.0)) * 1.01
        ext = torch.stack([torch.sqrt(t2 * A), torch.sqrt(t2 * C)], 1)
    return rec, ext, cw.detach(), show


def _composite(rec, xs, ys):
    """Front-to-back composite of depth-ordered records over the pixels (xs, ys): [pixels, 4] (rgb, T)."""
    dx, dy = rec[:, 0:1] - xs[None, :], rec[:, 1:2] - ys[None, :]
    power = -0.5 * (rec[:, 2:3] * dx * dx + 2 * rec[:, 3:4] * dx * dy + rec[:, 4:5] * dy * dy)
    alpha = (rec[:, 5:6] * torch.exp(power.clamp(max=0))).clamp(max=0.99)
    alpha = torch.where((power <= 0) & (alpha >= 1.0 / 255.0), alpha, torch.zeros((), dtype=alpha.dtype, device=DEV))
    t_in = torch.cumprod(1 - alpha, 0)
    used = t_in.detach() >= 1e-4
    alpha = torch.where(used, alpha, torch.zeros((), dtype=alpha.dtype, device=DEV))
    t_in = torch.cumprod(1 - alpha, 0)
    t_before = torch.cat([torch.ones_like(t_in[:1]), t_in[:-1]], 0)
    rgb = (alpha * t_before).transpose(0, 1) @ rec[:, 6:9]
    return torch.cat([rgb, t_in[-1][:, None]], 1)


def _blocks(rec, ext, depth, show, w, h):
    """(pixel columns, pixel rows, record indices in depth order) of every block that some Gaussian meets."""
    order = torch.argsort(depth.float(), stable=True)
    order = order[show[order]]
    r, e = rec.detach()[order], ext[order]
    x0, x1, y0, y1 = r[:, 0] - e[:, 0], r[:, 0] + e[:, 0], r[:, 1] - e[:, 1], r[:, 1] + e[:, 1]
    for by in range(0, h, _BLOCK):
        rows = (y1 >= by) & (y0 <= min(by + _BLOCK, h) - 1)
        sub = order[rows]
        sx0, sx1 = x0[rows], x1[rows]
        for bx in range(0, w, _BLOCK):
            idx = sub[(sx1 >= bx) & (sx0 <= min(bx + _BLOCK, w) - 1)]
            if idx.numel():
                ys, xs = torch.meshgrid(torch.arange(by, min(by + _BLOCK, h), device=DEV),
                                        torch.arange(bx, min(bx + _BLOCK, w), device=DEV), indexing="ij")
                yield xs.reshape(-1), ys.reshape(-1), idx


def _image_loss(kind, x, y):
    """The trainer's losses over the images [V, H, W, 3]."""
    if kind == "l1":
        return (x - y).abs().mean()
    if kind == "l2":
        return ((x - y) ** 2).mean()
    k = torch.arange(11, dtype=torch.float64, device=DEV) - 5
    g = torch.exp(-k * k / (2 * 1.5 ** 2))
    g = g / g.sum()

    def win(t):
        t = torch.nn.functional.conv2d(t, g.view(1, 1, 1, 11), padding=(0, 5))
        return torch.nn.functional.conv2d(t, g.view(1, 1, 11, 1), padding=(5, 0))

    ssim = 0.0
    for c in range(3):
        a, b = x[..., c][:, None], y[..., c][:, None]
        ma, mb = win(a), win(b)
        saa, sbb, sab = win(a * a) - ma * ma, win(b * b) - mb * mb, win(a * b) - ma * mb
        s = ((2 * ma * mb + 1e-4) * (2 * sab + 9e-4)) / ((ma * ma + mb * mb + 1e-4) * (saa + sbb + 9e-4))
        ssim = ssim + s.mean() / 3
    return 0.8 * (x - y).abs().mean() + 0.2 * (1 - ssim)


def _exact_gs(case, seed):
    w, h, nv = case["w"], case["h"], case["views"]
    params, tg, vp, vpi = _gs_inputs(case, seed)
    p = params.double().requires_grad_(True)
    img = torch.zeros((nv, h, w, 4), dtype=torch.float64, device=DEV)
    img[..., 3] = 1.0
    views = []
    for v in range(nv):
        iv = np.asarray(vpi[v], np.float32).astype(np.float64)
        centre = torch.tensor((iv[8:11] / iv[11]), device=DEV)
        rec, ext, depth, show = _project(p, np.asarray(vp[v], np.float32), centre, w, h, case["sh"])
        det = rec.detach()
        with torch.no_grad():
            blocks = list(_blocks(rec, ext, depth, show, w, h))
            for xs, ys, idx in blocks:
                img[v, ys, xs] = _composite(det[idx], xs.double(), ys.double())
        views.append((rec, blocks))
    if case["kind"] == "gs_render":
        return {"image": img}
    x = img[..., :3].clone().requires_grad_(True)
    (dx,) = torch.autograd.grad(_image_loss(case["loss"], x, tg[..., :3].double()), x)
    recs, grecs = [], []
    for v, (rec, blocks) in enumerate(views):
        det, grec = rec.detach(), torch.zeros_like(rec)
        for xs, ys, idx in blocks:
            sub = det[idx].requires_grad_(True)
            out = _composite(sub, xs.double(), ys.double())
            (gs,) = torch.autograd.grad((out[:, :3] * dx[v, ys, xs]).sum(), sub)
            grec.index_add_(0, idx, gs)
        recs.append(rec)
        grecs.append(grec)
    (g,) = torch.autograd.grad(recs, p, grecs)
    # the first Adam step of zero moments: both bias corrections cancel, m_hat = g and v_hat = g g
    lr = torch.zeros(64, dtype=torch.float64, device=DEV)
    for sl, val in zip((slice(0, 3), slice(3, 6), slice(6, 10), slice(10, 11), slice(12, 15), slice(15, 60)),
                       GaussianTrainer.LR_DEFAULT):
        lr[sl] = val
    new = p.detach() - lr * g / (g.abs() + 1e-15)
    return {"grads": g, "params": new}


def exact(case, seed):
    """64-bit values of the Gaussian cases (plain torch, dense blocks).  The optimisers of the reference are defined
    by their fixed-point sums and the path tracer by its float32 random walk: those have no such value."""
    if case["kind"] not in ("gs_step", "gs_render"):
        return None
    blocks = case["views"] * -(-case["w"] // _BLOCK) * -(-case["h"] // _BLOCK)
    if blocks > 6000 or case["n"] * case["views"] > 1_700_000:
        return None  # over about 20 seconds
    return _exact_gs(case, seed)
