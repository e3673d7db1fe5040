"""GPU parity of the reference-semantics splat path (libnprush_cuda) against
the CPU oracle (oracle/nps_oracle.cpp, itself pinned bit-exact to the
reference's shaders by test_oracle_pin.py).

Tolerances:
  forward composite (r, g, b, reciprocal depth): 1e-5 absolute per channel;
  gradients: the reference's own i32 fixed-point sums.  Every (pixel, splat)
    term is truncated separately; the kernel evaluates pow / exp / log on the
    special-function unit (WGSL's own accuracy for them), so a term may land
    one unit off across an integer boundary.  Checked per element against the
    number of terms it sums (the oracle counts them):
    |diff| <= 2 * terms + 1e-5 * |ref| + 1, relative L2 error <= 1e-4 over
    all gradients, and most elements exactly equal;
  Adam step: bit-exact (no transcendental on the device path);
  ADC: bit-exact except the clone jitter, which goes through sinf (5e-6).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

import oracle as orc  # noqa: E402
from scenes import camera, splat_scene, targets  # noqa: E402


@pytest.fixture(scope="module")
def mgr_cls():
    from nprush_b200 import build
    build.build()
    from nprush_b200.splat import GpuSplatOptimizerManager
    return GpuSplatOptimizerManager


def run_backward(cls, s, vps, vpis, tgts, depths):
    n = s.shape[0]
    v = len(vps)
    h, w = depths[0].shape
    m = cls(n, init=s)
    m.write_splat_vp_matrix(np.stack(vps), np.stack(vpis))
    m.set_backward_target(np.stack(tgts), np.stack(depths), w, h)
    img = torch.zeros((v, h, w, 4), device="cuda", dtype=torch.float32)
    m.backward(out_rgbd=img)
    st = m.read_state()
    return st["grads"], img.cpu().numpy(), m


def grad_close(g, ref, terms):
    """(relative L2 error, every element within 2 units per summed term,
    largest |diff| / (terms + 1), fraction of elements exactly equal)."""
    diff = np.abs(g.astype(np.int64) - ref.astype(np.int64))
    rel = np.linalg.norm(diff) / max(np.linalg.norm(ref.astype(np.float64)), 1.0)
    t = terms.astype(np.float64)[:, None]
    bound = 2 * t + 1e-5 * np.abs(ref) + 1
    return rel, bool((diff <= bound).all()), float((diff / (t + 1)).max()), float((diff == 0).mean())


@pytest.mark.parametrize("n,w,h,seed,shape", [(64, 32, 32, 0, False), (300, 48, 40, 1, True),
                                              (1100, 64, 48, 2, False), (4000, 128, 96, 3, False)])
def test_backward_matches_oracle(mgr_cls, n, w, h, seed, shape):
    s = splat_scene(n, seed, alive=n - 9, random_shape=shape)
    vp, vpi = camera(w, h)
    tgt, depth = targets(w, h, seed + 100)
    ref = orc.splat_backward(s, vp, vpi, tgt, depth)
    g, img, m = run_backward(mgr_cls, s, [vp], [vpi], [tgt], [depth])
    np.testing.assert_allclose(img[0], ref["image"], atol=1e-5, rtol=0)
    rel, ok, worst, exact = grad_close(g, ref["grads_q"], ref["terms"])
    print(f"n={n}: rel {rel:.2e}, worst |diff|/terms {worst:.3f}, exact {exact:.4f}")
    assert rel <= 1e-4, (rel, worst)
    assert ok, worst
    assert exact >= 0.5, exact
    assert m.stats()["pairs"] > 0


@pytest.mark.parametrize("n,w,h,shape", [(31, 16, 16, (0.1, 0.3)), (32, 17, 33, (2.0, 0.5)), (33, 40, 24, (8.0, 4.0)),
                                         (97, 64, 16, (1.0, 0.01))])
def test_strip_masks(mgr_cls, n, w, h, shape):
    """The warp strips' masks at their edges: splats much smaller and much larger than a strip, five to one
    elongated, shapes from a near-constant to a near-box falloff, opacities around the 0.001 cut, chunks of 32 splats
    one short, full and one over, ragged images.

    Tolerances: the pixel's form is evaluated fused on the device and unfused by the oracle, a relative error of at
    most 4 * 2^-24 * 25 = 6e-6 (25: the square of the elongation), which the exponent's derivative (a x e^-x / 2 <= 2)
    and the sums over the pairs of a pixel turn into at most 1e-4 of the composite and 1e-3 of the gradients."""
    rng = np.random.default_rng(n)
    s = splat_scene(n, 60 + n, spread=0.5)
    base = np.exp(rng.uniform(np.log(0.002), np.log(0.5), n))
    for k in (3, 12, 15):
        s[:, k] = base * np.exp(rng.uniform(-0.8, 0.8, n))
    s[:, 13], s[:, 14] = shape
    s[:, 7] = np.exp(rng.uniform(np.log(0.006), np.log(0.99), n))
    vp, vpi = camera(w, h)
    tgt, depth = targets(w, h, 70 + n)
    ref = orc.splat_backward(s, vp, vpi, tgt, depth)
    g, img, _ = run_backward(mgr_cls, s, [vp], [vpi], [tgt], [depth])
    np.testing.assert_allclose(img[0], ref["image"], atol=1e-4, rtol=0)
    diff = np.abs(g.astype(np.int64) - ref["grads_q"].astype(np.int64))
    assert (diff <= 2 * ref["terms"].astype(np.float64)[:, None] + 1e-3 * np.abs(ref["grads_q"]) + 1).all()
    assert np.linalg.norm(diff) <= 1e-3 * np.linalg.norm(ref["grads_q"].astype(np.float64))


def test_multi_view_sums_views(mgr_cls):
    n, w, h = 500, 48, 48
    s = splat_scene(n, 21)
    cams = [camera(w, h, eye=e) for e in ((0.3, 0.4, 1.6), (-1.2, 0.2, 1.0), (0.5, -1.4, 0.6))]
    tg = [targets(w, h, 30 + k) for k in range(3)]
    ref = np.zeros((n, 16), np.int32)
    terms = np.zeros(n, np.uint32)
    imgs = []
    for (vp, vpi), (t, d) in zip(cams, tg):
        r = orc.splat_backward(s, vp, vpi, t, d, grads_q=ref, terms=terms)
        imgs.append(r["image"])
    g, img, _ = run_backward(mgr_cls, s, [c[0] for c in cams], [c[1] for c in cams], [t for t, _ in tg],
                             [d for _, d in tg])
    for k in range(3):
        np.testing.assert_allclose(img[k], imgs[k], atol=1e-5, rtol=0)
    rel, ok, worst, exact = grad_close(g, ref, terms)
    assert rel <= 1e-4 and ok and exact >= 0.5, (rel, worst, exact)


def test_empty_and_all_dead(mgr_cls):
    n, w, h = 100, 40, 24
    s = splat_scene(n, 5)
    s[:, 7] = 0.0  # all culled: pure background
    vp, vpi = camera(w, h)
    tgt, depth = targets(w, h, 6)
    ref = orc.splat_backward(s, vp, vpi, tgt, depth)
    g, img, _ = run_backward(mgr_cls, s, [vp], [vpi], [tgt], [depth])
    np.testing.assert_allclose(img[0], ref["image"], atol=1e-6, rtol=0)
    assert (g == 0).all() and (ref["grads_q"] == 0).all()


def test_tile_cap_1024(mgr_cls):
    n = 1500
    s = splat_scene(n, 5, spread=0.02, scale=(0.002, 0.004))
    vp, vpi = camera(32, 32, dist=1.2, eye=(0, 0, 1.2))
    tgt, depth = targets(32, 32, 6)
    ref = orc.splat_backward(s, vp, vpi, tgt, depth)
    assert ref["tile_count"].max() == 1024
    g, img, m = run_backward(mgr_cls, s, [vp], [vpi], [tgt], [depth])
    np.testing.assert_allclose(img[0], ref["image"], atol=1e-5, rtol=0)
    # pairs composited after the cap = the oracle's capped list lengths; the longest list reaches the cap
    st = m.stats()
    assert st["pairs_capped"] == int(ref["tile_count"].sum()), (st, int(ref["tile_count"].sum()))
    assert st["max_tile_len"] >= 1024 and st["pairs_capped"] <= st["pairs"], st
    m.close()
    # splats beyond the cap get no gradient on either side
    beyond = np.arange(n) >= 1100
    assert (g[beyond] == ref["grads_q"][beyond]).all()
    rel, ok, worst, exact = grad_close(g, ref["grads_q"], ref["terms"])
    print(f"cap: rel {rel:.2e}, worst |diff|/terms {worst:.3f}, exact {exact:.4f}")
    assert rel <= 1e-4 and ok, (rel, worst, exact)


def test_dense_scene_cap_aware_binning(mgr_cls):
    """20k splats crowding a 64 x 64 view: most tile lists run past the 1024
    cap, so the binning keeps only the splat blocks a tile's first 1024
    entries need, and most pixels' transmittance reaches exactly 0 (the
    kernel's exact skips).  Image, gradients and list statistics against the
    oracle."""
    n, w, h = 20000, 64, 64
    s = splat_scene(n, 17, spread=0.25, scale=(0.04, 0.1))
    vp, vpi = camera(w, h)
    tgt, depth = targets(w, h, 18)
    ref = orc.splat_backward(s, vp, vpi, tgt, depth)
    assert ref["tile_count"].min() == 1024
    g, img, m = run_backward(mgr_cls, s, [vp], [vpi], [tgt], [depth])
    np.testing.assert_allclose(img[0], ref["image"], atol=1e-5, rtol=0)
    rel, ok, worst, exact = grad_close(g, ref["grads_q"], ref["terms"])
    print(f"dense: rel {rel:.2e}, worst |diff|/terms {worst:.3f}, exact {exact:.4f}")
    assert rel <= 1e-4 and ok, (rel, worst, exact)
    st = m.stats()
    assert st["pairs_capped"] == int(ref["tile_count"].sum()), st
    # the cut removed most overlapped pairs, yet kept every tile's first 1024
    assert st["pairs_capped"] <= st["pairs_kept"] < st["pairs"] // 2, st
    assert st["max_tile_len"] > 1024 and st["timeouts"] == 0, st
    m.close()


def test_raster_staging_timeout_is_reported(mgr_cls):
    """A staging wait that runs out (tile 0's first batch never issued, 1000
    polls): the raster's CTA for that tile stops and releases nothing in
    flight, the next backward reports NPS_ERR_TIMEOUT, and with the default
    bound the optimiser then matches the oracle again."""
    from nprush_b200._lib import NpsError
    n, w, h = 600, 48, 32
    s = splat_scene(n, 31)
    vp, vpi = camera(w, h)
    tgt, depth = targets(w, h, 32)
    ref = orc.splat_backward(s, vp, vpi, tgt, depth)
    assert ref["tile_count"][0, 0] > 32  # tile 0 stages more than one batch
    m = mgr_cls(n, init=s)
    m.write_splat_vp_matrix(vp, vpi)
    m.set_backward_target(tgt, depth, w, h)
    m.set_wait_guard(1000, 0)
    m.backward()
    m.sync()
    with pytest.raises(NpsError) as e:
        m.backward()
    assert e.value.code == -5  # NPS_ERR_TIMEOUT
    assert m.stats()["timeouts"] > 0
    m.set_wait_guard()
    m.write_state(grads=np.zeros((n, 16), np.int32))
    img = torch.zeros((1, h, w, 4), device="cuda")
    m.backward(out_rgbd=img)
    st = m.read_state()
    np.testing.assert_allclose(img.cpu().numpy()[0], ref["image"], atol=1e-5, rtol=0)
    rel, ok, worst, exact = grad_close(st["grads"], ref["grads_q"], ref["terms"])
    assert rel <= 1e-4 and ok, (rel, worst, exact)
    m.close()


def test_step_bit_exact(mgr_cls):
    n = 3000
    rng = np.random.default_rng(3)
    s = splat_scene(n, 3, alive=2900)
    s[5, 7] = 0.051
    s[6, 3] = 0.0012; s[6, 12] = 0.0012; s[6, 15] = 0.001
    g = rng.integers(-200000, 200000, (n, 16), dtype=np.int32)
    m0 = rng.normal(0, 1e-3, (n, 16)).astype(np.float32)
    v0 = np.abs(rng.normal(0, 1e-5, (n, 16))).astype(np.float32)
    ga = (rng.random(n) * 1e-3).astype(np.float32)
    mg = mgr_cls(n, init=s)
    mg.write_state(m0, v0, 7.0, ga, grads=g)
    mg.step()
    st = mg.read_state()
    rs, rg, rm, rv, rga = s.copy(), g.copy(), m0.copy(), v0.copy(), ga.copy()
    t = orc.splat_step(rs, rg, rm, rv, 7.0, rga)
    assert st["adam_t"] == t
    np.testing.assert_array_equal(st["splats"], rs)
    np.testing.assert_array_equal(st["adam_m"], rm)
    np.testing.assert_array_equal(st["adam_v"], rv)
    np.testing.assert_array_equal(st["grad_accum"], rga)
    assert (st["grads"] == 0).all()


@pytest.mark.parametrize("n,seed", [(256, 4), (5000, 8)])
def test_adc_matches_oracle(mgr_cls, n, seed):
    rng = np.random.default_rng(seed)
    s = splat_scene(n, seed)
    dead = rng.random(n) < 0.35
    s[dead, 7] = 0.0
    s[::7, 3] = 0.002; s[::7, 12] = 0.002; s[::7, 15] = 0.002
    ga = (rng.random(n) * 4e-3).astype(np.float32)
    m0 = rng.normal(0, 1e-3, (n, 16)).astype(np.float32)
    v0 = np.abs(rng.normal(0, 1e-5, (n, 16))).astype(np.float32)
    mg = mgr_cls(n, init=s)
    mg.write_state(m0, v0, 50.0, ga)
    mg.adc()
    st = mg.read_state()
    rs, rm, rv, rga = s.copy(), m0.copy(), v0.copy(), ga.copy()
    orc.splat_adc(rs, rm, rv, 50.0, rga)
    np.testing.assert_array_equal(st["adam_m"], rm)
    np.testing.assert_array_equal(st["adam_v"], rv)
    np.testing.assert_array_equal(st["grad_accum"], rga)
    np.testing.assert_array_equal(st["splats"][:, 2:], rs[:, 2:])
    # clone jitter (fract(sin(seed * k) * 43758.5453) - 0.5) * 0.002: a 1-ulp
    # sinf difference moves the product by ~4e-3 at these seeds; where that
    # crosses an integer, fract wraps and the jitter flips by up to 0.002.
    diff = np.abs(st["splats"][:, :2] - rs[:, :2])
    off = diff > 1e-5
    clones = mg.stats()["adc_clones"]
    assert clones > 0
    assert off.sum() <= max(2, clones // 200), off.sum()
    assert (diff[off] <= 0.00201).all()


def test_dispatch_tracks_oracle(mgr_cls):
    """26 reference dispatches (backward, step, ADC at call 25) on a small scene:
    the trajectories stay together (fixed-point grads amplify ulp-level
    differences only through Adam's normalisation)."""
    n, w, h = 600, 48, 48
    s = splat_scene(n, 12, alive=450)
    vp, vpi = camera(w, h)
    tgt, depth = targets(w, h, 13)
    mg = mgr_cls(n, init=s)
    mg.write_splat_vp_matrix(vp, vpi)
    mg.set_backward_target(tgt, depth, w, h)
    rs = s.copy()
    rg = np.zeros((n, 16), np.int32)
    rm = np.zeros((n, 16), np.float32)
    rv = np.zeros((n, 16), np.float32)
    rga = np.zeros(n, np.float32)
    t = 0.0
    for k in range(26):
        mg.dispatch()
        orc.splat_backward(rs, vp, vpi, tgt, depth, grads_q=rg, want_float=False, want_image=False)
        t = orc.splat_step(rs, rg, rm, rv, t, rga)
        if (k + 1) % 25 == 0:
            orc.splat_adc(rs, rm, rv, t, rga)
    st = mg.read_state()
    assert st["adam_t"] == t
    live_ref = rs[:, 7] > 0
    live_gpu = st["splats"][:, 7] > 0
    assert (live_ref != live_gpu).sum() <= 3
    both = live_ref & live_gpu
    assert np.abs(st["splats"][both] - rs[both]).max() < 0.05


def test_edge_target_and_dispatch_edge(mgr_cls):
    """setEdgeTarget + dispatchEdge: the splat edge pass over the bound depth
    image into an rgba8unorm-like edge image equals the reference shader's
    output (tests/golden/preprocess.npz) at 8-bit levels; no target, or a
    dispatch that does not cover the image, raises."""
    from pathlib import Path

    from nprush_b200._lib import NpsError
    d = np.load(Path(__file__).resolve().parent / "golden" / "preprocess.npz")
    z = torch.from_numpy(d["depth"]).cuda()
    h, w = z.shape[:2]
    m = mgr_cls(64)
    with pytest.raises(NpsError):
        m.dispatch_edge(w, h)
    out = torch.zeros_like(z)
    m.setEdgeTarget(z, out)
    with pytest.raises(ValueError):
        m.dispatch_edge(w - 16, h)
    m.dispatchEdge(w, h)
    got = out.cpu().numpy()
    raw = np.clip(d["edge"], 0, 1) * 255
    on_edge = np.abs(raw - np.floor(raw) - 0.5) < 1e-5 * 255
    assert np.all((got == np.rint(raw) / 255) | on_edge)
    m.close()


@pytest.mark.parametrize("w,h,seed", [(33, 47, 5), (64, 50, 6), (16, 16, 7)])
def test_saturated_terms_wrap(mgr_cls, w, h, seed):
    """Targets of -1e8 and 1e8: every term of those colours' gradients saturates, and
    their i32 sums (an odd number of terms, down to pairs of pixels) wrap as the shader's
    atomicAdd does, exactly."""
    s = splat_scene(1, seed, spread=0.1)
    s[:, 7] = 0.9
    s[:, [3, 12, 15]] = 0.3
    vp, vpi = camera(w, h)
    tgt, depth = targets(w, h, seed)
    tgt[..., 0], tgt[..., 1] = -1e8, 1e8
    ref = orc.splat_backward(s, vp, vpi, tgt, depth)
    g, _, _ = run_backward(mgr_cls, s, [vp], [vpi], [tgt], [depth])
    n = int(ref["terms"][0])
    wrap = lambda t: (t * n + 2 ** 31) % 2 ** 32 - 2 ** 31  # noqa: E731
    assert ref["grads_q"][0, 4:6].tolist() == [wrap(2147483520), wrap(-2 ** 31)]
    np.testing.assert_array_equal(g[0, 4:6], ref["grads_q"][0, 4:6])


def test_sort_timeout_is_reported(mgr_cls):
    """The tile sort's look-back made to run out (tile 2 of its tiles never
    published, 1000 polls): the backward and the display forward see empty lists, the
    next of each reports NPS_ERR_TIMEOUT, and with the default bound they are those of a
    fresh optimiser again, bit for bit."""
    from nprush_b200._lib import NpsError
    n, w, h = 4000, 128, 96
    s = splat_scene(n, 33)
    vp, vpi = camera(w, h)
    tgt, depth = targets(w, h, 34)
    out = []
    for stall in (True, False):
        m = mgr_cls(n, init=s)
        m.write_splat_vp_matrix(vp, vpi)
        m.set_backward_target(tgt, depth, w, h)
        img = torch.zeros((1, h, w, 4), device="cuda")
        shown = torch.zeros((h, w, 4), device="cuda")
        for call in (lambda: m.backward(out_rgbd=img), lambda: m.render(vp, w, h, shown)):
            if stall:
                m.set_sort_guard(1000, 2)
                call()
                with pytest.raises(NpsError) as e:
                    call()
                assert e.value.code == -5  # NPS_ERR_TIMEOUT
                m.set_sort_guard()
            m.write_state(grads=np.zeros((n, 16), np.int32))
            call()
            m.sync()
        out.append((img.cpu().numpy(), shown.cpu().numpy(), m.read_state()["grads"]))
        assert m.stats()["pairs"] > 4096
        m.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    assert out[1][0].std() > 0 and out[1][1].std() > 0
