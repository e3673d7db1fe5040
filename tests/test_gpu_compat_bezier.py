"""GPU parity of the reference-semantics Bezier path against the CPU oracle
(oracle/nps_oracle.cpp, pinned bit-exact to the reference's own
bezier_{backward,step,adc}.wgsl by test_oracle_pin.py).

Tolerances: composite 1e-5 absolute; i32 gradient sums (per-pair truncation,
as for splats) bit-exact: the curve kernels use only +, -, *, / and sqrt,
each correctly rounded and unfused (--fmad=false), as the oracle does, and
integer sums do not depend on their order; pixel_loss (per-pixel i32, one term per
pixel) within 1 unit or 1e-4 relative; loss_accum 1e-4 relative (the reference
adds it with a non-atomic read-modify-write, a race; here it is an atomic
float sum); Adam step bit-exact; ADC bit-exact except the clone jitter (sinf).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

import oracle as orc  # noqa: E402
from scenes import bezier_scene, bezier_textures, camera  # noqa: E402


@pytest.fixture(scope="module")
def cls():
    from nprush_b200 import build
    build.build()
    from nprush_b200.bezier import GpuBezierOptimizerManager
    return GpuBezierOptimizerManager


def uni6(mode, max_width, pa, pw, bgp):
    return np.array([mode, max_width, pa, pw, bgp, 0.0], np.float32)


@pytest.mark.parametrize("n,w,h,mode,max_width,bgp,seed", [(96, 48, 32, 1.0, 0.0, 0.0, 7), (400, 64, 64, 1.0, 0.012, 0.3, 8),
                                                        (300, 80, 48, 0.0, 0.0, 0.0, 9), (2600, 32, 32, 1.0, 0.0, 0.0, 10)])
def test_backward_matches_oracle(cls, n, w, h, mode, max_width, bgp, seed):
    b = bezier_scene(n, seed, alive=n - 5)
    vp, vpi = camera(w, h, dist=1.4)
    tgt, depth, bg, bgd, nrm = bezier_textures(w, h, seed + 1)
    m = cls(n, init=b)
    m.write_vp(vp, vpi)
    m.write_mode(mode)
    m.write_max_width(max_width)
    m.write_bg_penalty(bgp)
    la0 = np.full(n, 0.25, np.float32)
    m.write_state(loss_accum=la0)
    m.set_backward_target(tgt, depth, bg, bgd, nrm, w, h)
    img = torch.zeros((1, h, w, 4), device="cuda")
    m.backward(out_rgbd=img)
    st = m.read_state()
    ref = orc.bezier_backward(b, vp, uni6(mode, max_width, 0, 0, bgp), tgt, depth, bg, bgd, nrm,
                              loss_accum=la0.copy())
    np.testing.assert_allclose(img.cpu().numpy()[0], ref["image"], atol=1e-5, rtol=0)
    assert ref["terms"].sum() > 0
    g, r = st["grads"].astype(np.float64), ref["grads_q"].astype(np.float64)
    assert np.abs(r).sum() > 0
    rel = np.linalg.norm(g - r) / np.linalg.norm(r)
    assert rel <= 1e-4, rel
    diff = np.abs(g - r)
    t = ref["terms"].astype(np.float64)[:, None]
    assert (diff == 0).all(), ((diff != 0).mean(), (diff / (t + 1)).max())
    pl, rpl = st["pixel_loss"].astype(np.int64), ref["pixel_loss"].astype(np.int64)
    assert (np.abs(pl - rpl) <= np.maximum(1, 1e-4 * np.abs(rpl))).all()
    np.testing.assert_allclose(st["loss_accum"], ref["loss_accum"], rtol=1e-4, atol=1e-6)
    if n >= 2600:
        assert ref["tile_count"].max() == 1024


@pytest.mark.parametrize("n,w,h,spread,width", [(1, 16, 16, 1.0, (0.01, 0.04)), (23, 17, 15, 0.3, (0.001, 0.003)),
                                                (24, 33, 31, 0.3, (0.2, 0.6)), (25, 16, 48, 8.0, (0.01, 0.04)),
                                                (49, 40, 24, 40.0, (0.05, 0.3)), (1100, 24, 16, 0.2, (0.002, 0.02))])
def test_raster_strip_segments(cls, n, w, h, spread, width):
    """The warp strips' segment lists at their edges: chunks of 24 curves with 1, 23, 24, 25, 49 and the 1024 cap,
    ragged images, hairlines and strokes wider than the image, curves reaching far beyond it, and curves whose
    control points coincide (zero-length segments).  Every sum bit-exact, as the walk over all segments gives it."""
    b = bezier_scene(n, 40 + n, width=width)
    b[:, [0, 1, 4, 5, 8, 9, 12, 13]] *= spread
    b[::7, 4:7] = b[::7, 8:11] = b[::7, 12:15] = b[::7, 0:3]
    vp, vpi = camera(w, h, dist=1.4)
    tgt, depth, bg, bgd, nrm = bezier_textures(w, h, n)
    m = cls(n, init=b)
    m.write_vp(vp, vpi)
    m.write_mode(1.0)
    m.write_max_width(0.012)
    m.set_backward_target(tgt, depth, bg, bgd, nrm, w, h)
    img = torch.zeros((1, h, w, 4), device="cuda")
    m.backward(out_rgbd=img)
    st = m.read_state()
    ref = orc.bezier_backward(b, vp, uni6(1.0, 0.012, 0, 0, 0.0), tgt, depth, bg, bgd, nrm,
                              loss_accum=np.zeros(n, np.float32))
    np.testing.assert_array_equal(img.cpu().numpy()[0], ref["image"])
    np.testing.assert_array_equal(st["grads"], ref["grads_q"])


def test_step_bit_exact(cls):
    n = 500
    rng = np.random.default_rng(9)
    b = bezier_scene(n, 9, alive=480)
    b[3, 19] = 0.0011
    b[4, 3] = 0.0009
    b[5, 0:16:4] = 30.0
    vp, vpi = camera(64, 48)
    g = rng.integers(-200000, 200000, (n, 18), dtype=np.int32)
    m0 = rng.normal(0, 1e-3, (n, 18)).astype(np.float32)
    v0 = np.abs(rng.normal(0, 1e-5, (n, 18))).astype(np.float32)
    ga = (rng.random(n) * 1e-3).astype(np.float32)
    for max_width, no_kill in ((0.0, False), (0.012, True)):
        mg = cls(n, init=b)
        mg.write_vp(vp, vpi)
        mg.write_max_width(max_width)
        mg.write_no_kill(no_kill)
        tgt, depth, bg, bgd, nrm = bezier_textures(64, 48, 3)
        mg.set_backward_target(tgt, depth, bg, bgd, nrm, 64, 48)  # pixel_count = 64 * 48
        mg.write_state(grads=g, adam_m=m0, adam_v=v0, adam_t=3.0, grad_accum=ga)
        mg.step()
        st = mg.read_state()
        rb, rg, rm, rv, ra = b.copy(), g.copy(), m0.copy(), v0.copy(), ga.copy()
        t = orc.bezier_step(rb, rg, rm, rv, 3.0, 64.0 * 48.0, 1.0 if no_kill else 0.0, ra, vp,
                            uni6(1.0, max_width, 0, 0, 0))
        assert st["adam_t"] == t
        np.testing.assert_array_equal(st["beziers"], rb)
        np.testing.assert_array_equal(st["adam_m"], rm)
        np.testing.assert_array_equal(st["adam_v"], rv)
        np.testing.assert_array_equal(st["grad_accum"], ra)
        assert (st["grads"] == 0).all()


@pytest.mark.parametrize("no_kill,n,seed", [(False, 300, 11), (True, 300, 12), (False, 3000, 13)])
def test_adc_matches_oracle(cls, no_kill, n, seed):
    rng = np.random.default_rng(seed)
    b = bezier_scene(n, seed)
    b[rng.random(n) < 0.3, 19] = 0.0
    b[7, 0:16:4] = 40.0
    vp, vpi = camera(256, 256, dist=1.5)
    ga = (rng.random(n) * 0.02).astype(np.float32)
    la = (rng.random(n) * 0.1).astype(np.float32)
    pl = np.zeros(512 * 512, np.int32)
    pl[rng.integers(0, 512 * 512, 3000)] = rng.integers(1, 10000, 3000)
    m0 = rng.normal(0, 1e-3, (n, 18)).astype(np.float32)
    v0 = np.abs(rng.normal(0, 1e-5, (n, 18))).astype(np.float32)
    mg = cls(n, init=b)
    mg.write_vp(vp, vpi)
    mg.write_no_kill(no_kill)
    mg.write_state(adam_m=m0, adam_v=v0, adam_t=77.0, grad_accum=ga, loss_accum=la, pixel_loss=pl)
    mg.adc()
    st = mg.read_state()
    rb, rm, rv, rga, rla, rpl = b.copy(), m0.copy(), v0.copy(), ga.copy(), la.copy(), pl.copy()
    orc.bezier_adc(rb, rm, rv, 77.0, 1.0 if no_kill else 0.0, rga, rla, rpl, vp, vpi)
    np.testing.assert_array_equal(st["adam_m"], rm)
    np.testing.assert_array_equal(st["adam_v"], rv)
    np.testing.assert_array_equal(st["grad_accum"], rga)
    np.testing.assert_array_equal(st["loss_accum"], rla)
    np.testing.assert_array_equal(st["pixel_loss"], rpl)
    # alpha, width, softness and colour are exact, so every kill, clone, split
    # and spawn went to the same slot; control points agree up to the clone
    # jitter (fract(sin(seed * k) * 43758.5453) - 0.5) * 0.001, where CUDA's
    # sinf (2 ulp) and glibc's differ by enough, at these seeds, to wrap fract
    # in about 1% of evaluations: such elements differ by at most 0.001.
    np.testing.assert_array_equal(st["beziers"][:, 16:20], rb[:, 16:20])
    np.testing.assert_array_equal(st["beziers"][:, [3, 7]], rb[:, [3, 7]])
    diff = np.abs(st["beziers"][:, :16] - rb[:, :16])
    off = diff > 2e-5
    assert off.mean() <= 0.02, off.mean()
    assert (diff[off] <= 0.0011).all(), diff.max()
    assert mg.stats()["adc_clones"] + mg.stats()["spawns"] > 0


def test_dispatch_runs_and_learns(cls):
    """Five reference dispatches of a colour-mode layer: the composite error drops."""
    n, w, h = 2000, 96, 96
    from nprush_b200.bezier import reference_init
    b = reference_init(n, 3)
    vp, vpi = camera(w, h, dist=1.5, eye=(0.0, 0.0, 1.5))
    tgt, depth, bg, bgd, nrm = bezier_textures(w, h, 4)
    tgt[..., :3] = 0.8  # a flat target the strokes can match
    m = cls(n, init=b)
    m.write_vp(vp, vpi)
    m.write_mode(1.0)
    m.set_backward_target(tgt, depth, bg, bgd, nrm, w, h)
    img = torch.zeros((1, h, w, 4), device="cuda")
    m.backward(out_rgbd=img)
    e0 = float(np.abs(img.cpu().numpy()[0, ..., :3] - 0.8).mean())
    for _ in range(60):
        m.dispatch()
    m.backward(out_rgbd=img)
    e1 = float(np.abs(img.cpu().numpy()[0, ..., :3] - 0.8).mean())
    assert e1 < e0, (e0, e1)


def test_separate_vp_writes_equal_the_combined_write(cls):
    """writeVPMatrix then writeVPInvMatrix (either order) leaves the same
    uniforms as writing both at once: the dispatched states are bit-identical."""
    n, w, h = 500, 64, 48
    from nprush_b200.bezier import reference_init
    b = reference_init(n, 5)
    vp, vpi = camera(w, h, dist=1.5, eye=(0.3, -0.2, 1.5))
    tgt, depth, bg, bgd, nrm = bezier_textures(w, h, 6)
    states = []
    for order in ("both", "vp_first", "inv_first"):
        m = cls(n, init=b)
        if order == "both":
            m.write_vp(vp, vpi)
        elif order == "vp_first":
            m.writeVPMatrix(vp)
            m.writeVPInvMatrix(vpi)
        else:
            m.write_vp_inv_matrix(vpi)
            m.write_vp_matrix(vp)
        m.write_mode(1.0)
        m.set_backward_target(tgt, depth, bg, bgd, nrm, w, h)
        for _ in range(3):
            m.dispatch()
        states.append(m.read_state())
        m.close()
    for st in states[1:]:
        for k in ("beziers", "adam_m", "adam_v", "grad_accum"):
            np.testing.assert_array_equal(st[k], states[0][k])


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("channel", [16, 18])
def test_colour_that_is_not_finite(cls, channel, value):
    """A curve whose colour is not finite makes every pixel of its tiles NaN or
    infinite, near or far from the curve, as the reference's composite does (T * 0 * inf);
    the pattern equals the oracle's, and so do the gradient sums (a NaN term is 0)."""
    n, w, h = 60, 48, 32
    b = bezier_scene(n, 7)
    b[5, channel] = value
    vp, vpi = camera(w, h, dist=1.4)
    tgt, depth, bg, bgd, nrm = bezier_textures(w, h, 8)
    m = cls(n, init=b)
    m.write_vp(vp, vpi)
    m.write_mode(1.0)
    m.set_backward_target(tgt, depth, bg, bgd, nrm, w, h)
    img = torch.zeros((1, h, w, 4), device="cuda")
    m.backward(out_rgbd=img)
    ref = orc.bezier_backward(b, vp, uni6(1.0, 0.0, 0, 0, 0.0), tgt, depth, bg, bgd, nrm,
                              loss_accum=np.zeros(n, np.float32))
    got = img.cpu().numpy()[0]
    assert np.isnan(ref["image"]).any()
    np.testing.assert_array_equal(np.isnan(got), np.isnan(ref["image"]))
    np.testing.assert_allclose(got, ref["image"], atol=1e-5, rtol=0, equal_nan=True)
    np.testing.assert_array_equal(m.read_state()["grads"], ref["grads_q"])


def test_more_pairs_than_a_sort_takes(cls):
    """Curves that each cover all 2500 tiles of 8 views: 3.6e9 pairs, where a 25%
    margin on the count passes 2^32.  The dispatch reports that they are too many, and
    the handle then composites a small scene as a fresh one does."""
    n, w, h = 180_000, 800, 800
    big = bezier_scene(n, 5, width=(6.0, 7.0))
    vp, vpi = zip(*(camera(w, h, dist=1.4, eye=e) for e in ((1.4, 0.1, 0.2), (-1.4, 0.3, 0.1), (0.1, 0.2, 1.4), (0.2, 0.1, -1.4),
                                                       (1.0, 0.2, 1.0), (-1.0, 0.1, 1.0), (1.0, 0.2, -1.0), (-1.0, 0.3, -1.0))))
    from nprush_b200._lib import NpsError
    tex = [torch.zeros((8, h, w, 4), device="cuda") if k in (0, 2, 4) else torch.ones((8, h, w), device="cuda") for k in range(5)]
    imgs = []
    for first in (big, None):
        m = cls(n, init=first)
        m.write_vp(np.stack(vp), np.stack(vpi))
        m.write_mode(1.0)
        m.set_backward_target(*tex, w, h)
        if first is not None:
            with pytest.raises(NpsError) as e:
                m.backward()
            assert e.value.code == -1  # NPS_ERR_INVALID
        small = bezier_scene(n, 6)
        small[300:, 19] = 0.0
        m.write_params(small)
        img = torch.zeros((8, h, w, 4), device="cuda")
        m.backward(out_rgbd=img)
        imgs.append(img.cpu().numpy())
        m.close()
    np.testing.assert_array_equal(imgs[0], imgs[1])
    assert imgs[0].std() > 0


def test_sort_timeout_is_reported(cls):
    """The tile sort's look-back made to run out (tile 2 of its tiles never
    published, 1000 polls): the backward and the display forward see empty lists, the
    next of each reports NPS_ERR_TIMEOUT, and with the default bound they are those of a
    fresh optimiser again, bit for bit."""
    from nprush_b200._lib import NpsError
    n, w, h = 3000, 128, 96
    b = bezier_scene(n, 35)
    vp, vpi = camera(w, h, dist=1.4)
    tex = bezier_textures(w, h, 36)
    out = []
    for stall in (True, False):
        m = cls(n, init=b)
        m.write_vp(vp, vpi)
        m.write_mode(1.0)
        m.set_backward_target(*tex, w, h)
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
            m.write_state(grads=np.zeros((n, 18), np.int32))
            call()
        m.read_state()  # waits
        out.append((img.cpu().numpy(), shown.cpu().numpy(), m.read_state()["grads"]))
        assert m.stats()["pairs"] > 4096
        m.close()
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
    assert out[1][0].std() > 0 and out[1][1].std() > 0
