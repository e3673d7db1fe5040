"""CPU check of the rule by which a warp of the splat raster leaves splats out (compat_splat.cu:strip_masks): over a
rectangle of pixel centres, the least value of the splat's form on the rectangle's edges, less 2e-6 of the form's
size, stays at or below every pixel's own float32 value, however elongated the form is."""
import re
from pathlib import Path

import numpy as np
import pytest

F = np.float32


def strip_least(cx, cy, A, B, C, x0, x1, y0, y1):
    lx, hx, ly, hy = F(x0 - cx), F(x1 - cx), F(y0 - cy), F(y1 - cy)
    if (lx <= 0 <= hx and ly <= 0 <= hy) or not (A > 0 and C > 0):
        return F(0)
    ba, bc = F(-B * F(1 / A)), F(-B * F(1 / C))
    clip = lambda v, lo, hi: F(min(max(v, lo), hi))  # noqa: E731
    yl, yh = clip(F(bc * lx), ly, hy), clip(F(bc * hx), ly, hy)
    xl, xh = clip(F(ba * ly), lx, hx), clip(F(ba * hy), lx, hx)
    form = lambda x, y: F(F(x * F(F(A * x) + F(F(2 * B) * y))) + F(F(C * y) * y))  # noqa: E731
    mx, my = max(abs(lx), abs(hx)), max(abs(ly), abs(hy))
    size = F(F(mx * F(F(A * mx) + F(abs(F(2 * B)) * my))) + F(F(C * my) * my))
    return F(min(form(lx, yl), form(hx, yh), form(xl, ly), form(xh, hy)) - F(2e-6) * size)


@pytest.mark.parametrize("elongation", [1.0, 10.0, 300.0])
def test_least_value_bounds_every_pixel(elongation):
    rng = np.random.default_rng(int(elongation))
    px = F(2.0 / 512)
    for _ in range(1500):
        long_ = np.exp(rng.uniform(np.log(0.002), np.log(1.0)))
        short = max(long_ / elongation, 0.001)
        th = rng.uniform(0, np.pi)
        c, s = np.cos(th), np.sin(th)
        cov = np.array([[c, -s], [s, c]]) @ np.diag([long_ ** 2, short ** 2]) @ np.array([[c, s], [-s, c]])
        inv = np.linalg.inv(cov)
        A, B, C = F(inv[0, 0]), F(inv[0, 1]), F(inv[1, 1])
        cx, cy = F(rng.uniform(-1.2, 1.2)), F(rng.uniform(-1.2, 1.2))
        x0, y0 = F(rng.uniform(-1, 1)), F(rng.uniform(-1, 1))
        xs = (x0 + px * np.arange(8, dtype=F)).astype(F)
        ys = (y0 + px * np.arange(4, dtype=F)).astype(F)
        least = strip_least(cx, cy, A, B, C, xs[0], xs[-1], ys[0], ys[-1])
        dx, dy = (xs - cx).astype(F)[None, :], (ys - cy).astype(F)[:, None]
        spx, spy = A * dx + B * dy, B * dx + C * dy
        q = (dx * spx + dy * spy).astype(F)
        assert q.dtype == F and float(q.min()) >= float(least)


@pytest.mark.parametrize("elongation", [1.0, 10.0, 300.0])
def test_least_value_bounds_every_pixel_of_the_kernels_strip(elongation):
    """The same over the strip of pixels that a warp of the kernel has, its size read from the source."""
    src = (Path(__file__).resolve().parent.parent / "nprush_b200" / "csrc" / "compat_splat.cu").read_text()
    size = int(re.search(r"constexpr uint32_t kStrip = (\d+);", src).group(1))
    assert size * size == 2 * 32  # two pixels per lane
    rng = np.random.default_rng(100 + int(elongation))
    px = F(2.0 / 512)
    outside = 0
    for _ in range(1500):
        long_ = np.exp(rng.uniform(np.log(0.002), np.log(1.0)))
        short = max(long_ / elongation, 0.001)
        th = rng.uniform(0, np.pi)
        c, s = np.cos(th), np.sin(th)
        cov = np.array([[c, -s], [s, c]]) @ np.diag([long_ ** 2, short ** 2]) @ np.array([[c, s], [-s, c]])
        inv = np.linalg.inv(cov)
        A, B, C = F(inv[0, 0]), F(inv[0, 1]), F(inv[1, 1])
        cx, cy = F(rng.uniform(-1.2, 1.2)), F(rng.uniform(-1.2, 1.2))
        x0, y0 = F(rng.uniform(-1, 1)), F(rng.uniform(-1, 1))
        xs = (x0 + px * np.arange(size, dtype=F)).astype(F)
        ys = (y0 + px * np.arange(size, dtype=F)).astype(F)
        least = strip_least(cx, cy, A, B, C, xs[0], xs[-1], ys[0], ys[-1])
        dx, dy = (xs - cx).astype(F)[None, :], (ys - cy).astype(F)[:, None]
        q = (dx * (A * dx + B * dy) + dy * (B * dx + C * dy)).astype(F)
        assert q.dtype == F and float(q.min()) >= float(least)
        outside += least > 0
    assert outside > 1000
