"""The tile lists a step builds hold only the tiles a splat can reach
(splat_footprint and row_columns in raster_common.cuh): the tiles of the
reference's 3-sigma square, less those where no pixel centre lies in the ellipse
of powers at or above the alpha floor. Leaving out a tile where a pixel does take
the splat would change the image.

On the CPU the formulas, restated in float32, are held against every pixel centre
of random conics: any pixel whose float32 alpha reaches the floor has to lie in
the columns kept for its row. On the GPU images of clouds that stress the cut
(needles, specks, opacities at the floor, splats larger than the image, other
floors, none) are held against the oracle's, which walks the reference's whole
lists."""
from __future__ import annotations

import numpy as np
import pytest

import oracle_lib as O
import parallax_b200 as px
from parallax_b200._abi import RasterOptions

F = np.float32


def footprint(co, opacity, min_alpha):
    a, b, c = co
    floor = F(np.log(F(min_alpha) / F(opacity))) - F(1e-5)
    det = F(a * c) - F(b * b)
    mild = F(a * c) < F(10) * det
    k = F(-2) * floor
    if mild:
        k = k * F(1.0001) + F(1e-4)
    widen, pad = (F(1.0001), F(0.02)) if mild else (F(1.1), F(0.5))
    with np.errstate(all="ignore"):
        ex = np.sqrt(k * c / det) * widen + pad
        ey = np.sqrt(k * a / det) * widen + pad
    return k, ex, ey, pad, mild, not (det > 0) or not (ex < 1e4 and ey < 1e4), det


def tiles(lo, hi):
    return int(np.ceil((lo - F(15.5)) / F(16))), int(np.floor((hi - F(0.5)) / F(16)))


def row_columns(co, mean, fp, row, x0, x1):
    k, ex, ey, pad, mild, bounds_nothing, det = fp
    if bounds_nothing or not mild:
        return x0, x1
    a, b, c = co
    lo = F(row * 16) + (F(0.5) - F(0.02)) - mean[1]
    hi = lo + F(15) + F(0.04)
    end = -b / c * np.sqrt(k * c / det)
    yr, yl = min(max(end, lo), hi), min(max(-end, lo), hi)
    right = (np.sqrt(max(a * k - det * yr * yr, F(0))) - b * yr) / a
    left = -(np.sqrt(max(a * k - det * yl * yl, F(0))) + b * yl) / a
    l, r = tiles(mean[0] + left - F(0.02), mean[0] + right + F(0.02))
    return max(x0, l), min(x1, r)


@pytest.mark.parametrize("seed,min_sigma,max_sigma", [(1, 0.55, 3.0), (2, 0.55, 30.0),
                                                     (3, 5.0, 60.0), (4, 0.55, 300.0)])
def test_no_pixel_that_takes_a_splat_is_cut(seed, min_sigma, max_sigma):
    rs = np.random.default_rng(seed)
    W, H = 400, 304
    X, Y = np.meshgrid(np.arange(W, dtype=F) + F(0.5), np.arange(H, dtype=F) + F(0.5))
    kept = whole = 0
    for _ in range(250):
        s = np.exp(rs.uniform(np.log(min_sigma), np.log(max_sigma), 2))
        t = rs.uniform(0, np.pi)
        R = np.array([[np.cos(t), -np.sin(t)], [np.sin(t), np.cos(t)]])
        inv = np.linalg.inv(R @ np.diag(s * s) @ R.T).astype(F)
        co = (inv[0, 0], inv[0, 1], inv[1, 1])
        mean = rs.uniform((-40, -40), (W + 40, H + 40)).astype(F)
        min_alpha = F(rs.choice([1 / 255, 0.01, 0.3]))
        opacity = F(min(0.999, float(min_alpha) * (1 + 10 ** rs.uniform(-6, 2.5))))
        fp = footprint(co, opacity, min_alpha)
        dx, dy = X - mean[0], Y - mean[1]
        power = F(-0.5) * (co[0] * dx * dx + co[2] * dy * dy) - co[1] * dx * dy
        with np.errstate(over="ignore"):
            taken = (power <= 0) & (opacity * np.exp(power) >= min_alpha)
        cut = np.zeros((H, W), bool)
        x0, x1 = tiles(mean[0] - fp[1], mean[0] + fp[1]) if not fp[5] else (0, W // 16)
        y0, y1 = tiles(mean[1] - fp[2], mean[1] + fp[2]) if not fp[5] else (0, H // 16)
        for row in range(H // 16):
            l, r = row_columns(co, mean, fp, row, max(x0, 0), min(x1, W // 16 - 1))
            if not y0 <= row <= y1:
                l, r = 1, 0
            cut[row * 16: row * 16 + 16] = True
            cut[row * 16: row * 16 + 16, max(l, 0) * 16: (r + 1) * 16] = False
            kept += max(0, r - l + 1)
        whole += W * H // 256
        assert not (taken & cut).any(), (co, mean, opacity, min_alpha)
    assert kept < 0.8 * whole  # and the cut is one


def stressed_cloud(kind):
    P, rest = O.random_cloud(7, 6000, 1, log_scale_mean=-3.5)
    rs = np.random.default_rng(8)
    if kind == "needles":
        P[3:6] = rs.normal(-3.5, 1.6, P[3:6].shape)
    elif kind == "specks":
        P[3:6] = rs.normal(-7.0, 0.5, P[3:6].shape)
    elif kind == "floor":  # opacities from just over 1/255 up
        a = (1 / 255) * (1 + 10 ** rs.uniform(-6, 1.5, P.shape[1]))
        P[10] = np.log(a / (1 - a))
    elif kind == "large":
        P[3:6, ::20] = rs.normal(0.0, 0.5, P[3:6, ::20].shape)
    return np.ascontiguousarray(P, dtype=np.float32), rest


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["plain", "needles", "specks", "floor", "large"])
@pytest.mark.parametrize("min_alpha", [None, 0.0, 0.05])
def test_images_from_cut_lists_are_those_of_the_whole_lists(kind, min_alpha):
    from test_gpu_parity import check_image

    P, rest = stressed_cloud(kind)
    cloud = px.GaussianCloud(P, 1, rest)
    for view in O.orbit_views(2, 213, 149, radius=2.6, seed=9):
        cam = view.camera()
        opt = RasterOptions(sh_degree=1, background=(0.1, 0.2, 0.3), min_alpha=min_alpha)
        rgb, T = px.render_splats(cloud, cam, opt)
        ora = O.oracle_project(P, rest, 1, cam, opt)
        o_rgb, o_T = O.oracle_rasterize(ora, cam, opt)
        margin, _, _ = O.oracle_pixel_decisions(ora, cam, opt)
        check_image(rgb, o_rgb, 3, margin, label=kind)
        check_image(T, o_T, 1, margin, label=kind + " T")
