"""Adjoint of splats of next to no width (no screen dilation): pixels beside the
line, where the conic's products overflow, add nothing."""
from __future__ import annotations

import ctypes as ct

import numpy as np
import pytest

import oracle_lib as O
import parallax_b200 as px
from parallax_b200._abi import RasterOptions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pixels", [1, 2, 4])
@pytest.mark.parametrize("axis", [0, 1])
def test_a_line_through_pixel_centres(pixels, axis):
    w, h = 40, 24
    b = O.CloudBuilder(0)
    log_scale = np.array([-26.9, -26.9, -3.0])
    log_scale[axis] = np.log(600.0)  # 3e4 px long, 1e-10 px wide
    b.add([0, 0, 2], log_scale, [1, 0, 0, 0], 2.0, [0.5, 0, 0])
    b.add([0.01, 0, 2.1], [-3, -3, -3], [1, 0, 0, 0], 0.0, [0.1, 0.4, 0])
    cloud = px.GaussianCloud(b.params(), 0, 0)
    view = O.View((100.0, 100.0, 20.5, 10.5), w, h, np.eye(3), np.zeros(3))
    opt = RasterOptions(screen_dilation=0.0)
    target = np.random.default_rng(1).uniform(0, 1, w * h * 3).astype(np.float32)
    lib = px.lib()
    before = ct.c_int32(), ct.c_int32()
    lib.pxs_get_raster_config(ct.byref(before[0]), ct.byref(before[1]))
    assert lib.pxs_set_raster_config(pixels, pixels) == 0
    try:
        grads = px.SplatGradients.zeros(cloud)
        loss = px.render_and_accumulate(cloud, view.camera(), opt, target, 0.2, grads)
    finally:
        lib.pxs_set_raster_config(before[0].value, before[1].value)
    want_loss, want, want_screen, _ = O.oracle_render_and_accumulate(
        cloud.params, 0, 0, view.camera(), opt, target, 0.2)
    assert abs(loss - want_loss) <= 1e-5 * want_loss
    # float32 sums over the image's pixels in two orders, and the documented relative
    # errors (2^-22 and less) of the device's approximations
    assert np.all(np.abs(grads.screen_gradient - want_screen) <= 1e-4 * want_screen)
    for got, ref in zip(grads.params.T, want.T):
        assert np.linalg.norm(got - ref) <= 1e-4 * np.linalg.norm(ref)
