"""Renders into page-locked memory go to the host in more bands than those into
pageable memory (or where one of the two arrays is): bit for bit what one launch over
all tiles gives."""
from __future__ import annotations

import ctypes as ct

import numpy as np
import pytest

import oracle_lib as O
import parallax_b200 as px
from parallax_b200._abi import RasterOptions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height", [(592, 512), (592, 513), (1601, 1203), (2100, 2099),
                                          (20000, 9), (9, 20000)])
def test_bands_into_any_memory(width, height):
    torch = pytest.importorskip("torch")
    P, rest = O.random_cloud(width + height, 6000, 1, log_scale_mean=-3.5)
    cam = O.orbit_views(1, width, height, seed=3)[0].camera()
    cloud, opt = px.GaussianCloud(P, 1, rest), RasterOptions(background=(0.25, 0.5, 0.75))
    c, ctx, lib = cloud.c_struct(), px.default_context(), px.lib()
    try:
        # heaviest tiles first: no bands
        assert lib.pxs_set_raster_schedule(0, 0, 1, -1) == 0
        want_rgb, want_transmittance = px.render_splats(cloud, cam, opt)
    finally:
        assert lib.pxs_set_raster_schedule(0, 0, 0, -1) == 0

    def array(n, locked):
        a = torch.full((n,), float("nan"))
        return a.pin_memory() if locked else a

    n = width * height
    for rgb_locked, transmittance_locked in ((1, 1), (1, 0), (0, 1), (0, 0), (1, None), (0, None)):
        rgb = array(3 * n, rgb_locked)
        transmittance = None if transmittance_locked is None else array(n, transmittance_locked)
        ctx.check(lib.pxs_render(ctx.handle, ct.byref(c), ct.byref(cam), ct.byref(opt),
                                 rgb.data_ptr(),
                                 None if transmittance is None else transmittance.data_ptr()))
        assert np.array_equal(rgb.numpy(), want_rgb)
        if transmittance is not None:
            assert np.array_equal(transmittance.numpy(), want_transmittance)
