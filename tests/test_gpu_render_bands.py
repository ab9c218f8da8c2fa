"""Images large enough to go to the host in bands of tile rows, while later bands
are composited: one band, two, the most there are, a last band of one row, one
tile row or column. Bit for bit what one launch over all tiles gives."""
from __future__ import annotations

import ctypes as ct

import numpy as np
import pytest

import oracle_lib as O
import parallax_b200 as px
from parallax_b200._abi import RasterOptions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height", [
    (592, 512),    # 37 x 32 tiles: one band exactly
    (592, 513),    # 33 tile rows: a second band of one
    (700, 701), (1601, 1203),
    (2100, 2099),  # 132 x 132 tiles: eight bands
    (20000, 9), (9, 20000),
])
def test_bands_equal_one_launch(width, height):
    P, rest = O.random_cloud(width + height, 6000, 1, log_scale_mean=-3.5)
    cam = O.orbit_views(1, width, height, seed=3)[0].camera()
    cloud, opt = px.GaussianCloud(P, 1, rest), RasterOptions(background=(0.25, 0.5, 0.75))
    lib = px.lib()
    rgb, transmittance = px.render_splats(cloud, cam, opt)
    try:
        # heaviest tiles first: no bands
        assert lib.pxs_set_raster_schedule(0, 0, 1, -1) == 0
        want_rgb, want_transmittance = px.render_splats(cloud, cam, opt)
    finally:
        assert lib.pxs_set_raster_schedule(0, 0, 0, -1) == 0
    assert np.array_equal(rgb, want_rgb)
    assert np.array_equal(transmittance, want_transmittance)
    # a trainer renders its own cloud the same way
    view = (cam, np.zeros(width * height * 3, np.float32))
    trainer = px.SplatTrainer(cloud, [view], px.TrainConfig(sh_degree=1))
    got_rgb, got_transmittance = np.empty_like(rgb), np.empty_like(transmittance)
    trainer._check(lib.pxs_trainer_render(trainer.handle, ct.byref(cam), ct.byref(opt),
                                          got_rgb.ctypes.data, got_transmittance.ctypes.data))
    assert np.array_equal(got_rgb, want_rgb)
    assert np.array_equal(got_transmittance, want_transmittance)
    trainer.close()
