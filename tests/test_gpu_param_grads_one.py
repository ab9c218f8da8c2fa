"""Gradients of a batch of one view (a thread per gaussian, everything in
registers) at the edges of its blocks and at every SH degree, added onto what the
gradients held, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle_lib as O
import parallax_b200 as px
from parallax_b200._abi import RasterOptions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sh_degree", [0, 1, 2, 3])
@pytest.mark.parametrize("count", [1, 127, 128, 129, 1000])
def test_one_view_gradients_match_the_oracle(count, sh_degree):
    P, rest = O.random_cloud(100 * sh_degree + count, count, sh_degree, log_scale_mean=-3.0)
    view = O.orbit_views(1, 75, 50, seed=count)[0]
    cam, opt = view.camera(), RasterOptions()
    rs = np.random.default_rng(count)
    dL = rs.normal(0, 1, 75 * 50 * 3).astype(np.float32)
    cloud = px.GaussianCloud(P, sh_degree, rest)
    grads = px.SplatGradients.zeros(cloud)
    held = rs.integers(-4, 5, grads.params.shape).astype(np.float32)
    grads.params[:] = held
    px.rasterize_splats_backward(cloud, cam, opt, dL, grads)
    ora = O.oracle_project(P, rest, sh_degree, cam, opt)
    want, screen, visible = O.oracle_backward(P, rest, sh_degree, cam, opt, ora, dL)
    assert np.array_equal(grads.visible_count, visible)
    # both sum in float32: 1e-4 of the norm, and half a unit of the sum with `held`
    got = grads.params.astype(np.float64) - held
    rounding = 2.0 ** -24 * np.abs(grads.params)
    for c in range(want.shape[0]):
        bound = 1e-4 * np.linalg.norm(want[c]) + np.linalg.norm(rounding[c])
        assert np.linalg.norm(got[c] - want[c]) <= bound, c
    assert np.linalg.norm(grads.screen_gradient - screen) <= 1e-4 * np.linalg.norm(screen)
    assert np.array_equal(grads.params[:, visible == 0], held[:, visible == 0])
