"""Views without a pixel: splats whose squares span the missing image list no tile,
and every call returns nothing to composite."""
from __future__ import annotations

import numpy as np
import pytest

import oracle_lib as O
import parallax_b200 as px
from parallax_b200._abi import RasterOptions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(0, 48), (64, 0), (0, 0), (0, 32768)])
@pytest.mark.parametrize("options", [RasterOptions(), RasterOptions(min_alpha=0.0)])
def test_a_view_without_pixels(size, options):
    w, h = size
    params, rest = O.random_cloud(41, 3000, 0, log_scale_mean=-2.0)
    params[0:2] *= 0.02  # about the axis: the squares span pixel (0, 0)
    cloud = px.GaussianCloud(params, 0, rest)
    view = O.View((60.0, 60.0, 0.0, 0.0), w, h, np.eye(3), np.array([0.0, 0.0, 3.0]))
    # the reference still projects what its square brings to the image's corner
    want = O.oracle_project(params, rest, 0, view.camera(), options)
    got = px.project_splats(cloud, view.camera(), options)
    assert len(want) > 0 and np.array_equal(np.sort(got["index"]), np.sort(want["index"]))
    offsets, entries = px.tile_lists(cloud, view.camera(), options)
    assert np.array_equal(offsets, [0]) and len(entries) == 0
    rgb, transmittance = px.render_splats(cloud, view.camera(), options)
    assert len(rgb) == 0 and len(transmittance) == 0
    grads = px.SplatGradients.zeros(cloud)
    px.render_and_accumulate(cloud, view.camera(), options, np.zeros(0, np.float32), 0.2, grads)
    assert not grads.params.any() and not grads.screen_gradient.any()
    assert grads.visible_count.sum() == len(want)


def test_a_view_without_pixels_beside_another():
    # several views' gradients, in the other view's the ones it has alone
    params, rest = O.random_cloud(42, 3000, 0, log_scale_mean=-2.0)
    cloud = px.GaussianCloud(params, 0, rest)
    view = O.orbit_views(1, 64, 48, seed=2)[0]
    image = np.random.default_rng(3).uniform(0, 1, 64 * 48 * 3).astype(np.float32)
    none = O.View((60.0, 60.0, 0.0, 0.0), 0, 48, np.eye(3), np.array([0.0, 0.0, 3.0]))
    cfg = px.TrainConfig(iterations=10, sh_degree=0, sh_increase_interval=0,
                         densify_from_iteration=100, densify_until_iteration=100)

    def gradients(views, ids):
        import torch
        trainer = px.SplatTrainer(cloud, views, cfg)
        trainer.accumulate(ids, graph=False)
        pointer, count, _ = trainer.gradient_buffers()[0]

        class Buffer:
            __cuda_array_interface__ = {"data": (pointer, False), "shape": (count,),
                                        "typestr": "<f4", "version": 3}
        out = torch.as_tensor(Buffer(), device="cuda").cpu().numpy().copy()
        trainer.close()
        return out

    alone = gradients([(view.camera(), image)], [0])
    both = gradients([(none.camera(), np.zeros(0, np.float32)), (view.camera(), image)], [0, 1])
    # float32 sums in two orders
    assert np.linalg.norm(both - alone) <= 1e-4 * np.linalg.norm(alone)


def test_a_large_cloud_and_no_pixel():
    # more slots than the direct lists take
    params, rest = O.random_cloud(43, 270000, 0, log_scale_mean=-5.0)
    cloud = px.GaussianCloud(params, 0, rest)
    for w, h in ((64, 0), (0, 64)):
        view = O.View((60.0, 60.0, 0.0, 0.0), w, h, np.eye(3), np.array([0.0, 0.0, 3.0]))
        offsets, entries = px.tile_lists(cloud, view.camera(), RasterOptions())
        assert np.array_equal(offsets, [0]) and len(entries) == 0
        rgb, _ = px.render_splats(cloud, view.camera(), RasterOptions())
        assert len(rgb) == 0
