"""Batches whose depth sort or tile lists go another way than each view's alone: more
slots together than the counting passes take (scanned counts, a segment per view),
and more counts of tiles and chunks than the direct lists take. Every gaussian has its
own colour and opacity and many overlap, so that another order within a view, or
another view's slots, would show in every gradient."""
from __future__ import annotations

import numpy as np
import pytest

import oracle_lib as O
import parallax_b200 as px
from parallax_b200._abi import RasterOptions, TrainConfig

pytestmark = pytest.mark.gpu


def check_batch(params, views, images):
    import torch
    cloud = px.GaussianCloud(params, 0, 0)
    cfg = TrainConfig(iterations=10, sh_degree=0, sh_increase_interval=0,
                      densify_from_iteration=100, densify_until_iteration=100)
    trainer = px.SplatTrainer(cloud, list(zip(views, images)), cfg)
    trainer.accumulate(list(range(len(views))))
    got = []
    for pointer, count, _ in trainer.gradient_buffers():
        class Buffer:
            __cuda_array_interface__ = {"data": (pointer, False), "shape": (count,),
                                        "typestr": "<f4", "version": 3}
        got.append(torch.as_tensor(Buffer(), device="cuda").cpu().numpy().copy())
    trainer.close()
    want = px.SplatGradients.zeros(cloud)
    for camera, image in zip(views, images):  # one view after another
        px.render_and_accumulate(cloud, camera, RasterOptions(), image, cfg.ssim_weight, want)
    assert np.array_equal(got[2], want.visible_count)
    # float32 sums over the views' pixels in two orders
    assert np.linalg.norm(got[1] - want.screen_gradient) <= 1e-4 * np.linalg.norm(
        want.screen_gradient)
    for row, ref in zip(got[0].reshape(want.params.shape), want.params):
        assert np.linalg.norm(row - ref) <= 1e-4 * np.linalg.norm(ref)


def scene(count, views, width, height, seed, log_scale):
    params, _ = O.random_cloud(seed, count, 0, log_scale_mean=log_scale)
    rs = np.random.default_rng(seed + 1)
    params[11:14] = rs.normal(0, 1, (3, count))  # any colour
    params[2, ::3] = np.round(params[2, ::3] * 8) / 8  # equal depths in the first view
    cameras = [v.camera() for v in O.orbit_views(views, width, height, seed=seed)]
    images = [rs.uniform(0, 1, width * height * 3).astype(np.float32) for _ in cameras]
    return params, cameras, images


@pytest.mark.parametrize("count,views", [
    (120000, 9),  # 1.1M slots: scanned counts
    (120000, 8),  # 983,040: counted as the passes go
    (4097, 129),  # 1.06M slots in segments of 8192
])
def test_views_sorted_together(count, views):
    check_batch(*scene(count, views, 96, 72, 3, -3.5))


@pytest.mark.parametrize("count", [
    100000,  # two views of 1900 tiles and 400 chunks each: 1.52M counts, by rows
    90000,   # 352 chunks: 1.34M, directly
])
def test_lists_of_views_together(count):
    check_batch(*scene(count, 2, 800, 608, 5, -4.0))


@pytest.mark.parametrize("count", [
    180000,  # 1984 tiles x 704 chunks: 1.40M counts, directly
    200000,  # x 784: 1.56M, by rows
])
def test_lists_of_one_view(count):
    params, _ = O.random_cloud(count, count, 0, log_scale_mean=-4.0)
    view = O.orbit_views(1, 1024, 496, seed=5)[0]
    offsets, entries = px.tile_lists(px.GaussianCloud(params, 0, 0), view.camera(),
                                     RasterOptions())
    ora = O.oracle_project(params, 0, 0, view.camera(), RasterOptions())
    want_offsets, want = O.oracle_tiles(ora, 1024, 496)
    assert np.array_equal(offsets, want_offsets)
    # the oracle's entries index its projected splats
    assert np.array_equal(entries, ora["index"][want])
