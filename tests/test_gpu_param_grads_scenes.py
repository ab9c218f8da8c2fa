"""Gradients of a batch of more views than a block of the parameter chain lists at
once (128), over scenes whose gaussians share blocks: scene by scene what one view
after another accumulates."""
from __future__ import annotations

import numpy as np
import pytest

import oracle_lib as O
import parallax_b200 as px
from parallax_b200._abi import RasterOptions, TrainConfig

pytestmark = pytest.mark.gpu


def accumulated(trainer, ids):
    import torch
    trainer.accumulate(ids, graph=False)
    out = []
    for pointer, count, _ in trainer.gradient_buffers():
        class Buffer:
            __cuda_array_interface__ = {"data": (pointer, False), "shape": (count,),
                                        "typestr": "<f4", "version": 3}
        out.append(torch.as_tensor(Buffer(), device="cuda").cpu().numpy())
    return out


@pytest.mark.parametrize("counts", [(1, 126, 200), (300, 5), (257,)])
def test_scenes_of_many_views_match_their_own_trainers(counts):
    views_each, (w, h) = 300 // len(counts), (33, 20)
    clouds, scene_views = [], []
    for s, count in enumerate(counts):
        params, rest = O.random_cloud(70 + s, count, 2, log_scale_mean=-2.5)
        clouds.append(px.GaussianCloud(params, 2, rest))
        image = np.random.default_rng(s).uniform(0, 1, w * h * 3).astype(np.float32)
        scene_views.append([(v.camera(), image)
                            for v in O.orbit_views(views_each, w, h, seed=s)])
    cfg = TrainConfig(iterations=100, sh_degree=2, sh_increase_interval=0,
                      densify_from_iteration=1000, densify_until_iteration=1000)
    joint = px.SplatTrainer.from_scenes(clouds, scene_views, cfg)
    # the views of a scene are not neighbours in the batch
    ids = [s * views_each + k for k in range(views_each) for s in range(len(counts))]
    grads, screen, visible = accumulated(joint, ids)
    total = sum(counts)
    grads = grads.reshape(-1, total)
    at = 0
    for cloud, views in zip(clouds, scene_views):
        want = px.SplatGradients.zeros(cloud)
        for camera, image in views:  # one view after another
            px.render_and_accumulate(cloud, camera, RasterOptions(sh_degree=2), image,
                                     cfg.ssim_weight, want)
        mine = slice(at, at + cloud.count)
        at += cloud.count
        assert np.array_equal(visible[mine], want.visible_count)
        # float32 sums of up to 300 views in two orders
        for got, ref in [(screen[mine], want.screen_gradient)] + list(
                zip(grads[:, mine], want.params)):
            assert np.linalg.norm(got - ref) <= 1e-4 * np.linalg.norm(ref)
    joint.close()
