"""A captured step replayed for views of another shape: batches that agree in
gaussians, views, pixels and tiles but not in the launches a step takes are stepped
in turn from graphs and plainly, with the same losses and gradients."""
from __future__ import annotations

import numpy as np
import pytest

import oracle_lib as O
import parallax_b200 as px
from parallax_b200._abi import TrainConfig

pytestmark = pytest.mark.gpu


def config():
    # learning rates of 0: the cloud stays as it is, so every step is comparable
    return TrainConfig(iterations=1000, sh_degree=1, sh_increase_interval=0,
                       densify_from_iteration=2000, densify_until_iteration=2000,
                       opacity_reset_interval=0, position_lr_initial=0.0, position_lr_final=0.0,
                       scale_lr=0.0, rotation_lr=0.0, opacity_lr=0.0, dc_lr=0.0)


def gradients(trainer):
    import torch
    out = []
    for pointer, count, _ in trainer.gradient_buffers():
        class Buffer:
            __cuda_array_interface__ = {"data": (pointer, False), "shape": (count,),
                                        "typestr": "<f4", "version": 3}
        out.append(torch.as_tensor(Buffer(), device="cuda").cpu().numpy().copy())
    return out


def views(count, size, seed):
    w, h = size
    image = np.random.default_rng(seed).uniform(0, 1, w * h * 3).astype(np.float32)
    return [(v.camera(), image) for v in O.orbit_views(count, w, h, seed=seed)]


def compare(make, batches, rounds=3):
    graphs, plain = make(), make()
    for _ in range(rounds):  # from the second round on nothing is allocated
        for ids in batches:
            losses, grads = [], []
            for trainer, graph in ((graphs, True), (plain, False)):
                losses.append(trainer.accumulate(ids, graph=graph))
                grads.append(gradients(trainer))
                trainer.apply()
            # the images are the same bits; the losses are sums in double, in two orders
            assert abs(losses[0] - losses[1]) <= 1e-6 * abs(losses[1])
            assert np.array_equal(grads[0][2], grads[1][2])
            for got, ref in zip(grads[0][:2], grads[1][:2]):  # float32 sums in two orders
                assert np.linalg.norm(got - ref) <= 1e-4 * np.linalg.norm(ref)
            # the whole step's graph
            losses = [t.step_batch(len(ids), ids, graph=g) for t, g in ((graphs, True),
                                                                        (plain, False))]
            assert abs(losses[0] - losses[1]) <= 1e-6 * abs(losses[1])
    for trainer in (graphs, plain):
        trainer.close()


@pytest.mark.parametrize("first, second", [
    ((1402, 1408), (1408, 1402)),  # one grid of tiles, another grid of the loss
    ((640, 480), (480, 640)),      # lists built directly
    ((1280, 720), (720, 1280)),    # lists by tile rows: other rows, other columns
    ((512, 1024), (2048, 256)),    # 2048 tiles of one view: 32x64 and 128x16
])
def test_views_of_equal_pixels_and_tiles(first, second):
    params, rest = O.random_cloud(91, 6000, 1, log_scale_mean=-3.0)
    cloud = px.GaussianCloud(params, 1, rest)
    pairs = views(1, first, 5) + views(1, second, 6)
    compare(lambda: px.SplatTrainer(cloud, pairs, config()), [[0], [1], [1, 0], [0, 1]])


def test_batches_of_equal_pixels_and_tiles():
    # two views whose own sizes differ and whose sums agree
    params, rest = O.random_cloud(92, 5000, 1, log_scale_mean=-3.0)
    cloud = px.GaussianCloud(params, 1, rest)
    pairs = (views(1, (320, 320), 7) + views(1, (320, 320), 8) + views(1, (320, 160), 9)
             + views(1, (320, 480), 10))
    compare(lambda: px.SplatTrainer(cloud, pairs, config()), [[0, 1], [2, 3], [3, 2]])


@pytest.mark.parametrize("size", [(320, 240), (1280, 720)])
def test_scenes_of_other_counts(size):
    clouds, scene_views = [], []
    for s, count in enumerate((3000, 20000, 1)):
        params, rest = O.random_cloud(93 + s, count, 1, log_scale_mean=-3.0)
        clouds.append(px.GaussianCloud(params, 1, rest))
        scene_views.append(views(2, size, 20 + s))
    compare(lambda: px.SplatTrainer.from_scenes(clouds, scene_views, config()),
            [[0, 1], [2, 3], [4, 5], [2, 0], [0, 4]])


def test_single_view_steps_of_scenes_of_other_counts():
    # step() replays one graph for every scene's views
    clouds, scene_views = [], []
    for s, count in enumerate((2500, 18000)):
        params, rest = O.random_cloud(97 + s, count, 1, log_scale_mean=-3.0)
        clouds.append(px.GaussianCloud(params, 1, rest))
        scene_views.append(views(2, (320, 240), 30 + s))
    trainer = px.SplatTrainer.from_scenes(clouds, scene_views, config())
    plain = px.SplatTrainer.from_scenes(clouds, scene_views, config())
    want = sorted(plain.step_batch(1, [k], graph=False) for k in range(4))
    for _ in range(3):  # an epoch takes every view once
        got = []
        for _ in range(4):
            assert trainer.step()
            got.append(trainer.state()["last_loss"])
        assert np.allclose(sorted(got), want, rtol=1e-5, atol=0)  # quaternions renormalised in between
    trainer.close()
    plain.close()


@pytest.mark.parametrize("order", [[0, 1, 2, 3, 4, 5], [0, 1, 0, 2, 0, 3, 0, 4, 0, 5]])
def test_more_shapes_than_graphs_are_kept(order):
    # the graphs of the last four shapes are kept
    params, rest = O.random_cloud(99, 4000, 1, log_scale_mean=-3.0)
    cloud = px.GaussianCloud(params, 1, rest)
    sizes = [(320, 240), (240, 320), (640, 120), (120, 640), (160, 480), (480, 160)]
    pairs = [views(1, size, 40 + k)[0] for k, size in enumerate(sizes)]
    compare(lambda: px.SplatTrainer(cloud, pairs, config()), [[k] for k in order])
