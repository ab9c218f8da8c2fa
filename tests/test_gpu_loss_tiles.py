"""The loss by 32x32 tiles (small batches that a march down their columns would take
longer over), at the tiles' edges, over single images, batches of one size and of
several. Tolerances as test_gpu_loss_march's."""
from __future__ import annotations

import ctypes as ct

import numpy as np
import pytest

import oracle_lib as O
import parallax_b200 as px

pytestmark = pytest.mark.gpu


def images(seed, shape):
    rs = np.random.default_rng(seed)
    target = rs.uniform(0, 1, shape).astype(np.float32)
    near = np.clip(target + 0.05 * rs.standard_normal(target.shape), 0, 1).astype(np.float32)
    near.reshape(-1)[::7] = target.reshape(-1)[::7]  # no L1 gradient there
    return near, target


@pytest.mark.parametrize("width,height", [(1, 1500), (5, 2000), (31, 2000), (32, 2100),
                                          (33, 1500), (64, 800), (65, 1500)])
@pytest.mark.parametrize("weight", [0.2, 1.0])
def test_one_image(width, height, weight):
    near, target = images(width, width * height * 3)
    loss, grad = px.photometric_loss(near, target, width, height, weight)
    o_loss = O.oracle_loss_f64(near, target, width, height, weight)
    _, o_grad = O.oracle_loss(near, target, width, height, weight)
    assert abs(loss - o_loss) <= 1e-5 * abs(o_loss)
    assert np.abs(grad - o_grad).max() <= 1e-5 * np.abs(o_grad).max()
    ssim, d = px.mean_ssim(near, target, width, height)
    o_ssim = 1.0 - O.oracle_loss_f64(near, target, width, height, 1.0)
    _, o_d = O.oracle_ssim(near, target, width, height)
    assert abs(ssim - o_ssim) <= 1e-5 * abs(o_ssim)
    assert np.abs(d - o_d).max() <= 1e-5 * np.abs(o_d).max()


@pytest.mark.parametrize("n,w,h", [(8, 109, 109), (9, 96, 129), (40, 1, 65), (64, 33, 65),
                                   (64, 109, 23)])
def test_a_batch(n, w, h):
    torch = pytest.importorskip("torch")
    near, target = images(n, (n, h * w * 3))
    a, b = torch.from_numpy(near).cuda(), torch.from_numpy(target).cuda()
    grad = torch.full_like(a, float("nan"))
    per, loss = torch.empty(n, device="cuda"), torch.empty(1, device="cuda")
    error = ct.create_string_buffer(256)
    for want_grad in (True, False):  # the second call meets the first one's sums
        assert px.lib().pxs_photometric_loss_static(
            a.data_ptr(), b.data_ptr(), w, h, n, 0.2, grad.data_ptr() if want_grad else None,
            per.data_ptr(), loss.data_ptr(), torch.cuda.current_stream().cuda_stream, error,
            256) == 0
        torch.cuda.synchronize()
        losses = np.array([O.oracle_loss_f64(near[k], target[k], w, h, 0.2) for k in range(n)])
        assert (np.abs(per.cpu().numpy() - losses) <= 1e-5 * losses).all()
        assert abs(loss.item() - losses.mean()) <= 1e-5 * losses.mean()
    grads = np.stack([O.oracle_loss(near[k], target[k], w, h, 0.2)[1] for k in range(n)])
    assert np.abs(grad.cpu().numpy() - grads).max() <= 1e-5 * np.abs(grads).max()


def test_a_batch_of_several_sizes():
    # against each view alone (marches and tiles)
    params, rest = O.random_cloud(17, 2000, 0, log_scale_mean=-3.0)
    cloud = px.GaussianCloud(params, 0, rest)
    sizes = [(33, 480), (130, 310), (500, 333)]
    views = [O.orbit_views(1, w, h, seed=w)[0] for w, h in sizes]
    targets = [images(w, w * h * 3)[1] for w, h in sizes]
    cfg = px.TrainConfig(iterations=10, sh_degree=0, sh_increase_interval=0,
                         densify_from_iteration=100, densify_until_iteration=100)
    trainer = px.SplatTrainer(cloud, [(v.camera(), t) for v, t in zip(views, targets)], cfg)
    loss = trainer.accumulate([0, 1, 2], graph=False)
    import torch
    pointer, count, _ = trainer.gradient_buffers()[0]

    class Buffer:
        __cuda_array_interface__ = {"data": (pointer, False), "shape": (count,),
                                    "typestr": "<f4", "version": 3}
    got = torch.as_tensor(Buffer(), device="cuda").cpu().numpy().copy()
    want = px.SplatGradients.zeros(cloud)
    losses = [px.render_and_accumulate(cloud, v.camera(), px.RasterOptions(), t, cfg.ssim_weight,
                                       want) for v, t in zip(views, targets)]
    assert abs(loss - np.mean(losses)) <= 1e-6 * np.mean(losses)
    # float32 sums in two orders
    assert np.linalg.norm(got - want.params.reshape(-1)) <= 1e-4 * np.linalg.norm(want.params)
    trainer.close()
