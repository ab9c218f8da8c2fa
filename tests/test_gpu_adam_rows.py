"""Adam over rows that all start on 16 bytes (counts that are a multiple of four):
the rotation goes by groups and through shared memory to a thread per quaternion.
Held bit for bit to the oracle's per-gaussian loop around a block of 256 gaussians,
with quaternions that vanish, and with the scenes' own position rates."""
from __future__ import annotations

import ctypes as ct

import numpy as np
import pytest

import oracle_lib as O
import parallax_b200 as px

pytestmark = pytest.mark.gpu


def oracle_adam(params, grads, m, v, rest, lr, c1, c2):
    p, m, v = params.copy(), m.copy(), v.copy()
    O.pxo().pxo_adam_f32(O.as_ptr(p), O.as_ptr(grads), O.as_ptr(m), O.as_ptr(v),
                         params.shape[1], rest, O.as_ptr(lr), ct.c_float(0.9), ct.c_float(0.999),
                         ct.c_float(1e-15), ct.c_float(c1), ct.c_float(c2))
    return p, m, v


@pytest.mark.parametrize("n", [4, 8, 252, 256, 260, 508, 1024, 4100])
@pytest.mark.parametrize("rest", [0, 3, 8, 15])
@pytest.mark.parametrize("zero_grads", [0, 1])
def test_counts_about_a_block(n, rest, zero_grads):
    torch = pytest.importorskip("torch")
    rs = np.random.default_rng(1000 * rest + n)
    P = px.param_count(rest)
    params = rs.normal(0, 1, (P, n)).astype(np.float32)
    grads = rs.normal(0, 1e-3, (P, n)).astype(np.float32)
    m = rs.normal(0, 1e-4, (P, n)).astype(np.float32)
    v = np.abs(rs.normal(0, 1e-6, (P, n))).astype(np.float32)
    gone = rs.random(n) < 0.2  # a quaternion of no length becomes the identity
    for a in (params, grads, m, v):
        a[6:10, gone] = 0.0
    lr = np.array([5e-4, 5e-3, 1e-3, 0.05, 2.5e-3, 1.25e-4], dtype=np.float32)
    c1, c2 = np.float32(1) - np.float32(0.9) ** 3, np.float32(1) - np.float32(0.999) ** 3
    d = [torch.from_numpy(a).cuda().contiguous() for a in (params, grads, m, v)]
    torch.cuda.synchronize()
    ctx = px.Context(0)
    ctx.check(px.lib().pxs_adam_device(ctx.handle, d[0].data_ptr(), d[1].data_ptr(),
                                       d[2].data_ptr(), d[3].data_ptr(), n, rest,
                                       lr.ctypes.data, 0.9, 0.999, 1e-15, float(c1), float(c2),
                                       zero_grads))
    torch.cuda.synchronize()
    want = oracle_adam(params, grads, m, v, rest, lr, c1, c2)
    got = [t.cpu().numpy() for t in d]
    for a, b in zip((got[0], got[2], got[3]), want):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    assert (got[1] == 0).all() if zero_grads else np.array_equal(got[1], grads)
    ctx.close()


@pytest.mark.parametrize("counts", [(300, 724), (301, 724), (4, 252), (1, 2)])
def test_position_rates_of_scenes(counts):
    torch = pytest.importorskip("torch")
    w, h, rest = 48, 36, 3
    cfg = px.TrainConfig(iterations=100, sh_degree=1, sh_increase_interval=0,
                         densify_from_iteration=1000, densify_until_iteration=1000,
                         position_lr_initial=0.01, position_lr_final=0.001)
    clouds, scene_views, extents = [], [], []
    for s, count in enumerate(counts):
        params, _ = O.random_cloud(80 + s, count, 1, log_scale_mean=-2.5)
        clouds.append(px.GaussianCloud(params, 1, rest))
        image = np.random.default_rng(s).uniform(0, 1, w * h * 3).astype(np.float32)
        scene_views.append([(v.camera(), image)
                            for v in O.orbit_views(2, w, h, radius=3.0 + s, seed=s)])
        alone = px.SplatTrainer(clouds[s], scene_views[s], cfg)
        extents.append(np.float32(alone.state()["extent"]))
        alone.close()
    assert extents[0] != extents[1]
    joint = px.SplatTrainer.from_scenes(clouds, scene_views, cfg)
    joint.accumulate([0, 1, 2, 3], graph=False)
    pointer, count, _ = joint.gradient_buffers()[0]

    class Buffer:
        __cuda_array_interface__ = {"data": (pointer, False), "shape": (count,),
                                    "typestr": "<f4", "version": 3}
    grads = torch.as_tensor(Buffer(), device="cuda").cpu().numpy().reshape(-1, sum(counts))
    joint.apply()
    got = joint.cloud_params()
    joint.close()
    f = np.float32
    c1, c2 = f(1) - f(0.9), f(1) - f(0.999)
    at = 0
    for cloud, extent in zip(clouds, extents):
        mine = slice(at, at + cloud.count)
        at += cloud.count
        lr = np.array([f(cfg.position_lr_initial) * extent, cfg.scale_lr, cfg.rotation_lr,
                       cfg.opacity_lr, cfg.dc_lr, f(cfg.dc_lr) / f(cfg.sh_rest_lr_divider)],
                      dtype=np.float32)
        zero = np.zeros_like(cloud.params)
        want, _, _ = oracle_adam(cloud.params, np.ascontiguousarray(grads[:, mine]), zero, zero,
                                 rest, lr, c1, c2)
        assert np.array_equal(got[:, mine].view(np.uint32), want.view(np.uint32))
