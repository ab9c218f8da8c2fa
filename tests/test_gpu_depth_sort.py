"""The depth sort over its forms: passes that count as they go with 4, 8 or 16
items per thread, and passes with scanned counts, by the number of slots of a
view and in all. Every gaussian is in view and many share a depth, so the sorted
order has to be the one permutation by (depth, index)."""
from __future__ import annotations

import numpy as np
import pytest

import parallax_b200 as px

pytestmark = pytest.mark.gpu


def cloud_in_view(n, planes, seed):
    rs = np.random.default_rng(seed)
    p = np.zeros((14, n), np.float32)
    p[0:2] = rs.uniform(-0.4, 0.4, (2, n))
    z = rs.uniform(-0.9, 0.9, n) if planes == 0 else rs.integers(0, planes, n) / planes
    p[2] = z.astype(np.float32)
    p[3:6] = -6.0
    p[6] = 1.0
    p[10] = 2.0
    return p


@pytest.mark.parametrize("n", [1, 31, 4095, 4096, 4097, 65536, 65537, 262144, 262145, 655360,
                               655361])
@pytest.mark.parametrize("planes", [0, 1, 37])
def test_the_order_is_by_depth_then_index(n, planes):
    p = cloud_in_view(n, planes, n + planes)
    view = px.SplatView((60.0, 60.0, 47.5, 35.5), 96, 72, np.eye(3), np.array([0.0, 0.0, 3.0]))
    got = px.project_splats(px.GaussianCloud(p, 0, 0), view.camera(), px.RasterOptions())
    assert len(got) == n
    # depth is z + 3 in single precision, as the camera's identity rotation gives it
    depth = (p[2] + np.float32(3.0)).astype(np.float32)
    assert np.array_equal(got["index"], np.argsort(depth, kind="stable"))
    assert np.array_equal(got["depth"], depth[got["index"]])


def test_more_slots_than_the_counting_passes_take():
    """Nine views of 120k slots together pass their limit, each view alone does
    not: the batched gradients match the views' own."""
    n, rest = 120000, 0
    p = cloud_in_view(n, 37, 3)
    rs = np.random.default_rng(4)
    views, images = [], []
    for k in range(9):
        t = np.array([0.02 * k, 0.0, 3.0])
        views.append(px.SplatView((60.0, 60.0, 47.5, 35.5), 96, 72, np.eye(3), t).camera())
        images.append(rs.uniform(0, 1, 96 * 72 * 3).astype(np.float32))
    cfg = px.TrainConfig(iterations=10, sh_degree=0, densify_from_iteration=100,
                         densify_until_iteration=100)
    pairs = list(zip(views, images))
    batched = px.SplatTrainer(px.GaussianCloud(p, 0, rest), pairs, cfg)
    single = px.SplatTrainer(px.GaussianCloud(p, 0, rest), pairs, cfg)
    a = batched.step_batch(9, list(range(9)))
    b = single.step_views(9, list(range(9)))
    # the same lists in the same order: only the order of the atomic sums differs
    assert abs(a - b) <= 1e-6 * abs(b)
    batched.close()
    single.close()
