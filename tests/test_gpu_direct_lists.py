"""Tile lists built directly (views of up to 2048 tiles, while tiles times chunks of
256 slots stay few) and by tile rows: the lists on both sides of the lines between
them equal the oracle's, and images of one tile and of one row or column too."""
from __future__ import annotations

import numpy as np
import pytest

import oracle_lib as O
import parallax_b200 as px
from parallax_b200._abi import RasterOptions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,width,height", [
    (1, 16, 16), (255, 17, 15), (257, 700, 10), (4096, 9, 700), (4097, 320, 240),
    (20000, 1024, 512), (20000, 1040, 512),  # 2048 tiles, and 2080
    (262144, 96, 64), (262145, 96, 64),      # the most slots of a view, and one more
    (180000, 1024, 496),                     # 1984 tiles: too many counts
])
def test_lists_on_both_sides_of_the_rule(count, width, height):
    P, rest = O.random_cloud(count, count, 0, log_scale_mean=-4.0)
    view = O.orbit_views(1, width, height, seed=5)[0]
    opt = RasterOptions()
    offsets, entries = px.tile_lists(px.GaussianCloud(P, 0, rest), view.camera(), opt)
    ora = O.oracle_project(P, rest, 0, view.camera(), opt)
    want_offsets, want = O.oracle_tiles(ora, width, height)
    assert np.array_equal(offsets, want_offsets)
    # the oracle's entries index its projected splats
    assert np.array_equal(entries, ora["index"][want])


def test_a_direct_step_whose_lists_overflow_is_redone():
    """Far views set the capacity, near ones pass it; both are small images."""
    P, rest = O.random_cloud(61, 40000, 0, log_scale_mean=-2.2)
    far = O.orbit_views(1, 160, 120, radius=9.0, seed=5)
    near = O.orbit_views(1, 160, 120, radius=1.6, seed=6)
    rs = np.random.default_rng(1)
    pairs = [(v.camera(), rs.uniform(0, 1, 160 * 120 * 3).astype(np.float32)) for v in far + near]
    cfg = px.TrainConfig(iterations=10, sh_degree=0, densify_from_iteration=100,
                         densify_until_iteration=100)
    import ctypes as ct
    steps = []
    for mode in ("plain", "graph"):
        t = px.SplatTrainer(px.GaussianCloud(P, 0, rest), pairs, cfg)
        losses, listed = [], []
        for view in (0, 1):
            losses.append(t.step_views(1, [view]) if mode == "plain"
                          else t.step_batch(1, [view], graph=True))
            k, n = ct.c_int64(), ct.c_int64()
            t._check(px.lib().pxs_trainer_step_info(t.handle, ct.byref(k), ct.byref(n)))
            listed.append(k.value)
        steps.append((losses, listed))
        t.close()
    assert steps[0][1] == steps[1][1]
    assert steps[1][1][1] > 1.5 * steps[1][1][0] + 65536, steps  # it did overflow
    # the losses differ by the order of the first step's atomic sums alone
    assert np.allclose(steps[0][0], steps[1][0], rtol=1e-5)
