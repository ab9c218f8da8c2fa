"""pxs_project's records are built on the device from the sorted slots: clouds that fill
the slots of a sort tile (4096) exactly, by one less and by one more, seen whole, in
part and not at all."""
from __future__ import annotations

import numpy as np
import pytest

import oracle_lib as O
import parallax_b200 as px
from parallax_b200._abi import RasterOptions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 4095, 4096, 4097, 8192])
@pytest.mark.parametrize("seen", ["all", "some", "none"])
def test_records(count, seen):
    params, rest = O.random_cloud(count, count, 0, log_scale_mean=-3.0)
    params[0:2] *= 0.1
    params[2] = 4.0 + np.abs(params[2])
    if seen != "all":
        params[2, slice(None) if seen == "none" else slice(0, None, 2)] *= -1.0  # behind
    params[10] = 2.0
    view = O.View((60.0, 60.0, 32.0, 24.0), 64, 48, np.eye(3), np.zeros(3))
    opt = RasterOptions()
    got = px.project_splats(px.GaussianCloud(params, 0, rest), view.camera(), opt)
    want = O.oracle_project(params, rest, 0, view.camera(), opt)
    assert len(got) == {"all": count, "some": count // 2, "none": 0}[seen] == len(want)
    assert np.all(np.diff(got["depth"]) >= 0)
    # the oracle sorts equal depths its own way: by gaussian
    got, want = np.sort(got, order="index"), np.sort(want, order="index")
    for name in ("index", "clamped"):
        assert np.array_equal(got[name], want[name])
    for name in ("mean", "cov2d", "conic", "depth", "radius", "color", "opacity"):
        # single float operations in the reference's order, exp within 2 ulp
        assert np.allclose(got[name], want[name], rtol=1e-5, atol=1e-6)
