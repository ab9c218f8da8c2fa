"""The Adam kernel cuts the flat P x N arrays into groups of four floats that
run across rows, leaves the rotation rows to other threads and takes groups that
straddle a change of learning rate element by element; a parameter without any
gradient so far skips its divisions. Held bit for bit to the oracle's per-gaussian
loop where that can go wrong: counts of every remainder, arrays that do not
start on 16 bytes (one float per group), states of zeros of either sign, and an
epsilon of 0, for which 0 / 0 has to stay NaN."""
from __future__ import annotations

import ctypes as ct

import numpy as np
import pytest

import oracle_lib as O
import parallax_b200 as px

pytestmark = pytest.mark.gpu


def same_bits(a, b):
    nan = np.isnan(b)
    return np.array_equal(np.isnan(a), nan) and np.array_equal(
        a.view(np.uint32)[~nan], b.view(np.uint32)[~nan])


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 63, 255, 1023, 4098])
@pytest.mark.parametrize("rest", [0, 3, 8, 15])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("epsilon", [1e-15, 0.0])
def test_every_group_of_the_flat_arrays(n, rest, offset, epsilon):
    torch = pytest.importorskip("torch")
    rs = np.random.default_rng(1000 * rest + n)
    P = px.param_count(rest)
    params = rs.normal(0, 1, (P, n)).astype(np.float32)
    grads = rs.normal(0, 1e-3, (P, n)).astype(np.float32)
    m = rs.normal(0, 1e-4, (P, n)).astype(np.float32)
    v = np.abs(rs.normal(0, 1e-6, (P, n))).astype(np.float32)
    still = rs.random((P, n)) < 0.5  # never a gradient
    grads[still] = rs.choice(np.array([0.0, -0.0], np.float32), int(still.sum()))
    m[still] = rs.choice(np.array([0.0, -0.0], np.float32), int(still.sum()))
    v[still] = 0.0
    params[0, : n // 2] = -0.0
    lr = np.array([5e-4, 5e-3, 1e-3, 0.05, 2.5e-3, 1.25e-4], dtype=np.float32)
    c1, c2 = np.float32(1) - np.float32(0.9) ** 3, np.float32(1) - np.float32(0.999) ** 3
    held = [torch.zeros(P * n + offset, device="cuda") for _ in range(4)]
    d = [h[offset:] for h in held]
    for t, a in zip(d, (params, grads, m, v)):
        t.copy_(torch.from_numpy(a.reshape(-1)))
    torch.cuda.synchronize()
    ctx = px.Context(0)
    ctx.check(px.lib().pxs_adam_device(ctx.handle, d[0].data_ptr(), d[1].data_ptr(),
                                       d[2].data_ptr(), d[3].data_ptr(), n, rest,
                                       lr.ctypes.data, 0.9, 0.999, epsilon, float(c1),
                                       float(c2), offset))
    torch.cuda.synchronize()
    p_ref, m_ref, v_ref = params.copy(), m.copy(), v.copy()
    O.pxo().pxo_adam_f32(O.as_ptr(p_ref), O.as_ptr(grads), O.as_ptr(m_ref), O.as_ptr(v_ref), n,
                         rest, O.as_ptr(lr), ct.c_float(0.9), ct.c_float(0.999),
                         ct.c_float(epsilon), ct.c_float(c1), ct.c_float(c2))
    got = [t.cpu().numpy().reshape(P, n) for t in d]
    assert same_bits(got[0], p_ref)
    assert same_bits(got[2], m_ref)
    assert same_bits(got[3], v_ref)
    assert (got[1] == 0).all() if offset else same_bits(got[1], grads)
    ctx.close()
