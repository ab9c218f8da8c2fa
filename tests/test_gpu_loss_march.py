"""The loss kernel marches down strips of 108 output columns in blocks of rows
chosen from the images' sizes, and the elementwise one takes blocks of 2048
values. Held against the oracle around the edges of those: widths at a strip's
end, heights at and around a block's, images narrower than the blur, and batches
whose sizes change the block height. The tolerances are test_gpu_parity's for the
loss: 1e-5 relative, and 1e-5 of the largest magnitude for the gradient. The loss
is held against the oracle's in double (its float one adds one value after
another and drifts by 1e-4 over 50,000 of them; the kernel sums in double). (A
gradient sums 121 taps of each of three planes in another order than the
reference: sqrt(121) * 2^-24 of the largest is 7e-7)."""
from __future__ import annotations

import ctypes as ct

import numpy as np
import pytest

import oracle_lib as O
import parallax_b200 as px

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (1, 40), (40, 1), (5, 5), (10, 11), (107, 9), (108, 8), (109, 12), (118, 13),
         (128, 7), (216, 31), (217, 33), (331, 150), (64, 700)]


@pytest.mark.parametrize("width,height", SIZES)
@pytest.mark.parametrize("weight", [0.0, 0.2, 1.0])
def test_loss_and_gradient_at_the_edges(width, height, weight):
    rs = np.random.default_rng(width * 1000 + height)
    target = rs.uniform(0, 1, width * height * 3).astype(np.float32)
    near = np.clip(target + 0.05 * rs.standard_normal(target.shape), 0, 1).astype(np.float32)
    near[::7] = target[::7]  # no L1 gradient there
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


@pytest.mark.parametrize("n", [1, 3, 33, 64])
@pytest.mark.parametrize("weight", [0.0, 0.2])
def test_every_image_of_a_batch(n, weight):
    torch = pytest.importorskip("torch")
    w, h = 109, 23
    rs = np.random.default_rng(n)
    target = rs.uniform(0, 1, (n, h * w * 3)).astype(np.float32)
    near = np.clip(target + 0.05 * rs.standard_normal(target.shape), 0, 1).astype(np.float32)
    a, b = torch.from_numpy(near).cuda(), torch.from_numpy(target).cuda()
    grad = torch.full_like(a, float("nan"))
    per, loss = torch.empty(n, device="cuda"), torch.empty(1, device="cuda")
    error = ct.create_string_buffer(256)
    for _ in range(2):  # the second call meets the first one's sums
        assert px.lib().pxs_photometric_loss_static(
            a.data_ptr(), b.data_ptr(), w, h, n, weight, grad.data_ptr(), per.data_ptr(),
            loss.data_ptr(), torch.cuda.current_stream().cuda_stream, error, 256) == 0
        torch.cuda.synchronize()
        want = [O.oracle_loss(near[k], target[k], w, h, weight) for k in range(n)]
        losses = np.array([O.oracle_loss_f64(near[k], target[k], w, h, weight)
                           for k in range(n)])
        assert (np.abs(per.cpu().numpy() - losses) <= 1e-5 * losses).all()
        assert abs(loss.item() - losses.mean()) <= 1e-5 * losses.mean()
        grads = np.stack([x[1] for x in want])
        assert np.abs(grad.cpu().numpy() - grads).max() <= 1e-5 * np.abs(grads).max()
