"""GPU tests of the blend's approximate arithmetic: the reciprocal of the backward passes against 64 bits, and the pixels that a gaussian
splat is taken to reach against those at which its weight passes the cut-off."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _call(which, x, out):
    from inpc_b200 import _cabi
    _cabi.check(_cabi.lib().inpc_debug_arithmetic(which, out.numel(), x.data_ptr(), out.data_ptr(), torch.cuda.current_stream().cuda_stream))
    return out.cpu().numpy()


def test_reciprocal_is_rounded_once():
    """From an approximation that is an ulp off, one step of Newton's method in fused operations leaves the rounding of the last one, half an ulp, and
    the square of the first error: 2^-22 of an ulp."""
    rng = np.random.default_rng(1)
    x = np.concatenate([np.exp(rng.uniform(math.log(1e-8), 0.0, 1 << 20)), 1.0 - np.arange(1 << 16) * 2.0 ** -24, rng.uniform(0.0, 1.0, 1 << 20), rng.uniform(1.0, 2.0, 1 << 18),
                        np.exp(rng.uniform(0.0, math.log(2.0 ** 125), 1 << 18)), 2.0 ** np.arange(-26, 126), [1e-8]]).astype(np.float32)
    got = _call(0, torch.from_numpy(x).to(DEV), torch.empty(len(x), device=DEV)).astype(np.float64)
    exact = 1.0 / np.maximum(x, np.float32(1e-8)).astype(np.float64)
    off = np.abs(got - exact) / np.spacing(exact.astype(np.float32)).astype(np.float64)
    # (where the exact value lies at a power of two, an ulp below it is half as large)
    assert off.max() <= 0.5 + 2.0 ** -20, off.max()


def test_reciprocal_of_what_is_no_ordinary_number():
    x = torch.tensor([0.0, -1.0, 1e-9, float("-inf"), float("nan"), float("inf")], device=DEV)
    got = _call(0, x, torch.empty(6, device=DEV))
    assert (got[:5] == np.float32(1.0) / np.float32(1e-8)).all() and got[5] == 0.0


# Sizes from the dilation alone to a screen, round to 100 times as long as wide (a splat that is round in the world is sqrt(1 + x^2 + y^2) times as long as wide at (x, y) of the image
# plane); cut-offs at a fraction of a standard deviation, at three, and far out.
# The widening is two thousandths of the squared distance and one of the half width.  The walk's own sum in 32 bits is off by up to 8 roundings of its terms, which at the cut-off of an ellipse k times
# as long as wide come to k^2 / 2 times the sum: 8 * 2^-24 * 100^2 / 2 = 0.0024.
@pytest.mark.parametrize("reach", [0.1, 1.0, 9.0, 60.0])
@pytest.mark.parametrize("longest", [1.0, 3.0, 30.0, 100.0])
def test_no_pixel_that_a_gaussian_splat_reaches_is_left_out(reach, longest):
    rng = np.random.default_rng(int(reach * 10 + longest))
    n = 200_000
    short = 0.4 * np.exp(rng.uniform(0.0, math.log(10.0), n))
    long = short * np.exp(rng.uniform(0.0, math.log(longest), n))
    turn = rng.uniform(0.0, math.pi, n)
    turn[::5] = np.round(turn[::5] / (math.pi / 4)) * (math.pi / 4)      # also along the axes and the diagonals
    c, s = np.cos(turn), np.sin(turn)
    xx, yy, xy = (c * long) ** 2 + (s * short) ** 2, (s * long) ** 2 + (c * short) ** 2, c * s * (long ** 2 - short ** 2)
    det = xx * yy - xy * xy
    px0, py0 = rng.integers(0, 50, n) * 8, rng.integers(0, 50, n) * 4
    # close to the half, or at the distance the ellipse ends at
    away = rng.uniform(-1.05, 1.05, (2, n)) * np.sqrt(reach) * np.sqrt(np.stack([xx, yy]))
    x, y = px0 + rng.uniform(-1.0, 9.0, n) + away[0], py0 + rng.uniform(-1.0, 5.0, n) + away[1]
    v = np.stack([x, y, yy / det, -xy / det, xx / det, np.full(n, reach), px0, py0], axis=1).astype(np.float32)
    got = _call(1, torch.from_numpy(v).to(DEV), torch.empty(n, dtype=torch.int32, device=DEV)).view(np.uint32)
    x, y, a, b, d, r = v[:, :6].astype(np.float64).T
    bit = np.arange(32)
    dx, dy = x[:, None] - (v[:, 6:7] + bit % 8 + 0.5), y[:, None] - (v[:, 7:8] + bit // 8 + 0.5)
    q, terms = a[:, None] * dx * dx + 2 * b[:, None] * dx * dy + d[:, None] * dy * dy, a[:, None] * dx * dx + d[:, None] * dy * dy
    # by the exact sum, or by one in 32 bits as the walk forms it, whose roundings put a pixel that is this close to the cut-off on either side
    f = np.float32
    dx32, dy32 = v[:, 0:1] - (v[:, 6:7] + (bit % 8).astype(f) + f(0.5)), v[:, 1:2] - (v[:, 7:8] + (bit // 8).astype(f) + f(0.5))
    e = f(-0.5) * (v[:, 2:3] * dx32 * dx32 + v[:, 4:5] * dy32 * dy32) - v[:, 3:4] * dx32 * dy32
    met = (q <= r[:, None] + 2 * 2.0 ** -24 * terms) | ((e <= 0) & (e >= f(-0.5) * v[:, 5:6]))
    reached = (got[:, None] >> bit.astype(np.uint32) & 1).astype(bool)
    assert met.any() and not (met & ~reached).any(), int((met & ~reached).sum())
    # and no half is taken whole: of a splat that ends more than a pixel before it nothing is left
    beside = (q > r[:, None]).all(axis=1) & ((np.abs(x - v[:, 6] - 4) > 6 + np.sqrt(r * xx)) | (np.abs(y - v[:, 7] - 2) > 4 + np.sqrt(r * yy)))
    assert not got[beside].any()
