"""FP64 reductions at the sizes where their row segments and warps split."""

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape,halo,nblocks", [
    ((1,), (0,), 1), ((255,), (0,), 296), ((1025,), (0,), 3), ((40000,), (7,), 296),
    ((3, 1024), (1, 0), 2), ((700, 9), (1, 1), 1), ((2, 2051), (0, 1), 1024),
    ((5, 6, 300), (1, 1, 16), 296), ((40, 3, 17), (1, 1, 1), 5)])
def test_reduction_segments(dtype, shape, halo, nblocks):
    """Sums against correctly rounded ones: at most 2^-46 of the sum of
    magnitudes (fewer than 128 roundings of 2^-53 lie on any element's path
    here, its own product's among them); maxima and their NaN exactly."""
    import torch

    from cutile.runtime import reductions as R

    rng = np.random.default_rng(sum(shape))
    a, b = (rng.standard_normal(shape).astype(dtype) for _ in range(2))
    inner = tuple(slice(h, s - h) for h, s in zip(halo, shape))
    ia, ib = a[inner].astype(np.float64), b[inner].astype(np.float64)
    ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    part = torch.full((nblocks,), float("nan"), dtype=torch.float64, device="cuda")

    def red(op, second=None):
        return R.reduce(op, ta, halo, b=second, nblocks=nblocks, partials=part).item()

    def close(got, terms):
        exact = math.fsum(terms.ravel())
        return abs(got - exact) <= 2.0 ** -46 * math.fsum(np.abs(terms).ravel())

    assert close(red(R.SUM), ia)
    assert close(red(R.SUMSQ), ia * ia)
    assert close(red(R.DIFF_SUMSQ, tb), (ia - ib) ** 2)
    assert red(R.MAXABS) == np.abs(ia).max()
    assert red(R.DIFF_MAXABS, tb) == np.abs(ia - ib).max()
    at = tuple(h + (s - 2 * h) // 2 for h, s in zip(halo, shape))
    ta[at] = float("nan")
    assert math.isnan(red(R.MAXABS)) and math.isnan(red(R.SUM))
