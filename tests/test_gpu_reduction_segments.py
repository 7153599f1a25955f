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


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_sums_are_rounded_once(dtype):
    """Sums of many like-signed or cancelling terms within one unit in the
    last place of the correctly rounded sum of the FP64 terms."""
    import torch

    from cutile.runtime import reductions as R

    rng = np.random.default_rng(2)
    for shape, halo in (((300, 700), (1, 16)), ((40, 50, 60), (1, 1, 1)), ((100001,), (3,))):
        inner = tuple(slice(h, s - h) for h, s in zip(halo, shape))
        for offset in (1.0, 0.0):
            a, b = ((offset + 0.1 * rng.standard_normal(shape)).astype(dtype) for _ in range(2))
            ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
            ia, ib = a[inner].astype(np.float64), b[inner].astype(np.float64)
            d = ia - ib
            for got, terms in ((R.mass(ta, halo), ia), (R.energy(ta, halo), ia * ia),
                               (R.reduce(R.DIFF_SUMSQ, ta, halo, b=tb), d * d)):
                want = math.fsum(terms.ravel())
                assert abs(got.item() - want) <= np.spacing(abs(want)), (shape, offset)
    big = torch.full((70, 70), 1e308, dtype=torch.float64, device="cuda")
    assert R.mass(big, (1, 1)).item() == math.inf
    big[5, 5] = -math.inf
    assert math.isnan(R.mass(big, (1, 1)).item()) or R.mass(big, (1, 1)).item() == -math.inf
