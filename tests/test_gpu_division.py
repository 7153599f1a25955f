"""Quotients by a shared divisor (a scalar parameter, a constant) are the
correctly rounded ones NumPy computes, for every kind of dividend."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 1 << 20


def over_s(u, s, i):
    return u[i] / s


def over_12(u, i):
    return u[i] / 12.0


def over_3(u, i):
    return u[i] / -3.0


def over_8(u, i):
    return u[i] / 8.0


def over_tiny(u, i):
    return u[i] / 1e-30


def over_huge(u, i):
    return u[i] / 3e38


def _bits(dtype, seed):
    """Random bit patterns (all exponents, subnormals, infinities, NaN), then
    random significands near one, zeros and powers of two."""
    rng = np.random.default_rng(seed)
    it = np.uint32 if dtype == np.float32 else np.uint64
    a = rng.integers(0, np.iinfo(it).max, N // 2, dtype=it, endpoint=True).view(dtype)
    b = (rng.random(N // 2) + 1.0).astype(dtype) * rng.choice([-1, 1], N // 2).astype(dtype)
    b[:64] = [0.0, -0.0] * 32
    b[64:128] = np.ldexp(dtype(1), np.arange(-32, 32)).astype(dtype)
    return np.concatenate([a, b])


def _run(fn, dtype, u, **scalars):
    import torch

    import cutile
    from cutile import stencil

    r = cutile.compile(stencil(ndim=1, dtype=np.dtype(dtype).name)(fn), temporal_blocking=False,
                       align_halo=False)
    t = torch.from_numpy(u).cuda()
    out = torch.zeros_like(t)
    r.load_module().program().launch([t], [out], scalars=scalars or None)
    h = r.halo_widths[0]
    return out.cpu().numpy()[h:len(u) - h], slice(h, len(u) - h)


def _same(got, want):
    it = np.uint32 if got.dtype == np.float32 else np.uint64
    nan = np.isnan(want)
    assert np.array_equal(nan, np.isnan(got))
    assert np.array_equal(got.view(it)[~nan], want.view(it)[~nan])


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_scalar_divisors(dtype):
    one = np.nextafter(dtype(2), dtype(0))      # all-ones significand
    rng = np.random.default_rng(1)
    values = [3.0, 0.1, -7.0, 1.0 / 1536, float(one), float(np.nextafter(dtype(1), dtype(2))), 2.0,
              0.0, -0.0, np.inf, np.nan, 1e-38, 3e38, 2.0 ** -60, 2.0 ** 60]
    values += [float(x) for x in (rng.random(8) + 1.0).astype(dtype)]
    for k, s in enumerate(values):
        u = _bits(dtype, k)
        got, inner = _run(over_s, dtype, u, s=s)
        with np.errstate(all="ignore"):
            _same(got, u[inner] / dtype(s))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("fn,y", [(over_12, 12.0), (over_3, -3.0), (over_8, 8.0),
                                  (over_tiny, 1e-30), (over_huge, 3e38)])
def test_constant_divisors(fn, y, dtype):
    u = _bits(dtype, 7)
    got, inner = _run(fn, dtype, u)
    with np.errstate(all="ignore"):
        _same(got, u[inner] / dtype(y))
