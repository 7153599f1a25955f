"""Plans of long 2-D flux stages (no GPU): narrow chunks where they keep
twelve warps per SM, 64-wide ones elsewhere."""

import pytest

import stencil_defs as D
from cutile import RKIntegrator, stencil


def euler(r, mu, mv, e, dx, i, j):
    pC = 0.4 * (e[i, j] - 0.5 * (mu[i, j] * mu[i, j] + mv[i, j] * mv[i, j]) / r[i, j])
    pE = 0.4 * (e[i, j + 1] - 0.5 * (mu[i, j + 1] * mu[i, j + 1] + mv[i, j + 1] * mv[i, j + 1]) / r[i, j + 1])
    pW = 0.4 * (e[i, j - 1] - 0.5 * (mu[i, j - 1] * mu[i, j - 1] + mv[i, j - 1] * mv[i, j - 1]) / r[i, j - 1])
    pN = 0.4 * (e[i + 1, j] - 0.5 * (mu[i + 1, j] * mu[i + 1, j] + mv[i + 1, j] * mv[i + 1, j]) / r[i + 1, j])
    pS = 0.4 * (e[i - 1, j] - 0.5 * (mu[i - 1, j] * mu[i - 1, j] + mv[i - 1, j] * mv[i - 1, j]) / r[i - 1, j])
    return (-(mu[i, j + 1] - mu[i, j - 1]) / dx - (mv[i + 1, j] - mv[i - 1, j]) / dx,
            -(mu[i, j + 1] * mu[i, j + 1] / r[i, j + 1] + pE - mu[i, j - 1] * mu[i, j - 1] / r[i, j - 1] - pW) / dx
            - (mu[i + 1, j] * mv[i + 1, j] / r[i + 1, j] - mu[i - 1, j] * mv[i - 1, j] / r[i - 1, j]) / dx,
            -(mu[i, j + 1] * mv[i, j + 1] / r[i, j + 1] - mu[i, j - 1] * mv[i, j - 1] / r[i, j - 1]) / dx
            - (mv[i + 1, j] * mv[i + 1, j] / r[i + 1, j] + pN - mv[i - 1, j] * mv[i - 1, j] / r[i - 1, j] - pS) / dx,
            -((e[i, j + 1] + pE) * mu[i, j + 1] / r[i, j + 1] - (e[i, j - 1] + pW) * mu[i, j - 1] / r[i, j - 1]) / dx
            - ((e[i + 1, j] + pN) * mv[i + 1, j] / r[i + 1, j] - (e[i - 1, j] + pS) * mv[i - 1, j] / r[i - 1, j]) / dx
            + 0.1 * (e[i, j + 1] + e[i, j - 1] + e[i + 1, j] + e[i - 1, j] - 4.0 * pC))


def _plans(fn, dtype, **kw):
    info = RKIntegrator(stencil(ndim=2, dtype=dtype)(fn), "rk2").compile(**kw).info
    assert info["analysis"]["body_ops"] > 120
    return [k["plan"] for k in info["kernels"].values()]


@pytest.mark.parametrize("fn,dtype,tile_x", [
    (D.sw_rhs, "float32", 32), (D.sw_rhs, "float64", 32), (euler, "float32", 32),
    (euler, "float64", 64)])
def test_narrow_chunks_keep_twelve_warps(fn, dtype, tile_x):
    for p in _plans(fn, dtype):
        assert p.tile_x == tile_x
        assert p.vec == (2 if tile_x == 32 else 16 // (4 if dtype == "float32" else 8))
        if tile_x == 32:
            assert p.threads // 32 * p.min_blocks >= 12


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_hints_refine_the_64_wide_plan(dtype):
    """A caller's threads, stages or occupancy mean what they mean for every
    other body: the narrow plan's blocks hold 128 threads at most."""
    vec = 16 // (4 if dtype == "float32" else 8)
    for p in _plans(D.sw_rhs, dtype, kernel_hints={"threads": 64}):
        assert (p.tile_x, p.vec, p.threads, p.occupancy) == (64, vec, 64, 0)
    for p in _plans(D.sw_rhs, dtype, kernel_hints={"min_blocks": 2}):
        assert (p.tile_x, p.vec, p.occupancy) == (64, vec, 2)
