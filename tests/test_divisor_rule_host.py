"""Which FP64 quotients share a kept reciprocal (no GPU): scalars that a body
divides by at least twice per point, in footprints of up to 16 loads; never
constants, never FP32."""

import pytest

import stencil_defs as D
from cutile import RKIntegrator, stencil
from cutile import compile as stencil_compile


def over_12(u, i, j):
    return (u[i, j - 1] + u[i, j + 1] - 2.0 * u[i, j]) / 12.0


def one_quotient(u, dx, i, j):
    return (u[i, j - 1] + u[i, j + 1] - 2.0 * u[i, j]) / dx


def two_quotients(u, dx, i, j):
    return (u[i, j + 1] - u[i, j]) / dx - (u[i + 1, j] - u[i, j]) / dx


def wide(u, dx, i, j):
    return ((u[i, j + 1] + u[i, j + 2] + u[i, j - 1] + u[i, j - 2]
             + u[i, j + 3] + u[i, j - 3] + u[i, j + 4] + u[i, j - 4]) / dx
            + (u[i + 1, j] + u[i + 2, j] + u[i - 1, j] + u[i - 2, j]
               + u[i + 3, j] + u[i - 3, j] + u[i + 4, j] + u[i - 4, j]) / dx - u[i, j])


@pytest.mark.parametrize("fn,dtype,shared", [
    (over_12, "float64", False), (one_quotient, "float64", False), (two_quotients, "float64", True),
    (two_quotients, "float32", False), (wide, "float64", False)])
def test_rule(fn, dtype, shared):
    r = stencil_compile(stencil(ndim=2, dtype=dtype)(fn), temporal_blocking=False)
    assert ("csd::div_by(" in r.cuda_source) == shared


def test_flux_stages_share_their_grid_spacing():
    r = RKIntegrator(stencil(ndim=2, dtype="float64")(D.sw_rhs), "rk2").compile()
    assert "csd::div_by(" in r.cuda_source
