"""Which chains keep a ring form for smaller arrays (no GPU), and which are
ring chains only."""

import pytest

import stencil_defs as D
from cutile import compile as stencil_compile
from cutile import stencil
from cutile.runtime import native


def star2(u, i, j):
    return (16.0 * (u[i - 1, j] + u[i + 1, j] + u[i, j - 1] + u[i, j + 1])
            - (u[i - 2, j] + u[i + 2, j] + u[i, j - 2] + u[i, j + 2]) - 60.0 * u[i, j]) / 12.0


def star2_half(u, i, j):
    return (u[i - 2, j] + u[i + 2, j] + u[i, j - 2] + u[i, j + 2] - u[i, j]) / 4.0


def mean9(u, i, j):
    return (u[i, j] + u[i - 1, j] + u[i + 1, j] + u[i, j - 1] + u[i, j + 1] + u[i - 1, j - 1]
            + u[i - 1, j + 1] + u[i + 1, j - 1] + u[i + 1, j + 1]) / 9.0


def ratio(u, dx, i, j):
    return u[i, j] * (0.5 / dx) + 0.25 * (u[i, j - 1] + u[i - 1, j])


@pytest.mark.parametrize("fn,ndim,dtype,T,below", [
    (D.heat1d, 1, "float64", 8, 0), (D.heat2d, 2, "float64", 5, 0), (D.heat2d, 2, "float32", 8, 0),
    (D.wave4, 2, "float64", 3, 0), (D.wave4, 2, "float32", 2, 0), (D.wave4, 2, "float32", 4, 4096),
    (star2, 2, "float32", 2, 16384), (star2, 2, "float64", 2, None),
    (star2_half, 2, "float64", 2, 0),            # a quotient by 4 is a product
    (ratio, 2, "float64", 2, 0),                 # a quotient of scalars is no field's
    (mean9, 2, "float32", 4, 4096), (mean9, 2, "float32", 2, 0), (mean9, 2, "float32", 6, 1536),
    (mean9, 2, "float64", 5, 4096), (mean9, 2, "float64", 6, 2048),
    (mean9, 2, "float64", 2, None),
    (D.lap7, 3, "float64", 2, 256), (D.lap7, 3, "float64", 4, 0), (D.lap7, 3, "float32", 4, 288),
    (D.lap3d, 3, "float64", 2, None), (D.lap3d, 3, "float32", 3, None)])
def test_forms(fn, ndim, dtype, T, below):
    r = stencil_compile(stencil(ndim=ndim, dtype=dtype)(fn), temporal_steps=T)
    assert r.kernel_hints.get("ring_below") == below
    assert ("register_chain" in r.kernel_hints) == (below is not None)
    assert (f"{r.name}_ring_below" in r.cuda_source) == bool(below)


def test_both_forms_compile_and_hints_round_trip():
    op = stencil(ndim=2, dtype="float32")(star2)
    r = stencil_compile(op, temporal_steps=2)
    _, log = native.compile_source(r.cuda_source)
    for entry in ("star2_tma", "star2_ldg", "star2_ring_tma", "star2_ring_ldg"):
        assert f"'{entry}'" in log
    again = stencil_compile(op, temporal_steps=2, tile_sizes=r.tile_sizes,
                            kernel_hints=r.kernel_hints)
    assert again.cuda_source == r.cuda_source
