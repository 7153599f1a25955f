"""Shared memory of the 3-D register chains (no GPU): every plan the rule
picks fits a block, also where nothing but the registers bounds the depth."""

import itertools

import pytest

import stencil_defs as D
from cutile import compile as stencil_compile
from cutile import stencil
from cutile.passes.tiling import B200_SMEM_PER_BLOCK
from cutile.runtime import native
from cutile.runtime.launcher import register_chain_plan


def along_x(u, i, j, k):
    return u[i, j, k] + 0.1 * (u[i, j, k - 1] - 2.0 * u[i, j, k] + u[i, j, k + 1])


def pointwise(u, i, j, k):
    return 0.5 * u[i, j, k] + 0.25


def test_planned_chains_fit_a_block():
    chosen = 0
    for rz, ry, rx, T, esz in itertools.product(range(5), range(5), range(5), range(2, 17), (4, 8)):
        plan = register_chain_plan((rz, ry, rx), esz, 1, T, 8, 2 * rz + 1 if ry else 0)
        if not plan:
            continue
        chosen += 1
        plane = plan["chain_rows"] * plan["chain_warps"] * 32 * plan["register_chain"] * esz
        # four staged input planes, two of every intermediate field's where rows
        # beside a thread's own are read
        assert (4 + (2 * (T - 1) if ry else 0)) * plane <= B200_SMEM_PER_BLOCK, (rz, ry, rx, T, esz)
    assert chosen > 100


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("fn,T", [(along_x, None), (along_x, 16), (pointwise, 8), (D.lap7, 3)])
def test_emitted_chains_fit_a_block(fn, T, dtype):
    """What the compiled kernel asks for, by the compiler's own arithmetic
    (without T: the depth that compile() chooses by itself)."""
    r = stencil_compile(stencil(ndim=3, dtype=dtype)(fn), temporal_steps=T)
    if T is None:
        assert r.temporal_steps == 8
    name = r.name
    native.compile_source(r.cuda_source + "\n" + "\n".join(
        f"static_assert(Cfg_{name}_{e}::SMEM_BYTES <= {B200_SMEM_PER_BLOCK}, \"{e}\");"
        for e in ("tma", "ldg")))
