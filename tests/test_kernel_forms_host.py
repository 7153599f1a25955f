"""Forms of a generated source (no GPU): each compiles alone, holds its own
kernels only, and the kernels of all forms are those of the whole source."""

import re

import pytest

import stencil_defs as D
from cutile import RKIntegrator, stencil
from cutile import compile as stencil_compile
from cutile.lowering.target_to_cuda import source_forms
from cutile.runtime import native


def _entries(source, form=None):
    _, log = native.compile_source(source, () if form is None else native.form_option(form))
    return re.findall(r"Compiling entry function '([^']+)'", log)


def _lap7(**kw):
    return stencil_compile(stencil(ndim=3, boundary="periodic")(D.lap7), **kw).cuda_source


def test_rewritten_fields_are_known_without_the_direct_form():
    """Whether a launch may take the direct form is decided before it is there."""
    src = RKIntegrator(stencil(ndim=2)(D.heat2d), "rk4").compile().cuda_source
    for k, rewrites in enumerate((False, True, True, False)):
        mark = f"\n__device__ const unsigned* at = &heat2d_rk4_s{k}_direct_rewrites;"
        if rewrites:
            native.compile_source(src + mark, native.form_option(0))
        else:
            with pytest.raises(native.CsdError):
                native.compile_source(src + mark, native.form_option(0))


@pytest.mark.parametrize("source,names,forms", [
    (lambda: _lap7(temporal_blocking=False), {"lap7": (1,), "lap7_bc": ()},
     [["lap7_tma", "lap7_ldg", "lap7_bc_tma", "lap7_bc_ldg"], ["lap7_direct"], [], []]),
    (lambda: _lap7(temporal_steps=2), {"lap7": (2, 3), "lap7_bc": ()},
     [["lap7_tma", "lap7_ldg", "lap7_bc_tma", "lap7_bc_ldg"], [],
      ["lap7_ring_tma", "lap7_ring_ldg"], ["lap7_batch_tma", "lap7_batch_ldg"]]),
    (lambda: stencil_compile(stencil(ndim=2)(D.heat2d)).cuda_source, {"heat2d": (3,)},
     [["heat2d_tma", "heat2d_ldg"], [], [], ["heat2d_batch_tma", "heat2d_batch_ldg"]]),
    (lambda: RKIntegrator(stencil(ndim=2)(D.heat2d), "rk2").compile().cuda_source,
     {"heat2d_rk2_s0": (1,), "heat2d_rk2_s1": (1,)},
     [[f"heat2d_rk2_s{k}_{e}" for k in (0, 1) for e in ("tma", "ldg")],
      [f"heat2d_rk2_s{k}_direct" for k in (0, 1)], [], []])])
def test_forms_hold_their_own_kernels(source, names, forms):
    src = source()
    for name, want in names.items():
        assert source_forms(src, name) == want
    for form, want in enumerate(forms):
        assert sorted(_entries(src, form)) == sorted(want)
    assert sorted(_entries(src)) == sorted(sum(forms, []))
