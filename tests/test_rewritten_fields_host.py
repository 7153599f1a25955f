"""Fields that a Runge-Kutta stage reads and writes (no GPU): the direct form
of such a stage does not load them as read-only data."""

import re

import pytest

import stencil_defs as D
from cutile import RKIntegrator, stencil
from cutile.runtime.rk_integrator import stage_table


def _masks(source):
    return {k: int(v) for k, v in re.findall(r"(\w+)_direct_rewrites = (\d+);", source)}


@pytest.mark.parametrize("method", ["euler", "rk2", "rk4", "ssprk3"])
def test_masks_name_the_inputs_that_are_outputs(method):
    r = RKIntegrator(stencil(ndim=2, dtype="float32")(D.heat2d), method).compile()
    masks = _masks(r.cuda_source)
    prog = r.load_module().program()
    bufs = {n: (n,) for n in ("u", "s1", "s2", "s3", "acc")}
    for k, name in enumerate(r.info["stages"]):
        inputs, outputs = prog.stage_io(k, bufs, ())
        both = sum(1 << i for i, f in enumerate(inputs) if f in outputs)
        assert masks.get(name, 0) == both, (k, stage_table(method)[k])
        body = r.cuda_source.split(f"struct Body_{name}_direct {{")[1].split("};")[0]
        assert f"rewritten(int f) {{ return {both} >> f & 1; }}" in body


def test_plain_sweeps_rewrite_nothing():
    import cutile

    r = cutile.compile(stencil(ndim=2)(D.heat2d), temporal_blocking=False)
    assert "rewritten(int f) { return 0 >> f & 1; }" in r.cuda_source
    assert not _masks(r.cuda_source)
