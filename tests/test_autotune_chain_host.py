"""What the autotuner times is what compile() builds (no GPU): depths above
one are timed as the chains that compile() would use, and a tuned plan is
compiled as it was timed."""

from dataclasses import asdict

import pytest

import cutile
import stencil_defs as D
from cutile import stencil
from cutile.passes.tiling import EnginePlan
from cutile.runtime import autotune as A


def _candidates(fn, ndim, esz):
    fp = A._footprint(fn, esz)
    return fp, A.candidates(ndim, esz, fp["radius"], fp["inputs"], fp["loads"], fp["body_ops"],
                            True, 30, fp["outputs"], A.chain_hints(fp, ndim, esz))


@pytest.mark.parametrize("body,ndim,dtype", [
    (D.heat1d, 1, "float64"), (D.heat2d, 2, "float64"), (D.heat2d, 2, "float32"),
    (D.wave4, 2, "float32"), (D.lap7, 3, "float64"), (D.lap3d, 3, "float32")])
def test_untuned_plans_of_every_depth_are_candidates(body, ndim, dtype):
    op = stencil(ndim=ndim, dtype=dtype)(body)
    esz = 8 if dtype == "float64" else 4
    fp, plans = _candidates(op, ndim, esz)
    assert len(plans) <= 30
    depths = {1, *A._depths(ndim), fp["depth"]}
    assert fp["depth"] == cutile.compile(op).temporal_steps
    for T in sorted(depths - {1}):
        r = cutile.compile(op, temporal_steps=T)
        same = [p for p in plans if p.temporal == T and p.hints() == r.kernel_hints
                and p.tile_sizes() == r.tile_sizes]
        assert len(same) == 1, (T, r.kernel_hints)
        # the probe compiles exactly it
        probe = cutile.compile(op, tile_sizes=same[0].tile_sizes(), temporal_steps=T,
                               kernel_hints=A.probe_hints(same[0]), autotune=False)
        assert probe.cuda_source == r.cuda_source


@pytest.mark.parametrize("chain", [True, False])
def test_a_tuned_plan_is_compiled_as_it_was_timed(monkeypatch, chain):
    op = stencil(ndim=2)(D.heat2d)
    _, plans = _candidates(op, 2, 8)
    plan = next(p for p in plans if p.temporal == 2 and bool(p.register_chain) == chain
                and (chain or p.tile_sizes() != cutile.compile(op, temporal_steps=2).tile_sizes))
    kept = EnginePlan(**asdict(plan))           # as the cache keeps it
    assert kept == plan
    result = A.AutotuneResult(kept.tile_sizes(), kept.temporal, 1.0, 1.0, 1.0, kept.hints(), kept, 1)
    monkeypatch.setattr(A, "autotune", lambda *a, **kw: result)
    r = cutile.compile(op, domain=(512, 512))
    assert r.temporal_steps == 2
    assert r.tile_sizes == plan.tile_sizes() and r.kernel_hints == plan.hints()
    probe = cutile.compile(op, tile_sizes=plan.tile_sizes(), kernel_hints=A.probe_hints(plan),
                           temporal_steps=2, autotune=False)
    assert r.cuda_source == probe.cuda_source
    # a depth of the caller's own is compiled as without a domain
    other = cutile.compile(op, domain=(512, 512), temporal_steps=3)
    assert other.kernel_hints == cutile.compile(op, temporal_steps=3).kernel_hints


def test_bricked_layouts_are_timed_without_register_chains(monkeypatch):
    seen = {}

    def tune(fn, domain, **kw):
        seen.update(kw)
        plan = A.candidates(3, 8, (1, 1, 1), 1, 7, 19, True)[0]
        return A.AutotuneResult(plan.tile_sizes(), 1, 1.0, 1.0, 1.0, plan.hints(), plan, 1)

    monkeypatch.setattr(A, "autotune", tune)
    cutile.compile(stencil(ndim=3)(D.lap7), domain=(64, 64, 64), layout="bricked", brick_size=8)
    assert seen["chains"] is False
    cutile.compile(stencil(ndim=3)(D.lap7), domain=(64, 64, 64))
    assert seen["chains"] is True
