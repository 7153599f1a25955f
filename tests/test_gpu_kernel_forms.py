"""Forms that are compiled when a launch wants them: the first launch that does
is as right as the next, and a capture does without."""

import numpy as np
import pytest

import stencil_defs as D
from oracle import stencil_oracle as O

pytestmark = pytest.mark.gpu


def _case(fn, ndim, size, seed=0, **kw):
    import torch

    import cutile
    from cutile import stencil

    r = cutile.compile(stencil(ndim=ndim)(fn), **kw)
    shape = tuple(s + 2 * h for s, h in zip(size, r.halo_widths))
    u = np.random.default_rng(seed).standard_normal(shape)
    T = r.temporal_steps
    want = O.temporal_launch(u, np.full(shape, np.nan), fn, ndim, r.halo_widths, T)
    t = torch.from_numpy(u).cuda()
    return r.load_module().program(), t, torch.full_like(t, float("nan")), want


def _equal(out, want):
    return np.array_equal(out.cpu().numpy(), want, equal_nan=True)


@pytest.mark.parametrize("fn,ndim,size,form,kw", [
    (D.wave4, 2, (41, 67), 1, dict(temporal_blocking=False, align_halo=False)),
    (D.lap7, 3, (9, 33, 40), 2, dict(temporal_steps=2))])
def test_first_launch_attaches_the_form(fn, ndim, size, form, kw):
    prog, t, out, want = _case(fn, ndim, size, **kw)
    kernel = prog.kernel()
    assert form in kernel._missing
    for _ in range(2):
        out.fill_(float("nan"))
        prog.launch([t], [out])
        assert form not in kernel._missing
        assert _equal(out, want)
    assert prog.kernel()._module._forms.keys() == {form}


@pytest.mark.parametrize("fn,ndim,size,form,kw", [
    (D.wave4, 2, (41, 67), 1, dict(temporal_blocking=False, align_halo=False)),
    (D.lap7, 3, (9, 33, 40), 2, dict(temporal_steps=2))])
def test_a_capture_does_without(fn, ndim, size, form, kw):
    import torch

    prog, t, out, want = _case(fn, ndim, size, **kw)
    kernel = prog.kernel()                  # loaded, but not its form
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        prog.launch([t], [out], side)
    assert form in kernel._missing
    out.fill_(float("nan"))
    graph.replay()
    torch.cuda.synchronize()
    assert _equal(out, want)
    out.fill_(float("nan"))
    prog.launch([t], [out])
    assert form not in kernel._missing and _equal(out, want)


@pytest.mark.parametrize("method", ["rk2", "rk4", "ssprk3"])
def test_every_stage_of_a_step_takes_the_direct_form(method):
    """Also the stages that rewrite a field they read."""
    import torch

    from cutile import RKIntegrator, stencil

    r = RKIntegrator(stencil(ndim=2)(D.wave4), method).compile(align_halo=False)
    mod = r.load_module()
    u = torch.randn((41, 67), dtype=torch.float64, device="cuda")
    getattr(mod, f"rk_{method}_step")(u, 0.01)
    torch.cuda.synchronize()
    prog = mod.program()
    assert all(1 not in prog.kernel(k)._missing for k in range(len(prog.table)))


def test_launches_of_several_threads_share_the_form():
    import threading

    import torch

    prog, t, out, want = _case(D.wave4, 2, (301, 1003), temporal_blocking=False, align_halo=False)
    prog.kernel()
    outs = [torch.full_like(t, float("nan")) for _ in range(6)]
    errors = []

    def run(o):
        try:
            for _ in range(3):
                prog.launch([t], [o])
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(e)

    threads = [threading.Thread(target=run, args=(o,)) for o in outs]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    torch.cuda.synchronize()
    assert not errors and all(_equal(o, want) for o in outs)


def test_aot_modules_hold_every_form(tmp_path):
    import torch

    import cutile
    from cutile import stencil
    from cutile.runtime.launcher import load_aot

    r = cutile.compile(stencil(ndim=3)(D.lap7), temporal_steps=2)
    mod = load_aot(r.build_aot(str(tmp_path)).module)
    kernel = mod.program().kernel()
    assert not kernel._missing and kernel.batch_form(0).desc["nslot"] > 0
    t = torch.randn(tuple(s + 2 * h for s, h in zip((9, 33, 40), r.halo_widths)),
                    dtype=torch.float64, device="cuda")
    a, b = torch.zeros_like(t), torch.zeros_like(t)
    mod.launch_lap7(t, a)
    r.load_module().launch_lap7(t, b)
    torch.cuda.synchronize()
    assert torch.equal(a, b)
