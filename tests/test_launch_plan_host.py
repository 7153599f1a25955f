"""Launch plans over a stand-in library (no GPU): a kept plan refuses what a
new one refuses."""

from types import SimpleNamespace

import pytest

from cutile.runtime import native


@pytest.fixture
def launch(monkeypatch):
    import torch

    calls = []

    def csd_launch(kernel, fin, nin, fout, nout, opts, stream):
        calls.append((opts._obj.zchunk, opts._obj.grid, opts._obj.loader, list(opts._obj.bc_odd)))
        return 0

    monkeypatch.setattr(native, "library", lambda: SimpleNamespace(csd_launch=csd_launch))
    monkeypatch.setattr(native, "stream_handle", lambda stream, device: None)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    plans = native.LaunchPlans()
    u, v = (torch.zeros(8, 8) for _ in range(2))

    class Kernel(native.NativeKernel):
        handle = None

        def __init__(self):
            pass

    def run(**kw):
        native.launch(Kernel(), [u], [v], (1, 1), plans=plans, kind="main",
                      describe=lambda t: native.Field(t.data_ptr(), 2, 1), **kw)
        return calls[-1]

    run.plans = plans
    return run


@pytest.mark.parametrize("good,bad", [
    ({"zchunk": 4}, {"zchunk": 4.0}), ({"grid": 2}, {"grid": 2.0}), ({"loader": 1}, {"loader": 1.0}),
    ({"timeout_ns": 5}, {"timeout_ns": 5.0})])
def test_options_of_another_type_are_refused_after_a_good_launch(launch, good, bad):
    with pytest.raises(TypeError):
        launch(**bad)
    launch(**good)
    launch(**good)
    assert len(launch.plans.by_kind) == 1
    with pytest.raises(TypeError):
        launch(**bad)


def test_equal_options_share_a_plan(launch):
    assert launch(zchunk=4, bc_odd=(1, 0))[3][:2] == [1, 0]
    assert launch(zchunk=4, bc_odd=(1, 0))[0] == 4
    assert launch(zchunk=5, bc_odd=(0, 2))[3][:2] == [0, 2]
    assert len(launch.plans.by_kind) == 2
