"""Device memory of finished solves goes back with the budget."""

import pytest

import stencil_defs as D

pytestmark = pytest.mark.gpu


def test_nothing_of_the_solves_stays_allocated():
    import torch

    from cutile.runtime.serving import SolveRequest, StencilServer

    reqs = [SolveRequest(kind, "float64", (258, 258), 5)
            for kind in ("heat2d", "upwind2d", "wave2d") for _ in range(4)]
    server = StencilServer(D.serving_kinds(), budget_bytes=1 << 28)
    per = server.memory_of(reqs[0])
    server.run(reqs[:1], realtime=False, keep_state=False)    # pools and group lists
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    server.run(reqs, realtime=False, keep_state=False)
    torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() - before < per
