"""Runge-Kutta steps on a stream of the caller's: dt, the workspace and the
copy back belong to that stream, whatever the current one is busy with."""

import pytest

import stencil_defs as D

pytestmark = pytest.mark.gpu

BUSY = 20_000_000      # cycles: some 10 ms


def _program(method):
    from cutile import RKIntegrator, stencil

    r = RKIntegrator(stencil(ndim=2, dtype="float64")(D.heat2d), method).compile()
    return r.load_module(), r.info["halo"]


def _state(halo, seed=0):
    import torch

    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(tuple(96 + 2 * h for h in halo), dtype=torch.float64, device="cuda",
                       generator=gen)


DTS = (0.1, 0.2, 0.05)


@pytest.mark.parametrize("method", ["rk2", "rk4", "euler", "ssprk3"])
def test_steps_do_not_wait_for_the_current_stream(method):
    """A new state and a dt of its own in every step while the current stream
    is busy: values that it still has to write must not be needed."""
    import torch

    mod, halo = _program(method)
    step = getattr(mod, f"rk_{method}_step")
    want = _state(halo)
    for dt in DTS:
        step(want, dt)
    u = _state(halo)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    torch.cuda._sleep(BUSY)
    for dt in DTS:
        step(u, dt, stream=side)
    side.synchronize()
    got = u.clone()
    torch.cuda.synchronize()
    assert torch.equal(got, want) and torch.equal(u, want)


def test_steps_on_two_streams_have_their_own_dt():
    import torch

    mod, halo = _program("rk4")
    dts = (0.1, 0.3)
    want = [_state(halo, k) for k in range(2)]
    for u, dt in zip(want, dts):
        for _ in range(40):
            mod.rk_rk4_step(u, dt)
    got = [_state(halo, k) for k in range(2)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(40):
        for u, dt, s in zip(got, dts, streams):
            mod.rk_rk4_step(u, dt, stream=s)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_solve_copies_its_state_on_the_stream():
    import torch

    mod, halo = _program("rk2")
    u = _state(halo)
    want = mod.rk_rk2_solve(u, 0.1, 3)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    torch.cuda._sleep(BUSY)
    got = mod.rk_rk2_solve(u, 0.1, 3, stream=side)
    side.synchronize()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
