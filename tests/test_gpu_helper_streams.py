"""Scratch of the helpers that take a stream (max reductions, bricked launches
of flat arrays): prepared on that stream, whatever the current one runs."""

import pytest

import stencil_defs as D

pytestmark = pytest.mark.gpu

BUSY = 20_000_000      # cycles: some 10 ms


def magnitude(u, i, j):
    return abs(u[i, j])


def test_max_reduction_starts_from_its_own_zero():
    import torch

    import cutile
    from cutile import stencil

    r = cutile.compile(stencil(ndim=2)(magnitude), reduce="max", align_halo=False)
    mod = r.load_module()
    u = torch.randn((70, 90), dtype=torch.float64, device="cuda")
    want = mod.reduce_magnitude(u).item()
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    torch.cuda._sleep(BUSY)
    got = mod.reduce_magnitude(u, stream=side)
    torch.cuda.synchronize()
    assert got.item() == want > 0.0


def test_bricked_launch_of_flat_arrays():
    import torch

    import cutile
    from cutile import stencil

    r = cutile.compile(stencil(ndim=3, dtype="float32")(D.lap7), temporal_blocking=False,
                       layout="bricked", brick_size=8)
    mod = r.load_module()
    u = torch.randn((26, 42, 50), device="cuda")
    want = torch.full_like(u, 7.0)
    mod.launch_lap7_bricked(u, want)
    side = torch.cuda.Stream()
    for _ in range(4):      # blocks that the copies will reuse hold NaN
        dirty = [torch.full((32, 48, 56), float("nan"), device="cuda") for _ in range(4)]
        with torch.cuda.stream(side):
            dirty += [torch.full((32, 48, 56), float("nan"), device="cuda") for _ in range(4)]
        torch.cuda.synchronize()
        del dirty
        torch.cuda._sleep(BUSY)
        got = torch.empty_like(u)
        mod.launch_lap7_bricked(u, got, stream=side)
        side.synchronize()
        torch.cuda.synchronize()
        assert torch.equal(got, want)
