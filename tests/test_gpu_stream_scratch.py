"""Scratch of the reductions on streams of the caller's: its own per stream,
filled and read in that stream's order."""

import pytest

pytestmark = pytest.mark.gpu


def _fields(n=3):
    import torch

    gen = torch.Generator(device="cuda").manual_seed(3)
    return [torch.randn((66, 67, 129), dtype=torch.float64, device="cuda", generator=gen)
            for _ in range(n)]


def test_two_streams_share_no_partials(monkeypatch):
    import torch

    from cutile.runtime import native, reductions

    lib, seen = native.library(), []

    class Recorder:
        def csd_reduce(self, *args):
            seen.append(args[4])
            return lib.csd_reduce(*args)

        def __getattr__(self, name):
            return getattr(lib, name)

    monkeypatch.setattr(native, "library", Recorder)
    u = _fields(1)[0]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    got = [reductions.mass(u, (1, 1, 1), stream=s) for s in streams]
    torch.cuda.synchronize()
    assert len(set(seen)) == 2
    assert got[0].item() == got[1].item() == reductions.mass(u, (1, 1, 1)).item()


def test_overlapping_reductions_keep_their_sums():
    import torch

    from cutile.runtime import reductions

    fields = _fields()
    want = [reductions.energy(u, (1, 1, 1)).item() for u in fields]
    streams = [torch.cuda.Stream() for _ in fields]
    torch.cuda.synchronize()
    got = [[reductions.energy(u, (1, 1, 1), stream=s) for u, s in zip(fields, streams)]
           for _ in range(100)]
    torch.cuda.synchronize()
    assert all([x.item() for x in row] == want for row in got)


@pytest.mark.parametrize("as_handle", [False, True])
def test_the_root_of_a_residual_waits_for_its_sum(as_handle):
    import torch

    from cutile.runtime import reductions

    a, b, _ = _fields()
    want = reductions.residual(a, b, (1, 1, 1)).item()
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)       # the side stream is busy for some 10 ms
    got = reductions.residual(a, b, (1, 1, 1), stream=side.cuda_stream if as_handle else side)
    torch.cuda.synchronize()
    assert got.item() == want
