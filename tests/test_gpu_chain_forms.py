"""Register chains and their ring forms: the same bits on either side of the
size at which a launch changes from one to the other, and in batches."""

import numpy as np
import pytest

import stencil_defs as D
from oracle import stencil_oracle as O
from test_chain_form_host import mean9, star2

pytestmark = pytest.mark.gpu


def _compiled(fn, ndim, dtype, T, **kw):
    import cutile
    from cutile import stencil

    return cutile.compile(stencil(ndim=ndim, dtype=dtype)(fn), temporal_steps=T, **kw)


@pytest.mark.parametrize("fn,ndim,dtype,T", [
    (D.lap7, 3, "float64", 2), (D.lap7, 3, "float32", 3), (mean9, 2, "float32", 3),
    (star2, 2, "float32", 2), (D.wave4, 2, "float32", 4)])
@pytest.mark.parametrize("align_halo", [True, False])
def test_either_side_of_the_limit(fn, ndim, dtype, T, align_halo):
    """A row less than the limit and the limit itself (2-D: three ragged tiles of
    128 columns; 3-D: two by two of the chain's), odd rows too; asked for by
    loader or items a launch keeps the chain."""
    import torch

    r = _compiled(fn, ndim, dtype, T, align_halo=align_halo)
    prog = r.load_module().program()
    kern = prog.kernel()
    d, below = kern.desc, r.kernel_hints["ring_below"]
    ring = kern.batch_form(below - 1)
    assert ring.desc["nslot"] > 0 and d["nslot"] == 0
    across = (2 * 128 + 9,) if ndim == 2 else (d["tile_y"] + 1, d["tile_x"] + 9)
    limit = -(-below // (3 if ndim == 2 else 4))
    rng = np.random.default_rng(T)
    for rows in (limit - 1, limit):
        shape = tuple(s + 2 * h for s, h in zip((rows,) + across, r.halo_widths))
        assert (kern.chain_size(shape, r.halo_widths) < below) == (rows < limit)
        u = rng.standard_normal(shape).astype(dtype)
        want = O.temporal_launch(u, np.full(shape, np.nan, dtype=dtype), fn, ndim, r.halo_widths, T)
        t = torch.from_numpy(u).cuda()
        for kw in ({}, {"zchunk": 24}, {"loader": 1}):
            out = torch.full_like(t, float("nan"))
            prog.launch([t], [out], **kw)
            assert np.array_equal(out.cpu().numpy(), want, equal_nan=True), (rows, kw)


@pytest.mark.parametrize("fn,ndim,dtype,T,sides", [
    (D.lap7, 3, "float64", 2, (9, 33, 40)), (D.lap7, 3, "float32", 2, (300, 290, 280)),
    (star2, 2, "float32", 2, (65, 130)), (D.heat2d, 2, "float64", 5, (33, 258, 120))])
def test_batches_take_the_form_for_their_size(fn, ndim, dtype, T, sides):
    import torch

    from cutile.runtime.rk_runtime import BatchLaunch, batch_zchunk, pack_grids

    r = _compiled(fn, ndim, dtype, T, align_halo=False)
    prog = r.load_module().program()
    kern = prog.kernel()
    shapes = [tuple(s + 2 * h + 3 * d for d, h in enumerate(r.halo_widths)) for s in sides]
    _, grids = pack_grids(shapes, 2, getattr(torch, dtype), "cuda")
    per, alone = [], []
    for src, dst in grids:
        src.copy_(torch.randn(src.shape, dtype=src.dtype, device="cuda"))
        per.append({"inputs": [src], "outputs": [dst]})
        alone.append(torch.zeros(src.shape, dtype=src.dtype, device="cuda"))
        prog.launch([src.contiguous()], [alone[-1]], loader=1)
    batch = BatchLaunch(kern, per, r.halo_widths, zchunk=batch_zchunk(kern))
    size = sum(kern.chain_size(s, r.halo_widths) for s in shapes)
    below = r.kernel_hints["ring_below"]
    assert (batch.kernel.desc["nslot"] > 0) == (below > 0 and (ndim < 3 or size < 16 * below))
    batch.launch()
    torch.cuda.synchronize()
    for (_, dst), want in zip(grids, alone):
        assert torch.equal(dst, want)


def test_3d_batches_of_register_chains():
    """A chain asked for by hints has no ring form: its batches are chains."""
    import torch

    from cutile.runtime.rk_runtime import BatchLaunch, pack_grids

    r = _compiled(D.lap7, 3, "float64", 2, align_halo=False, kernel_hints={
        "register_chain": 2, "chain_rows": 2, "chain_warps": 16})
    prog = r.load_module().program()
    _, grids = pack_grids([(11, 42, 72), (32, 7, 35), (5, 31, 63)], 2, torch.float64, "cuda")
    per, alone = [], []
    for src, dst in grids:
        src.copy_(torch.randn(src.shape, dtype=src.dtype, device="cuda"))
        per.append({"inputs": [src], "outputs": [dst]})
        alone.append(torch.zeros(src.shape, dtype=src.dtype, device="cuda"))
        prog.launch([src.contiguous()], [alone[-1]])
    batch = BatchLaunch(prog.kernel(), per, r.halo_widths, zchunk=7)
    assert batch.kernel.desc["nslot"] == 0
    batch.launch()
    torch.cuda.synchronize()
    for (_, dst), want in zip(grids, alone):
        assert torch.equal(dst, want)
