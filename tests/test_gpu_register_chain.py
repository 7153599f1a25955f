"""Register chains (1-D and 2-D temporal blocking without shared memory)
against T oracle steps, at the edges of the warps' strips and row windows."""

import numpy as np
import pytest

import stencil_defs as D
from oracle import stencil_oracle as O

pytestmark = pytest.mark.gpu


def along_x(u, i, j):
    return 0.25 * u[i, j - 1] + 0.5 * u[i, j] + 0.25 * u[i, j + 1]


BODIES = {"heat1d": (D.heat1d, 1), "lap4_1d": (D.lap4_1d, 1), "heat2d": (D.heat2d, 2),
          "upwind2d": (D.upwind2d, 2), "wave4": (D.wave4, 2), "along_x": (along_x, 2)}


def _compiled(name, dtype, T, **kw):
    import cutile
    from cutile import stencil

    fn, ndim = BODIES[name]
    r = cutile.compile(stencil(ndim=ndim, dtype=dtype)(fn), temporal_steps=T, **kw)
    assert r.temporal_steps == T and r.kernel_hints["register_chain"] > 0
    return r, fn, ndim


def _launch(r, u, **kw):
    import torch

    t = torch.from_numpy(u).cuda()
    out = torch.full_like(t, float("nan"))
    r.load_module().program().launch([t], [out], **kw)
    torch.cuda.synchronize()
    assert np.array_equal(t.cpu().numpy(), u)   # the input is not modified
    return out.cpu().numpy()


@pytest.mark.parametrize("align_halo", [True, False])
@pytest.mark.parametrize("name,dtype,T", [
    ("heat1d", "float64", 8), ("heat1d", "float32", 2), ("lap4_1d", "float32", 3),
    ("heat2d", "float64", 5), ("heat2d", "float32", 8), ("upwind2d", "float32", 3),
    ("wave4", "float64", 3), ("along_x", "float64", 4)])
def test_strip_and_row_edges(name, dtype, T, align_halo):
    """Widths around whole strips (the aligned and the per-element copies),
    one row to several items of rows, first-step halos that are not zero."""
    r, fn, ndim = _compiled(name, dtype, T, align_halo=align_halo)
    tx = r.load_module().program().kernel().desc["tile_x"]
    rng = np.random.default_rng(T)
    rows = {1: [()], 2: [(1,), (2,), (37,)]}[ndim]
    for inner_rows in rows:
        for nx in (1, tx - 1, tx, tx + 1, 2 * tx + 3):
            shape = tuple(s + 2 * h for s, h in zip(inner_rows + (nx,), r.halo_widths))
            u = rng.standard_normal(shape).astype(dtype)
            want = O.temporal_launch(u, np.full(shape, np.nan, dtype=dtype), fn, ndim,
                                     r.halo_widths, T)
            for zchunk in (0, 5) if ndim == 2 else (0,):
                got = _launch(r, u, zchunk=zchunk)
                assert np.array_equal(got, want, equal_nan=True), (shape, zchunk)


def test_strided_and_offset_fields():
    """A row-pitched view takes the aligned copies up to its ragged end; a
    base that is not 16-byte aligned takes the per-element ones."""
    import torch

    r, fn, _ = _compiled("heat2d", "float32", 8, align_halo=False)
    rng = np.random.default_rng(5)
    shape = (41, 131)
    u = rng.standard_normal(shape).astype(np.float32)
    want = O.temporal_launch(u, np.full(shape, np.nan, np.float32), fn, 2, r.halo_widths, 8)
    prog = r.load_module().program()
    for pitch, offset in ((160, 0), (160, 1), (133, 2)):
        flat = [torch.full((41 * pitch + 8,), float("nan"), device="cuda") for _ in range(2)]
        view = [f.as_strided(shape, (pitch, 1), offset) for f in flat]
        view[0].copy_(torch.from_numpy(u))
        prog.launch([view[0]], [view[1]])
        assert np.array_equal(view[1].cpu().numpy(), want, equal_nan=True), (pitch, offset)
        pad = flat[1].clone()
        pad.as_strided(shape, (pitch, 1), offset).fill_(float("nan"))
        assert torch.isnan(pad).all()          # nothing outside the view is written


def test_batched_chain_equals_single_launches():
    import torch

    from cutile.runtime.rk_runtime import BatchLaunch

    r, _, _ = _compiled("heat2d", "float64", 5)
    prog = r.load_module().program()
    ins, outs, alone = [], [], []
    for k, (ny, nx) in enumerate([(33, 50), (7, 300), (120, 64)]):
        shape = tuple(s + 2 * h for s, h in zip((ny, nx), r.halo_widths))
        ins.append(torch.randn(shape, dtype=torch.float64, device="cuda"))
        outs.append(torch.zeros_like(ins[-1]))
        alone.append(torch.zeros_like(ins[-1]))
        prog.launch([ins[-1]], [alone[-1]])
    per = [{"inputs": [i], "outputs": [o]} for i, o in zip(ins, outs)]
    BatchLaunch(prog.kernel(), per, r.halo_widths, zchunk=16).launch()
    torch.cuda.synchronize()
    for a, b in zip(outs, alone):
        assert torch.equal(a, b)


def skewed(u, i, j, k):
    return (0.5 * u[i, j, k] + 0.25 * u[i + 1, j - 1, k] - 0.125 * u[i, j + 1, k - 1]
            + 0.0625 * u[i - 1, j, k + 1])


@pytest.mark.parametrize("align_halo", [True, False])
@pytest.mark.parametrize("fn,dtype,T", [
    (D.lap7, "float64", 2), (D.lap7, "float32", 3), (D.lap7, "float64", 4), (D.box27, "float64", 2),
    (skewed, "float32", 2)])
def test_3d_tile_edges(fn, dtype, T, align_halo):
    """Columns and rows around whole tiles, one plane to several items of
    planes, halos that are not zero, aligned and per-element copies."""
    import cutile
    from cutile import stencil

    r = cutile.compile(stencil(ndim=3, dtype=dtype)(fn), temporal_steps=T, align_halo=align_halo)
    assert r.temporal_steps == T and r.kernel_hints["chain_rows"] > 0
    d = r.load_module().program().kernel().desc
    tx, ty = d["tile_x"], d["tile_y"]
    rng = np.random.default_rng(T)
    for nz, ny, nx in ((1, 1, 1), (2, ty - 1, tx - 1), (9, ty, tx), (5, ty + 1, tx + 1),
                       (13, 2 * ty + 3, 2 * tx + 5)):
        shape = tuple(s + 2 * h for s, h in zip((nz, ny, nx), r.halo_widths))
        u = rng.standard_normal(shape).astype(dtype)
        want = O.temporal_launch(u, np.full(shape, np.nan, dtype=dtype), fn, 3, r.halo_widths, T)
        for zchunk in (0, 4):
            got = _launch(r, u, zchunk=zchunk)
            assert np.array_equal(got, want, equal_nan=True), (shape, zchunk)


def test_3d_kahan_chain_keeps_both_fields():
    """Two fields (u and its compensation) chained in three dimensions equal
    separate single steps through zero-halo buffers."""
    import torch

    import cutile
    from cutile import stencil

    fn = stencil(ndim=3, dtype="float32")(D.lap7)
    r = cutile.compile(fn, precision="fp32_kahan", temporal_steps=2, kernel_hints={
        "register_chain": 4, "chain_rows": 3, "chain_warps": 8})
    r1 = cutile.compile(fn, precision="fp32_kahan", temporal_blocking=False)
    shape = tuple(s + 2 * h for s, h in zip((9, 40, 150), r.halo_widths))
    inner = tuple(slice(h, s - h) for h, s in zip(r.halo_widths, shape))
    a = [torch.zeros(shape, device="cuda") for _ in range(2)]
    a[0][inner] = torch.randn(a[0][inner].shape, device="cuda")
    a[1][inner] = 1e-8 * torch.randn(a[0][inner].shape, device="cuda")
    got = [torch.zeros_like(x) for x in a]
    r.load_module().launch_lap7(*a, *got)
    for _ in range(2):
        b = [torch.zeros_like(x) for x in a]
        r1.load_module().launch_lap7(*a, *b)
        a = b
    assert torch.equal(got[0], a[0]) and torch.equal(got[1], a[1])


def test_3d_batched_chain_equals_single_launches():
    import torch

    import cutile
    from cutile import stencil
    from cutile.runtime.rk_runtime import BatchLaunch

    r = cutile.compile(stencil(ndim=3)(D.lap7), temporal_steps=2)
    prog = r.load_module().program()
    ins, outs, alone = [], [], []
    for shape in ((9, 40, 70), (30, 5, 33), (3, 29, 61)):
        shape = tuple(s + 2 * h for s, h in zip(shape, r.halo_widths))
        wide = torch.randn(shape[:2] + (-(-shape[2] // 16) * 16,), dtype=torch.float64, device="cuda")
        ins.append(wide[..., :shape[2]])
        outs.append(torch.zeros_like(wide)[..., :shape[2]])
        alone.append(torch.zeros_like(wide)[..., :shape[2]])
        prog.launch([ins[-1]], [alone[-1]])
    per = [{"inputs": [i], "outputs": [o]} for i, o in zip(ins, outs)]
    BatchLaunch(prog.kernel(), per, r.halo_widths, zchunk=7).launch()
    torch.cuda.synchronize()
    for a, b in zip(outs, alone):
        assert torch.equal(a, b)
