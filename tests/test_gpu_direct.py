"""Rows whose pitch is not a multiple of 16 bytes: the direct kernels against
the oracle at the edges of a warp's points, and against the ring kernels."""

import numpy as np
import pytest

import stencil_defs as D
from oracle import stencil_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,ndim,dtype", [
    ("heat1d", 1, "float32"), ("lap4_1d", 1, "float64"), ("heat2d", 2, "float32"),
    ("wave4", 2, "float64"), ("advect2d", 2, "float64"), ("lap7", 3, "float32"),
    ("lap7", 3, "float64"), ("box27", 3, "float64"), ("box27", 3, "float32"),
    ("cond3d", 3, "float32")])
def test_row_widths_around_a_warps_points(name, ndim, dtype):
    """One point to several warps per row, odd pitches (aligned ones take the
    tensor copies), one row to several items and blocks of rows; the ring
    kernel asked for by name gives the same bits."""
    import torch

    import cutile
    from cutile import stencil

    fn = D.CASES[name][0]
    r = cutile.compile(stencil(ndim=ndim, dtype=dtype)(fn), temporal_blocking=False,
                       align_halo=False)
    prog = r.load_module().program()
    rng = np.random.default_rng(3)
    outer = {1: [()], 2: [(1,), (29,)], 3: [(1, 1), (3, 7), (19, 18)]}[ndim]
    for rows in outer:
        for nx in (1, 31, 33, 63, 65, 127, 129, 255, 257):
            shape = tuple(s + 2 * h for s, h in zip(rows + (nx,), r.halo_widths))
            u = rng.standard_normal(shape).astype(dtype)
            want = np.full(shape, np.nan, dtype=dtype)
            inner = tuple(slice(h, s - h) for h, s in zip(r.halo_widths, shape))
            want[inner] = O.apply_stencil(u, fn, ndim, r.halo_widths)[inner]
            t = torch.from_numpy(u).cuda()
            for kw in ({}, {"zchunk": 3}, {"loader": 1}):
                out = torch.full_like(t, float("nan"))
                prog.launch([t], [out], **kw)
                assert np.array_equal(out.cpu().numpy(), want, equal_nan=True), (shape, kw)


def test_unaligned_bases_and_pitches():
    """Fields at any element offset, outputs at another one, rows of any
    pitch; nothing outside the interior is written."""
    import torch

    import cutile
    from cutile import stencil

    r = cutile.compile(stencil(ndim=2, dtype="float32")(D.heat2d), temporal_blocking=False,
                       align_halo=False)
    prog = r.load_module().program()
    shape = (23, 203)
    u = np.random.default_rng(4).standard_normal(shape).astype(np.float32)
    want = np.full(shape, np.nan, np.float32)
    want[1:-1, 1:-1] = O.apply_stencil(u, D.heat2d, 2, (1, 1))[1:-1, 1:-1]
    for pitch, a, b in ((203, 0, 0), (205, 1, 3), (208, 1, 0), (207, 2, 1)):
        flat = [torch.full((23 * pitch + 8,), float("nan"), device="cuda") for _ in range(2)]
        src, dst = flat[0].as_strided(shape, (pitch, 1), a), flat[1].as_strided(shape, (pitch, 1), b)
        src.copy_(torch.from_numpy(u))
        prog.launch([src], [dst])
        assert np.array_equal(dst.cpu().numpy(), want, equal_nan=True), (pitch, a, b)
        dst.fill_(float("nan"))
        assert torch.isnan(flat[1]).all()


@pytest.mark.parametrize("method", ["rk4", "ssprk3"])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_rk_stages_on_odd_widths(method, dtype):
    """Stage kernels with several inputs and outputs read at their centre."""
    import torch

    from cutile import RKIntegrator, stencil

    rk = RKIntegrator(stencil(ndim=2, dtype=dtype)(D.heat2d), method).compile(align_halo=False)
    h = rk.info["halo"]
    shape = (40 + 2 * h[0], 131 + 2 * h[1])
    u0 = np.zeros(shape, dtype)
    inner = tuple(slice(x, s - x) for x, s in zip(h, shape))
    u0[inner] = np.random.default_rng(3).random((40, 131))
    t = torch.from_numpy(u0.copy()).cuda()
    step = getattr(rk.load_module(), f"rk_{method}_step")
    want = (u0,)
    for _ in range(2):
        step(t, 0.1)
        want = O.rk_step(D.heat2d, ["u"], want, method, 0.1, 2, h)
    assert np.array_equal(t.cpu().numpy()[inner], want[0][inner])


def test_max_reduction_on_odd_widths():
    import torch

    import cutile
    from cutile import stencil

    r = cutile.compile(stencil(ndim=2, dtype="float32")(D.sw_speed), reduce="max", align_halo=False)
    rng = np.random.default_rng(6)
    f = [(rng.random((37, 150)) + 0.5).astype(np.float32) for _ in range(3)]
    t = [torch.from_numpy(x[:, :149].copy()).cuda() for x in f]
    got = r.load_module().reduce_sw_speed(*t).item()
    h, hu, hv = (x[:, :149] for x in f)
    want = np.maximum(np.abs(hu / h), np.abs(hv / h)) + np.sqrt(np.float32(D.G_SW) * h)
    hz, hx = r.halo_widths
    assert got == float(want[hz:37 - hz, hx:149 - hx].max())
