"""Deep 3-D chains of bodies that read no rows beside their own (their depth
is bounded by the registers alone) against oracle steps."""

import numpy as np
import pytest

from oracle import stencil_oracle as O
from test_chain_memory_host import along_x, pointwise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("fn,T", [(along_x, None), (along_x, 5), (pointwise, None)])
def test_default_depth_launches(fn, T, dtype):
    import torch

    import cutile
    from cutile import stencil

    r = cutile.compile(stencil(ndim=3, dtype=dtype)(fn), temporal_steps=T)
    T = r.temporal_steps
    prog = r.load_module().program()
    d = prog.kernel().desc
    rng = np.random.default_rng(T)
    for nz, ny, nx in ((1, 1, 1), (5, d["tile_y"] + 1, d["tile_x"] + 3), (11, 7, 2 * d["tile_x"])):
        shape = tuple(s + 2 * h for s, h in zip((nz, ny, nx), r.halo_widths))
        u = rng.standard_normal(shape).astype(dtype)
        want = O.temporal_launch(u, np.full(shape, np.nan, dtype=dtype), fn, 3, r.halo_widths, T)
        t = torch.from_numpy(u).cuda()
        out = torch.full_like(t, float("nan"))
        prog.launch([t], [out])
        assert np.array_equal(out.cpu().numpy(), want, equal_nan=True), shape
