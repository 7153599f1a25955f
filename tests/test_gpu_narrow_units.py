"""Units of less than a 16-byte vector (what long flux bodies run with)."""

import numpy as np
import pytest

import stencil_defs as D
from oracle import stencil_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,ndim,dtype,tile,vec", [
    ("lap7", 3, "float32", (1, 4, 64), 2), ("lap7", 3, "float64", (1, 4, 64), 1),
    ("heat2d", 2, "float32", (8, 32), 2), ("wave4", 2, "float32", (8, 32), 1),
    ("lap4_1d", 1, "float32", (128,), 2)])
@pytest.mark.parametrize("align_halo", [True, False])
def test_narrow_units_are_bit_exact(name, ndim, dtype, tile, vec, align_halo):
    """Ragged tiles, tensor copies and per-element copies (loader 1)."""
    import torch

    import cutile
    from cutile import stencil

    fn = D.CASES[name][0]
    r = cutile.compile(stencil(ndim=ndim, dtype=dtype)(fn), temporal_blocking=False,
                       align_halo=align_halo, tile_sizes=tile,
                       kernel_hints={"vec": vec, "threads": 128})
    assert r.kernel_hints["vec"] == vec
    size = {3: (13, 37, 152), 2: (75, 300), 1: (1000,)}[ndim]
    shape = tuple(s + 2 * h for s, h in zip(size, r.halo_widths))
    u = np.random.default_rng(5).standard_normal(shape).astype(dtype)
    want = np.full(shape, np.nan, dtype)
    inner = tuple(slice(h, s - h) for h, s in zip(r.halo_widths, shape))
    want[inner] = O.apply_stencil(u, fn, ndim, r.halo_widths)[inner]
    t = torch.from_numpy(u).cuda()
    for loader in (-1, 1):
        out = torch.full_like(t, float("nan"))
        r.load_module().program().launch([t], [out], loader=loader)
        assert np.array_equal(out.cpu().numpy(), want, equal_nan=True), loader
