"""Conversions to and from bricks around the row length at which the walk by
elements ends."""

import numpy as np
import pytest

from oracle import stencil_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [1, 12, 63, 64, 65])
@pytest.mark.parametrize("rows,brick", [((301,), 8), ((7, 9), 4), ((33, 18), 16), ((1, 5), 64)])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_short_and_long_rows(rows, nx, brick, dtype):
    """from_bricks walks the array's rows, to_bricks the padded ones: the two
    may take different walks."""
    import torch

    from cutile.runtime import native

    shape = rows + (nx,)
    u = np.random.default_rng(nx).standard_normal(shape).astype(dtype)
    t = torch.from_numpy(u).cuda()
    b = native.to_bricks(t, brick)
    assert np.array_equal(b.cpu().numpy(), O.to_bricks(u, brick))
    out = torch.full_like(t, float("nan"))
    native.from_bricks(b, shape, brick, out=out)
    assert np.array_equal(out.cpu().numpy(), u)
