"""The standalone halo fill against the oracle: every condition, halos from
none to as wide as the interior, every dimensionality."""

import numpy as np
import pytest

from oracle import stencil_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bc", ["dirichlet", "neumann", "periodic", "reflecting"])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_halo_fill(bc, dtype):
    import torch

    from cutile.runtime import native

    for shape, halo in (((9,), (3,)), ((70,), (16,)), ((5, 7), (1, 1)), ((20, 131), (2, 32)),
                        ((40, 9), (0, 3)), ((9, 40), (3, 0)), ((6, 7, 8), (1, 2, 2)),
                        ((5, 12, 100), (1, 1, 33)), ((11, 9, 44), (2, 0, 14)), ((7, 9, 5), (0, 1, 0)),
                        ((33, 35, 37), (1, 1, 1)), ((4, 4), (0, 0))):
        u = np.random.default_rng(len(shape)).standard_normal(shape).astype(dtype)
        t = torch.from_numpy(u.copy()).cuda()
        native.apply_boundary(t, halo, bc, 0.75)
        want = u.copy()
        O.apply_boundary(want, O.uniform_spec(bc, len(shape), 0.75), halo)
        assert np.array_equal(t.cpu().numpy(), want), (shape, halo)
