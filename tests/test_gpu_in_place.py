"""Outputs that are inputs, at widths whose rows are not aligned."""

import numpy as np
import pytest

import stencil_defs as D

pytestmark = pytest.mark.gpu


def halve(u, i, j):
    return 0.5 * u[i, j] + 1.0


def test_pointwise_launch_in_place():
    """A launch below the public entry points may write its input where the
    body reads its own point only."""
    import torch

    import cutile
    from cutile import stencil
    from cutile.runtime import native

    r = cutile.compile(stencil(ndim=2)(halve), temporal_blocking=False, align_halo=False)
    kernel = r.load_module().program().kernel()
    u = torch.randn((301, 1003), dtype=torch.float64, device="cuda")
    want = 0.5 * u + 1.0
    native.launch(kernel, [u], [u], r.halo_widths)
    torch.cuda.synchronize()
    assert torch.equal(u, want)


@pytest.mark.parametrize("method", ["rk2", "rk4", "ssprk3"])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_rk_steps_at_odd_widths_equal_aligned_ones(method, dtype):
    """The accumulator and the state are rewritten stage by stage: a row-pitched
    copy of the state (staged kernels) takes the same steps."""
    import torch

    from cutile import RKIntegrator, stencil

    r = RKIntegrator(stencil(ndim=2, dtype=dtype)(D.wave4), method).compile(align_halo=False)
    step = getattr(r.load_module(), f"rk_{method}_step")
    rng = np.random.default_rng(2)
    for shape in ((41, 67), (301, 259), (9, 20)):
        u = torch.from_numpy(rng.standard_normal(shape).astype(dtype)).cuda()
        if shape[1] % 2 == 0:
            u = u[:, :-1].contiguous()
        wide = torch.zeros((u.shape[0], u.shape[1] + 64 - u.shape[1] % 64), dtype=u.dtype,
                           device="cuda")
        v = wide[:, :u.shape[1]]
        v.copy_(u)
        for _ in range(3):
            step(u, 0.01)
            step(v, 0.01)
        assert torch.equal(u, v), shape
