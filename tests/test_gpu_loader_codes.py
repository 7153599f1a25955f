"""Loader values without a meaning of their own ask for the automatic choice,
in a batch's descriptors as in a launch."""

import ctypes

import pytest

import stencil_defs as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [65, 64])
def test_batch_descriptors_take_any_other_value_as_automatic(width):
    """Descriptors are for the staging kernels, whose tiles start on a vector
    also where the rows do not."""
    import torch

    import cutile
    from cutile import stencil
    from cutile.runtime import native

    r = cutile.compile(stencil(ndim=2, dtype="float32")(D.wave4), temporal_blocking=False,
                       align_halo=False)
    kernel = r.load_module().program().kernel()
    a, b = (torch.zeros((40, width), device="cuda") for _ in range(2))
    built = {}
    for loader in (-1, -2, 2, 7):
        dest = (ctypes.c_ubyte * native.grid_size())()
        used = native.grid_build(kernel, [a], [b], r.halo_widths, ctypes.addressof(dest),
                                 loader=loader)
        built[loader] = (used, bytes(dest))
    assert built[-1][0][1] == (native.CSD_LOADER_TMA if width == 64 else native.CSD_LOADER_LDG)
    assert all(v == built[-1] for v in built.values())
