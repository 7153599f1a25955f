"""Launches of one kind share their C arguments: new buffers, values, streams,
shapes and threads must still each get their own."""

import threading

import numpy as np
import pytest

import stencil_defs as D

pytestmark = pytest.mark.gpu


def scaled(u, s, i, j):
    return s * u[i, j] + 0.25 * (u[i - 1, j] + u[i + 1, j])


def _program():
    import cutile
    from cutile import stencil

    return cutile.compile(stencil(ndim=2)(scaled), temporal_blocking=False,
                          align_halo=False).load_module()


def _want(u, s):
    return s * u[1:-1, :] + 0.25 * (u[:-2, :] + u[2:, :])


def test_buffers_values_shapes_and_strides():
    import torch

    m = _program()
    rng = torch.Generator(device="cuda").manual_seed(1)
    keep = []
    for k in range(200):
        shape = (5 + k % 3, 16 + 2 * (k % 5))
        u = torch.randn(shape, generator=rng, device="cuda", dtype=torch.float64)
        if k % 4 < 2:
            u[0::2], u[1::2] = 0.0, -u[1::2].abs()   # 0 * u keeps the scalar's sign here
            u[0::2] = -0.0
        if k % 7 == 0:      # a row-pitched view of the same shape
            wide = torch.zeros(shape[0], shape[1] + 6, device="cuda", dtype=torch.float64)
            wide[:, :shape[1]] = u
            u = wide[:, :shape[1]]
        out = torch.empty_strided(u.shape, u.stride(), dtype=u.dtype, device="cuda").zero_()
        s = (0.0, -0.0, 1.5, float("nan"))[k % 4]
        m.launch_scaled(u, out, s=s)
        keep.append((u, out, s))
    h = m.program().spec["halo"]
    for u, out, s in keep:
        want = _want(u, s)[:, h[1]:u.shape[1] - h[1]]
        got = out[1:-1, h[1]:u.shape[1] - h[1]]
        got, want = got.cpu().numpy(), want.cpu().numpy()
        assert np.array_equal(got, want, equal_nan=True)
        assert np.array_equal(np.signbit(got), np.signbit(want)) or s != s   # -0.0 is not 0.0
    plans = m.program()._plans
    assert len(plans.by_kind) <= plans.LIMIT


def test_refusals_come_before_and_after_a_kind_is_known():
    import torch

    m = _program()
    u = torch.zeros(6, 20, dtype=torch.float64, device="cuda")
    out = torch.zeros_like(u)
    for _ in range(2):
        with pytest.raises(ValueError):
            m.launch_scaled(u, u, s=1.0)
        with pytest.raises(TypeError):
            m.launch_scaled(u.float(), out, s=1.0)
        with pytest.raises(TypeError):
            m.launch_scaled(u.cpu().numpy(), out, s=1.0)
        with pytest.raises(ValueError):
            m.launch_scaled(u, torch.zeros(6, 22, dtype=torch.float64, device="cuda"), s=1.0)
        with pytest.raises(ValueError):
            m.launch_scaled(u.t(), out.t(), s=1.0)
        with pytest.raises(ValueError):
            m.launch_scaled(u.cpu(), out.cpu(), s=1.0)
        with pytest.raises(TypeError):
            m.launch_scaled(u, out)
        m.launch_scaled(u, out, s=1.0)


def test_threads_and_streams():
    import torch

    m = _program()
    shape = (64, 200)
    failures = []

    def work(seed):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            g = torch.Generator(device="cuda").manual_seed(seed)
            for _ in range(30):
                u = torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)
                out = torch.zeros_like(u)
                s = float(seed)
                m.launch_scaled(u, out, s=s)
                h = m.program().spec["halo"][1]
                if not torch.equal(out[1:-1, h:-h], _want(u, s)[:, h:-h]):
                    failures.append(seed)
        stream.synchronize()

    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not failures
