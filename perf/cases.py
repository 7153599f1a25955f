"""Timed cases of the stencil framework, each through its public entry points.

``listed()`` names the cases, ``draw(rng)`` makes more of the same ranges,
``prepare`` builds what a program holds before the call (compiled modules,
fields, handles), ``run`` is one pass, ``work`` the bytes and operations a
pass cannot do without, ``exact`` the same result in 64-bit torch arithmetic.

Families (``case["family"]``):

* ``march``      1-D / 2-D time loops with ``compile()``'s defaults (one
                 ``launch_<name>`` advances ``temporal_steps`` steps);
* ``sweep``      one launch of a 3-D body, single-step or chained;
* ``gray_scott`` fused two-field steps with the periodic fill fused in;
* ``rk``         RK4 steps of a wide 2-D operator on one grid;
* ``sw_batch``   many shallow-water grids of uneven sizes advanced together;
* ``bricked``    a field taken to bricks, swept there, and taken back;
* ``diagnose``   a periodic step with its halo fill and global reductions;
* ``serve``      a queue of mixed solve requests run by the solve server.
"""

import functools
import math
import os
import random
import sys
import types

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "cutile-stencil-dsl_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import cutile  # noqa: E402
from cutile import RKIntegrator, compile_fused, stencil  # noqa: E402
from cutile.runtime import reductions  # noqa: E402
from cutile.runtime.rk_runtime import RKBatch, pack_grids  # noqa: E402
from cutile.runtime.serving import SolveKind, SolveRequest, StencilServer  # noqa: E402

# --------------------------------------------------------------------------- #
# Stencil bodies
# --------------------------------------------------------------------------- #


def heat1d(u, i):
    return 0.25 * u[i - 1] + 0.5 * u[i] + 0.25 * u[i + 1]


def heat2d(u, i, j):
    return 0.25 * (u[i - 1, j] + u[i + 1, j] + u[i, j - 1] + u[i, j + 1])


def lap7(u, i, j, k):
    return u[i, j, k] + 0.1 * (u[i - 1, j, k] + u[i + 1, j, k] + u[i, j - 1, k] + u[i, j + 1, k]
                               + u[i, j, k - 1] + u[i, j, k + 1] - 6 * u[i, j, k])


def box27(u, i, j, k):
    return (0.3 * u[i, j, k]
            + 0.05 * (u[i - 1, j, k] + u[i + 1, j, k] + u[i, j - 1, k] + u[i, j + 1, k]
                      + u[i, j, k - 1] + u[i, j, k + 1])
            + 0.02 * (u[i - 1, j - 1, k] + u[i - 1, j + 1, k] + u[i + 1, j - 1, k]
                      + u[i + 1, j + 1, k] + u[i - 1, j, k - 1] + u[i - 1, j, k + 1]
                      + u[i + 1, j, k - 1] + u[i + 1, j, k + 1] + u[i, j - 1, k - 1]
                      + u[i, j - 1, k + 1] + u[i, j + 1, k - 1] + u[i, j + 1, k + 1])
            + 0.01 * (u[i - 1, j - 1, k - 1] + u[i - 1, j - 1, k + 1] + u[i - 1, j + 1, k - 1]
                      + u[i - 1, j + 1, k + 1] + u[i + 1, j - 1, k - 1] + u[i + 1, j - 1, k + 1]
                      + u[i + 1, j + 1, k - 1] + u[i + 1, j + 1, k + 1]))


DU, DV, F_GS, K_GS = 0.16, 0.08, 0.037, 0.06


def gs_u(u, v, i, j):
    return u[i, j] + (DU * (u[i - 1, j] + u[i + 1, j] + u[i, j - 1] + u[i, j + 1] - 4 * u[i, j])
                      - u[i, j] * v[i, j] * v[i, j] + F_GS * (1.0 - u[i, j]))


def gs_v(u, v, i, j):
    return v[i, j] + (DV * (v[i - 1, j] + v[i + 1, j] + v[i, j - 1] + v[i, j + 1] - 4 * v[i, j])
                      + u[i, j] * v[i, j] * v[i, j] - (F_GS + K_GS) * v[i, j])


def lap4(u, i, j):
    return (16.0 * (u[i - 1, j] + u[i + 1, j] + u[i, j - 1] + u[i, j + 1])
            - (u[i - 2, j] + u[i + 2, j] + u[i, j - 2] + u[i, j + 2]) - 60.0 * u[i, j]) / 12.0


def upwind2d(u, i, j):
    return u[i, j] - 0.4 * (u[i, j] - u[i, j - 1]) - 0.2 * (u[i, j] - u[i - 1, j])


def leapfrog(u, up, i, j):
    return 2.0 * u[i, j] - up[i, j] + 0.25 * (u[i - 1, j] + u[i + 1, j] + u[i, j - 1]
                                              + u[i, j + 1] - 4.0 * u[i, j])


G_SW = 9.81


def sw_rhs(h, hu, hv, dx, i, j):
    hC = h[i, j]; huC = hu[i, j]; hvC = hv[i, j]
    hE = h[i, j + 1]; huE = hu[i, j + 1]; hvE = hv[i, j + 1]
    hW = h[i, j - 1]; huW = hu[i, j - 1]; hvW = hv[i, j - 1]
    hN = h[i + 1, j]; huN = hu[i + 1, j]; hvN = hv[i + 1, j]
    hS = h[i - 1, j]; huS = hu[i - 1, j]; hvS = hv[i - 1, j]
    uC = huC / hC; vC = hvC / hC; cC = sqrt(G_SW * hC)  # noqa: F821
    uE = huE / hE; cE = sqrt(G_SW * hE)  # noqa: F821
    uW = huW / hW; cW = sqrt(G_SW * hW)  # noqa: F821
    vN = hvN / hN; cN = sqrt(G_SW * hN)  # noqa: F821
    vS = hvS / hS; cS = sqrt(G_SW * hS)  # noqa: F821
    pC = 0.5 * G_SW * hC * hC
    fuC = huC * uC + pC; fvC = huC * vC
    fuE = huE * uE + 0.5 * G_SW * hE * hE; fvE = hvE * uE
    fuW = huW * uW + 0.5 * G_SW * hW * hW; fvW = hvW * uW
    guC = hvC * uC; gvC = hvC * vC + pC
    guN = huN * vN; gvN = hvN * vN + 0.5 * G_SW * hN * hN
    guS = huS * vS; gvS = hvS * vS + 0.5 * G_SW * hS * hS
    aE = max(abs(uC) + cC, abs(uE) + cE)
    aW = max(abs(uW) + cW, abs(uC) + cC)
    bN = max(abs(vC) + cC, abs(vN) + cN)
    bS = max(abs(vS) + cS, abs(vC) + cC)
    FhE = 0.5 * (huC + huE) - 0.5 * aE * (hE - hC)
    FhW = 0.5 * (huW + huC) - 0.5 * aW * (hC - hW)
    FuE = 0.5 * (fuC + fuE) - 0.5 * aE * (huE - huC)
    FuW = 0.5 * (fuW + fuC) - 0.5 * aW * (huC - huW)
    FvE = 0.5 * (fvC + fvE) - 0.5 * aE * (hvE - hvC)
    FvW = 0.5 * (fvW + fvC) - 0.5 * aW * (hvC - hvW)
    GhN = 0.5 * (hvC + hvN) - 0.5 * bN * (hN - hC)
    GhS = 0.5 * (hvS + hvC) - 0.5 * bS * (hC - hS)
    GuN = 0.5 * (guC + guN) - 0.5 * bN * (huN - huC)
    GuS = 0.5 * (guS + guC) - 0.5 * bS * (huC - huS)
    GvN = 0.5 * (gvC + gvN) - 0.5 * bN * (hvN - hvC)
    GvS = 0.5 * (gvS + gvC) - 0.5 * bS * (hvC - hvS)
    return (-(FhE - FhW) / dx - (GhN - GhS) / dx,
            -(FuE - FuW) / dx - (GuN - GuS) / dx,
            -(FvE - FvW) / dx - (GvN - GvS) / dx)


def sw_speed(h, hu, hv, i, j):
    return max(abs(hu[i, j] / h[i, j]), abs(hv[i, j] / h[i, j])) + sqrt(G_SW * h[i, j])  # noqa: F821


# body -> (function, array dimensions, stencil radius, operations per point)
BODIES = {"heat1d": (heat1d, 1, 1, 5), "heat2d": (heat2d, 2, 1, 4), "lap7": (lap7, 3, 1, 10),
          "box27": (box27, 3, 1, 30)}
# served kinds: (function, array dimensions, state fields, operations per point)
SERVED = {"heat2d": (heat2d, 2, 1, 4), "upwind2d": (upwind2d, 2, 1, 6),
          "wave2d": (leapfrog, 2, 2, 9), "lap7": (lap7, 3, 1, 10)}

_TORCH = {"float64": torch.float64, "float32": torch.float32}
_BYTES = {"float64": 8, "float32": 4}

# --------------------------------------------------------------------------- #
# The cases
# --------------------------------------------------------------------------- #


def listed():
    return [
        # The smallest call: one default launch (eight chained steps) of a
        # short 1-D rod, where the call itself costs more than the device.
        dict(name="heat1d_small_fp64", family="march", body="heat1d", dtype="float64", n=2000,
             steps=8),
        # The usual 2-D time loop: 1024 x 1024 for 100 steps with compile()'s
        # defaults (20 launches of five chained steps).
        dict(name="heat2d_1024_fp64", family="march", body="heat2d", dtype="float64", n=1024,
             steps=100),
        # RK4 on a single grid whose width is no multiple of a vector, with a
        # radius-2 operator in single precision.
        dict(name="rk4_ragged_fp32", family="rk", dtype="float32", ny=1537, nx=2049, steps=3),
        # The headline sweep: 7-point, 512^3, double precision.
        dict(name="lap7_512_fp64", family="sweep", body="lap7", dtype="float64", nz=512, ny=512,
             nx=512, chain=1),
        # An odd-sized domain in single precision: rows of any length.
        dict(name="lap7_ragged_fp32", family="sweep", body="lap7", dtype="float32", nz=301,
             ny=411, nx=523, chain=1),
        # Two steps chained per launch, the 3-D temporally blocked option.
        dict(name="lap7_chain2_fp64", family="sweep", body="lap7", dtype="float64", nz=384,
             ny=384, nx=384, chain=2),
        # The wide tier: a dense 27-point box.
        dict(name="box27_384_fp64", family="sweep", body="box27", dtype="float64", nz=384,
             ny=384, nx=384, chain=1),
        # Reaction-diffusion on a large periodic grid with compensated single
        # precision, the fused multi-field step.
        dict(name="gray_scott_4096_kahan", family="gray_scott", precision="fp32_kahan", n=4096,
             steps=4),
        # An ensemble of shallow-water runs of uneven sizes: one launch per
        # RK2 stage, dt from a device reduction, replayed from a CUDA graph.
        dict(name="sw_batch_fp32", family="sw_batch", dtype="float32", grids=20, largest=1536,
             steps=10),
        # The bricked layout: in, four sweeps on resident bricks, and out.
        dict(name="bricked8_320_fp64", family="bricked", dtype="float64", brick=8, nz=320,
             ny=320, nx=320, sweeps=4),
        # One monitored step of a periodic solver: halo fill, sweep, total
        # mass and step residual.
        dict(name="diagnose_periodic_fp64", family="diagnose", dtype="float64", nz=300, ny=320,
             nx=340),
        # The solve server on a queue of mixed 2-D and 3-D requests in both
        # precisions.
        dict(name="serve_mix", family="serve", requests=24, largest=768, longest=60),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims3(rng, lo, hi):
    return {k: _log_int(rng, lo, hi) for k in ("nz", "ny", "nx")}


def draw(rng: random.Random):
    family = rng.choice(["march1", "march2", "rk", "sweep", "sweep", "sweep", "gray_scott",
                         "sw_batch", "bricked", "diagnose", "serve"])
    dtype = rng.choice(["float64", "float32"])
    if family == "march1":
        return dict(family="march", body="heat1d", dtype=dtype, n=_log_int(rng, 1000, 4_000_000),
                    steps=8 * rng.randint(1, 4))
    if family == "march2":
        return dict(family="march", body="heat2d", dtype=dtype, n=_log_int(rng, 64, 2048),
                    steps=10 * rng.randint(1, 10))
    if family == "rk":
        return dict(family="rk", dtype=dtype, ny=_log_int(rng, 100, 2048),
                    nx=_log_int(rng, 100, 2048), steps=rng.randint(1, 4))
    if family == "sweep":
        body, chain = rng.choice([("lap7", 1), ("lap7", 1), ("lap7", 2), ("box27", 1)])
        if body == "box27":
            dtype = "float64"
        return dict(family="sweep", body=body, dtype=dtype, chain=chain, **_dims3(rng, 32, 480))
    if family == "gray_scott":
        return dict(family="gray_scott", precision=rng.choice(["fp32_kahan", "fp64", "fp32"]),
                    n=_log_int(rng, 200, 4096), steps=rng.randint(1, 4))
    if family == "sw_batch":
        return dict(family="sw_batch", dtype=dtype, grids=rng.randint(4, 20),
                    largest=_log_int(rng, 200, 1536), steps=rng.randint(2, 10))
    if family == "bricked":
        return dict(family="bricked", dtype=dtype, brick=rng.choice([8, 16]),
                    sweeps=rng.randint(1, 4), **_dims3(rng, 48, 320))
    if family == "diagnose":
        return dict(family="diagnose", dtype=dtype, **_dims3(rng, 48, 360))
    return dict(family="serve", requests=rng.randint(6, 24), largest=_log_int(rng, 128, 768),
                longest=rng.randint(10, 60))


# --------------------------------------------------------------------------- #
# Compiled modules (compiled once and kept, as a program does)
# --------------------------------------------------------------------------- #


@functools.lru_cache(maxsize=None)
def _compiled(body, dtype, chain=None):
    fn, ndim, _, _ = BODIES[body]
    op = stencil(ndim=ndim, dtype=dtype)(fn)
    if chain is None:
        return cutile.compile(op)
    return cutile.compile(op, temporal_blocking=chain > 1,
                          temporal_steps=chain if chain > 1 else None)


@functools.lru_cache(maxsize=None)
def _gray_scott(precision):
    return compile_fused([stencil(ndim=2)(gs_u), stencil(ndim=2)(gs_v)], precision=precision,
                         boundary="periodic")


@functools.lru_cache(maxsize=None)
def _rk4(dtype):
    return RKIntegrator(stencil(ndim=2, dtype=dtype)(lap4), "rk4").compile()


@functools.lru_cache(maxsize=None)
def _shallow_water(dtype):
    rk = RKIntegrator(stencil(ndim=2, dtype=dtype)(sw_rhs), "rk2").compile(
        boundary="reflecting", align_halo=False)
    speed = cutile.compile(stencil(ndim=2, dtype=dtype)(sw_speed), reduce="max", align_halo=False)
    return rk, speed


@functools.lru_cache(maxsize=None)
def _bricked(dtype, brick):
    return cutile.compile(stencil(ndim=3, dtype=dtype)(lap7), temporal_blocking=False,
                          layout="bricked", brick_size=brick)


@functools.lru_cache(maxsize=None)
def _periodic(dtype):
    return cutile.compile(stencil(ndim=3, dtype=dtype, boundary="periodic")(lap7),
                          temporal_blocking=False)


@functools.lru_cache(maxsize=None)
def _served_kinds():
    return tuple(SolveKind(name, {dt: cutile.compile(stencil(ndim=ndim, dtype=dt)(fn),
                                                     temporal_blocking=False, align_halo=False)
                                  for dt in ("float32", "float64")}, nstate)
                 for name, (fn, ndim, nstate, _) in SERVED.items())


def _call(result, prefix):
    return getattr(result.load_module(), f"{prefix}_{result.name}")


# --------------------------------------------------------------------------- #
# Inputs
# --------------------------------------------------------------------------- #


def _inner(shape, halo):
    return tuple(slice(h, s - h) for h, s in zip(halo, shape))


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _field(interior, halo, dtype, gen, *, fill_halo=False, offset=0.0, scale=1.0):
    """offset + scale * normal values in the interior (``fill_halo``: in the
    halo too, as fixed boundary data); a zero halo otherwise."""
    shape = tuple(n + 2 * h for n, h in zip(interior, halo))
    if fill_halo:
        return torch.randn(shape, generator=gen, device="cuda",
                           dtype=_TORCH[dtype]).mul_(scale).add_(offset)
    u = torch.zeros(shape, dtype=_TORCH[dtype], device="cuda")
    u[_inner(shape, halo)] = torch.randn(tuple(interior), generator=gen, device="cuda",
                                         dtype=_TORCH[dtype]).mul_(scale).add_(offset)
    return u


def _interior(case):
    if case["family"] == "march":
        return (case["n"],) * BODIES[case["body"]][1]
    if case["family"] == "rk":
        return (case["ny"], case["nx"])
    if case["family"] == "gray_scott":
        return (case["n"],) * 2
    return (case["nz"], case["ny"], case["nx"])


def _gs_init(n, halo, dtype, seed):
    """u = 1, v = 0 with twenty seeded squares of u = 0.5, v = 0.25 (+-1 %)."""
    rng = np.random.default_rng(seed)
    gen = _gen(seed)
    shape = (n + 2 * halo[0], n + 2 * halo[1])
    u = torch.ones(shape, dtype=_TORCH[dtype], device="cuda")
    v = torch.zeros(shape, dtype=_TORCH[dtype], device="cuda")
    for _ in range(20):
        y, x = (int(t) for t in rng.integers(0, n - 32, size=2))
        sl = (slice(halo[0] + y, halo[0] + y + 32), slice(halo[1] + x, halo[1] + x + 32))
        noise = torch.rand((2, 32, 32), generator=gen, device="cuda", dtype=torch.float64)
        u[sl] = (0.5 * (0.99 + 0.02 * noise[0])).to(u.dtype)
        v[sl] = (0.25 * (0.99 + 0.02 * noise[1])).to(v.dtype)
    return u, v


def _sw_sizes(case):
    """Grid widths spread over the logarithm of [64, largest] (the same for
    every seed: an ensemble keeps its members)."""
    g = case["grids"]
    ratio = case["largest"] / 64.0
    return [int(round(64.0 * ratio ** (k / (g - 1)))) for k in range(g)]


def _sw_init(n, rng, dtype):
    """h = 1 + 0.1 * Gaussian bump at a random centre, fluid at rest."""
    y = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n
    cy, cx = (float(t) for t in rng.uniform(0.2, 0.8, size=2))
    h = torch.ones((n + 2, n + 2), dtype=torch.float64, device="cuda")
    h[1:-1, 1:-1] = 1.0 + 0.1 * torch.exp(-((y[:, None] - cy) ** 2 + (y[None, :] - cx) ** 2)
                                          / (2 * 0.05 ** 2))
    h = h.to(_TORCH[dtype])
    return h, torch.zeros_like(h), torch.zeros_like(h)


def _serve_specs(case):
    """(kind, dtype, interior extent, steps) of every request: kinds and
    precisions in turn, sizes and step counts over their ranges."""
    rng = random.Random(case["requests"] * 1009 + case["largest"] * 31 + case["longest"])
    names = list(SERVED)
    specs = []
    for q in range(case["requests"]):
        kind = names[q % len(names)]
        if SERVED[kind][1] == 3:
            m = _log_int(rng, 24, max(25, case["largest"] // 6))
        else:
            m = _log_int(rng, 64, case["largest"])
        specs.append((kind, ("float32", "float64")[(q // 4) % 2], m,
                      rng.randint(5, case["longest"])))
    return specs


def _serve_fields(case, seed):
    """Initial state of every request (newest first), zero halo of one cell."""
    gen = _gen(seed)
    out = []
    for kind, dtype, m, _ in _serve_specs(case):
        ndim = SERVED[kind][1]
        u = torch.zeros((m + 2,) * ndim, dtype=_TORCH[dtype], device="cuda")
        u[(slice(1, -1),) * ndim] = torch.rand((m,) * ndim, generator=gen, device="cuda",
                                               dtype=_TORCH[dtype])
        out.append((u,) * SERVED[kind][2])
    return out


def _inputs(case, seed):
    """The seeded input fields of the case, laid out for its module."""
    family = case["family"]
    gen = _gen(seed)
    if family == "march":
        return _field(_interior(case), _compiled(case["body"], case["dtype"]).halo_widths,
                      case["dtype"], gen)
    if family == "sweep":
        halo = _compiled(case["body"], case["dtype"], case["chain"]).halo_widths
        return _field(_interior(case), halo, case["dtype"], gen, fill_halo=True)
    if family == "rk":
        return _field(_interior(case), _rk4(case["dtype"]).info["halo"], case["dtype"], gen)
    if family == "bricked":
        halo = _bricked(case["dtype"], case["brick"]).halo_widths
        return _field(_interior(case), halo, case["dtype"], gen)
    if family == "diagnose":
        return _field(_interior(case), _periodic(case["dtype"]).halo_widths, case["dtype"], gen,
                      offset=1.0, scale=0.1)
    if family == "gray_scott":
        dtype = "float64" if case["precision"] == "fp64" else "float32"
        return _gs_init(case["n"], _gray_scott(case["precision"]).halo_widths, dtype, seed)
    if family == "sw_batch":
        rng = np.random.default_rng(seed)
        return [_sw_init(n, rng, case["dtype"]) for n in _sw_sizes(case)]
    return _serve_fields(case, seed)


# --------------------------------------------------------------------------- #
# One pass
# --------------------------------------------------------------------------- #


def prepare(case, seed):
    family = case["family"]
    s = dict(case=case, family=family)
    x = _inputs(case, seed)
    if family == "march":
        r = _compiled(case["body"], case["dtype"])
        s.update(launch=_call(r, "launch"), u=x, a=torch.zeros_like(x), b=torch.zeros_like(x),
                 launches=-(-case["steps"] // r.temporal_steps))
    elif family == "sweep":
        r = _compiled(case["body"], case["dtype"], case["chain"])
        s.update(launch=_call(r, "launch"), u=x, out=torch.zeros_like(x))
    elif family == "rk":
        r = _rk4(case["dtype"])
        s.update(step=r.load_module().rk_rk4_step, u0=x, u=torch.zeros_like(x))
    elif family == "gray_scott":
        r = _gray_scott(case["precision"])
        first = list(x)
        if case["precision"] == "fp32_kahan":
            first += [torch.zeros_like(t) for t in x]
        s.update(step=_call(r, "step"), first=first, a=[torch.zeros_like(t) for t in first],
                 b=[torch.zeros_like(t) for t in first])
    elif family == "sw_batch":
        rk, speed = _shallow_water(case["dtype"])
        flat, states = pack_grids([g[0].shape for g in x], 3, _TORCH[case["dtype"]], "cuda")
        for st, g in zip(states, x):
            for dst, src in zip(st, g):
                dst.copy_(src)
        dx = [1.0 / n for n in _sw_sizes(case)]
        batch = RKBatch(rk, states, [{"dx": d} for d in dx],
                        cfl=(speed.load_module().program(), dx, 0.4), bc_odd=(0, 2, 1))
        s.update(flat=flat, start=flat.clone(), states=states, batch=batch)
        s["graph"] = batch.capture(case["steps"])
    elif family == "bricked":
        m = _bricked(case["dtype"], case["brick"]).load_module()
        s.update(mod=m, u=x, other=torch.zeros_like(m.to_bricks(x, brick_size=case["brick"])))
    elif family == "diagnose":
        r = _periodic(case["dtype"])
        s.update(fill=_call(r, "apply_boundary"), launch=_call(r, "launch"), halo=r.halo_widths,
                 u=x, out=torch.zeros_like(x))
    else:
        s.update(server=StencilServer(_served_kinds(), budget_bytes=6e9), fields=x,
                 specs=_serve_specs(case))
    return s


def run(s):
    case, family = s["case"], s["family"]
    if family == "march":
        cur, nxt, spare = s["u"], s["a"], s["b"]
        for _ in range(s["launches"]):
            s["launch"](cur, nxt)
            cur, nxt, spare = nxt, spare, nxt
        return cur
    if family == "sweep":
        s["launch"](s["u"], s["out"])
        return s["out"]
    if family == "rk":
        s["u"].copy_(s["u0"])
        for _ in range(case["steps"]):
            s["step"](s["u"], 0.05)
        return s["u"]
    if family == "gray_scott":
        cur, nxt, spare = s["first"], s["a"], s["b"]
        for _ in range(case["steps"]):
            s["step"](*cur, *nxt)
            cur, nxt, spare = nxt, spare, nxt
        return list(cur)
    if family == "sw_batch":
        s["flat"].copy_(s["start"])
        s["graph"].replay()
        return [list(st) for st in s["states"]]
    if family == "bricked":
        m, shape = s["mod"], tuple(s["u"].shape)
        on_bricks = getattr(m, "launch_lap7_on_bricks")
        cur, nxt = m.to_bricks(s["u"], brick_size=case["brick"]), s["other"]
        for _ in range(case["sweeps"]):
            on_bricks(cur, nxt, shape)
            cur, nxt = nxt, cur
        return m.from_bricks(cur, shape, brick_size=case["brick"])
    if family == "diagnose":
        s["fill"](s["u"])
        s["launch"](s["u"], s["out"])
        return [s["u"], s["out"], reductions.mass(s["out"], s["halo"]),
                reductions.residual(s["out"], s["u"], s["halo"])]
    reqs = [SolveRequest(kind, dtype, (m + 2,) * SERVED[kind][1], steps, init=init)
            for (kind, dtype, m, steps), init in zip(s["specs"], s["fields"])]
    return [list(r.state) for r in s["server"].run(reqs, realtime=False)]


# --------------------------------------------------------------------------- #
# Unavoidable work of one pass: per launch (or step, or sweep) a program asks
# for, its input fields read once and its output fields written once
# --------------------------------------------------------------------------- #


def work(case):
    family = case["family"]
    if family in ("sw_batch", "serve"):
        if family == "sw_batch":
            pts = sum(n * n for n in _sw_sizes(case)) * case["steps"]
            # speed: 3 reads; stage 1: 3 reads, 3 writes; stage 2: 6 reads, 3 writes
            return {"bytes": 18 * _BYTES[case["dtype"]] * pts, "flops": 2 * 190 * pts}
        nbytes = flops = 0
        for kind, dtype, m, steps in _serve_specs(case):
            _, ndim, nstate, ops = SERVED[kind]
            nbytes += steps * m ** ndim * (nstate + 1) * _BYTES[dtype]
            flops += steps * m ** ndim * ops
        return {"bytes": nbytes, "flops": flops}
    pts = 1
    for n in _interior(case):
        pts *= n
    if family == "march":
        r = _compiled(case["body"], case["dtype"])
        launches = -(-case["steps"] // r.temporal_steps)
        return {"bytes": launches * 2 * _BYTES[case["dtype"]] * pts,
                "flops": launches * r.temporal_steps * BODIES[case["body"]][3] * pts}
    if family == "sweep":
        return {"bytes": 2 * _BYTES[case["dtype"]] * pts,
                "flops": case["chain"] * BODIES[case["body"]][3] * pts}
    if family == "gray_scott":
        fields = 4 if case["precision"] == "fp32_kahan" else 2
        esz = 8 if case["precision"] == "fp64" else 4
        return {"bytes": case["steps"] * 2 * fields * esz * pts,
                "flops": case["steps"] * (26 + 4 * fields) * pts}
    if family == "rk":
        # stages: u -> s1, acc; u, s1, acc -> s2, acc; u, s2, acc -> s3, acc; acc, s3 -> u
        return {"bytes": case["steps"] * 16 * _BYTES[case["dtype"]] * pts,
                "flops": case["steps"] * 4 * 17 * pts}
    if family == "bricked":
        return {"bytes": (case["sweeps"] + 2) * 2 * _BYTES[case["dtype"]] * pts,
                "flops": case["sweeps"] * 10 * pts}
    # diagnose: the sweep reads and writes, mass reads one field, the residual two
    return {"bytes": 5 * _BYTES[case["dtype"]] * pts, "flops": 14 * pts}


# --------------------------------------------------------------------------- #
# The same results in 64-bit torch arithmetic
# --------------------------------------------------------------------------- #


class _Views:
    """``u[i + 1, j]`` at index 0: the interior of ``u`` shifted by (1, 0)."""

    def __init__(self, data, halo):
        self.data, self.halo = data, halo

    def __getitem__(self, key):
        key = key if isinstance(key, tuple) else (key,)
        return self.data[tuple(slice(h + k, s - h + k)
                               for k, h, s in zip(key, self.halo, self.data.shape))]


_ELEMENTWISE = {"max": torch.maximum, "min": torch.minimum, "abs": torch.abs, "sqrt": torch.sqrt}


def _evaluate(fn, fields, halo, *scalars):
    body = types.FunctionType(fn.__code__, {**globals(), **_ELEMENTWISE})
    return body(*[_Views(f, halo) for f in fields], *scalars, *([0] * len(halo)))


def _stepped(fn, fields, halo):
    """One step into a zero-halo field."""
    out = torch.zeros_like(fields[0])
    out[_inner(out.shape, halo)] = _evaluate(fn, fields, halo)
    return out


def _wrapped(x, halo):
    """``x`` with its halo filled periodically."""
    for d, h in enumerate(halo):
        if h:
            n = x.shape[d]
            x = x.narrow(d, h, n - 2 * h)
            x = torch.cat([x.narrow(d, x.shape[d] - h, h), x, x.narrow(d, 0, h)], d)
    return x


def _sum(x):
    """Sum with the rounding error of every addition carried along."""
    x = x.reshape(-1)
    low = torch.zeros((), dtype=torch.float64, device=x.device)
    while x.numel() > 1:
        if x.numel() % 2:
            x = torch.cat([x, x.new_zeros(1)])
        a, b = x.view(2, -1)
        s = a + b
        t = s - a
        low = low + ((a - (s - t)) + (b - t)).sum()
        x = s
    return x[0] + low


def _exact_sw(case, seed):
    out = []
    rng = np.random.default_rng(seed)
    for n in _sw_sizes(case):
        q = [f.double() for f in _sw_init(n, rng, case["dtype"])]
        dx = 1.0 / n
        inner = (slice(1, -1), slice(1, -1))

        def mirrored(fields):
            g = [f.clone() for f in fields]
            for f, (sy, sx) in zip(g, ((1, 1), (1, -1), (-1, 1))):
                f[:, 0], f[:, -1] = sx * f[:, 1], sx * f[:, -2]
                f[0], f[-1] = sy * f[1], sy * f[-2]
            return g

        for _ in range(case["steps"]):
            speed = _evaluate(sw_speed, q, (1, 1)).max()
            dt = 0.4 * dx / speed
            mid = [f.clone() for f in q]
            for f, g, d in zip(mid, q, _evaluate(sw_rhs, mirrored(q), (1, 1), dx)):
                f[inner] = g[inner] + 0.5 * dt * d
            new = [f.clone() for f in q]
            for f, g, d in zip(new, q, _evaluate(sw_rhs, mirrored(mid), (1, 1), dx)):
                f[inner] = g[inner] + dt * d
            q = new
        out.append(q)
    return out


def exact(case, seed):
    family = case["family"]
    if family == "sw_batch":
        return _exact_sw(case, seed)
    x = _inputs(case, seed)
    if family == "march":
        r = _compiled(case["body"], case["dtype"])
        u = x.double()
        for _ in range(-(-case["steps"] // r.temporal_steps) * r.temporal_steps):
            u = _stepped(BODIES[case["body"]][0], [u], r.halo_widths)
        return u
    if family == "sweep":
        u = x.double()
        halo = _compiled(case["body"], case["dtype"], case["chain"]).halo_widths
        for _ in range(case["chain"]):
            u = _stepped(BODIES[case["body"]][0], [u], halo)
        return u
    if family == "bricked":
        u = x.double()
        halo = _bricked(case["dtype"], case["brick"]).halo_widths
        for _ in range(case["sweeps"]):
            u = _stepped(lap7, [u], halo)
        return u
    if family == "rk":
        halo = _rk4(case["dtype"]).info["halo"]
        u, dt = x.double(), 0.05
        for _ in range(case["steps"]):
            k1 = _stepped(lap4, [u], halo)
            k2 = _stepped(lap4, [u + 0.5 * dt * k1], halo)
            k3 = _stepped(lap4, [u + 0.5 * dt * k2], halo)
            k4 = _stepped(lap4, [u + dt * k3], halo)
            u = u + dt * (k1 + 2 * k2 + 2 * k3 + k4) / 6.0
        return u
    if family == "gray_scott":
        halo = _gray_scott(case["precision"]).halo_widths
        u, v = (t.double() for t in x)
        for _ in range(case["steps"]):
            wu, wv = _wrapped(u, halo), _wrapped(v, halo)
            u, v = _stepped(gs_u, [wu, wv], halo), _stepped(gs_v, [wu, wv], halo)
        # the compensation fields have no value of their own in exact arithmetic
        return [u, v] + ([None, None] if case["precision"] == "fp32_kahan" else [])
    if family == "diagnose":
        halo = _periodic(case["dtype"]).halo_widths
        u = _wrapped(x.double(), halo)
        out = _stepped(lap7, [u], halo)
        inner = _inner(u.shape, halo)
        d = out[inner] - u[inner]
        # the reductions read the stored field, which is rounded to its type
        stored = out.to(x.dtype).double()
        ds = stored[inner] - u[inner]
        return [u, out, _sum(out[inner].contiguous()) if x.dtype == torch.float64
                else _sum(stored[inner].contiguous()),
                torch.sqrt(_sum((d * d) if x.dtype == torch.float64 else (ds * ds)))]
    out = []
    for (kind, _, _, steps), init in zip(_serve_specs(case), x):
        fn, ndim, nstate, _ = SERVED[kind]
        state = [t.double() for t in init]
        for _ in range(steps):
            state = [_stepped(fn, state, (1,) * ndim)] + state[:-1]
        out.append(state)
    return out
