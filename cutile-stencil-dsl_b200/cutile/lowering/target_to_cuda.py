"""Dialect 3 -> CUDA C++ for the sm_100a stencil engine.

Replaces the reference's Dialect 3 -> cuTile Python emitter
(cutile/lowering/target_to_python.py:464-526).  For each ``cutile.kernel``:

* the body becomes a device functor ``Body_<name>::compute``: for every
  distinct ``(field, z offset, y offset)`` it loads one row *strip* from the
  staged tile (16-byte shared-memory vector loads), then evaluates the
  thread's ``VEC`` points with one statement per SSA op of the DSL body, in
  DSL order, using round-to-nearest intrinsics (``__dadd_rn`` ...) so no
  multiply-add contraction or re-association can change a bit; a value that
  one point needs at an X shift of another point's value (a face flux, a
  neighbour's velocity) is computed once (``_ShiftClasses``);
* two kernels instantiate the engine template around it: ``<name>_tma``
  (TMA tile copies) and ``<name>_ldg`` (cp.async copies, for arrays whose
  row pitch is not 16-byte aligned);
* ``<name>_desc`` exports the compile-time configuration to the host runtime.

Constants are emitted as exact hexadecimal float literals (the reference
needed a device array of float64 constants because cuTile rounds Python
scalars to float32, target_to_python.py:170-180, 429-451).
"""

from __future__ import annotations

import math
import struct

from cutile.dialects.cutile_target import KernelOp
from cutile.ir.core import ModuleOp

BC_CODES = {"none": "CSD_BC_NONE", "dirichlet": "CSD_BC_DIRICHLET", "neumann": "CSD_BC_NEUMANN",
            "periodic": "CSD_BC_PERIODIC", "reflecting": "CSD_BC_REFLECTING"}

_CTYPE = {"f32": "float", "f64": "double", "w": "double", "b": "bool", "wb": "bool"}


def hex_literal(value: float, ctype: str = "double") -> str:
    """Exact C literal for *value* in *ctype* (``float`` literals are the
    float32 rounding of the double, as NumPy rounds a Python float)."""
    if ctype == "float":
        v32 = struct.unpack("<f", struct.pack("<f", value))[0]
        if math.isfinite(v32):
            return f"{float(v32).hex()}f"
        bits = struct.unpack("<I", struct.pack("<f", v32))[0]
        return f"__int_as_float(0x{bits:08x})"
    if math.isfinite(value):
        return float(value).hex()
    bits = struct.unpack("<Q", struct.pack("<d", value))[0]
    return f"__longlong_as_double(0x{bits:016x}LL)"


def _internal_offsets(ndim: int, offsets) -> tuple[int, int, int]:
    if ndim == 3:
        return tuple(offsets)
    if ndim == 2:
        return (offsets[0], 0, offsets[1])
    return (0, 0, offsets[0])


def _parse_line(line: str):
    """``v3 = addf v1, a0 : f64`` -> ("v3", "addf", ["v1", "a0"], "f64", extra)."""
    if line.startswith("return "):
        parts = line.split()
        idx = int(parts[2][1:]) if len(parts) > 2 else None
        return ("", "return", [parts[1]], "", idx)
    lhs, rhs = line.split(" = ", 1)
    body, typ = rhs.rsplit(" : ", 1)
    parts = body.split(" ", 1)
    op = parts[0]
    rest = parts[1] if len(parts) > 1 else ""
    extra = None
    if op == "const":
        return (lhs, op, [], typ, float(rest))
    if "@" in rest:
        rest, extra = rest.split(" @")
    args = [a.strip() for a in rest.split(",")] if rest else []
    return (lhs, op, args, typ, extra)


class _BodyEmitter:
    def __init__(self, prefix: str, shared_divisors=frozenset()):
        self.prefix = prefix
        self.shared_divisors = shared_divisors   # scalars whose reciprocal is kept
        self.types: dict[str, str] = {}
        self.consts: dict[str, float] = {}
        self.lines: list[str] = []
        self.divisors: list[str] = []   # declarations of the divisors in use

    def divide(self, x: str, y: str, tgt: str) -> str:
        """``x / y``, correctly rounded: by a power of two as the product with
        its exact reciprocal, in FP64 by a scalar of ``shared_divisors``
        through the divisor that its quotients share, else a full division (in
        FP32 that is as short: shallow-water RK2 batch 5.10 ms, 5.58 with shared
        divisors).  A constant takes the full division too, full -> by its
        reciprocal: 4096^2 FP64, a quotient by 12 per point, 66 -> 72 us, an RK4
        step of it on 2048^2 117 -> 136, 256^3 by 6 55 -> 62."""
        ct = _CTYPE[tgt]
        if self.types.get(y) == "w" and y in self.consts:
            v = self.consts[y]
            if (math.isfinite(v) and 2.0 ** -60 <= abs(v) < 2.0 ** 60
                    and abs(math.frexp(v)[0]) == 0.5):
                fn = "__fmul_rn" if tgt == "f32" else "__dmul_rn"
                return f"{fn}({x}, {hex_literal(1.0 / v, ct)})"
        if tgt == "f64" and y in self.shared_divisors:
            decl = f"const csd::Divisor div_{y} = csd::divisor({self.conv(y, tgt)});"
            if decl not in self.divisors:
                self.divisors.append(decl)
            return f"csd::div_by({x}, div_{y})"
        return f"csd::div_rn({x}, {self.conv(y, tgt)})"

    def name(self, v: str) -> str:
        # accesses a<j>, scalars s<k> and device scalars d<k> are shared names
        return v if v[0] in "asd" else f"{self.prefix}{v}"

    def conv(self, v: str, to: str) -> str:
        """Operand *v* as C type of numpy kind *to* (f32/f64)."""
        t = self.types[v]
        if t == "w" and v in self.consts:
            return hex_literal(self.consts[v], "float" if to == "f32" else "double")
        n = self.name(v)
        if t in ("w", "f64") and to == "f32":
            return f"(float){n}"
        if t == "f32" and to == "f64":
            return f"(double){n}"
        return n

    def emit(self, lines: list[str], access_types: dict[str, str]) -> str:
        self.types.update(access_types)
        self.returns = []
        for raw in lines:
            lhs, op, args, typ, extra = _parse_line(raw)
            if op == "return":
                self.returns.append((args[0], extra))
                continue
            self.types[lhs] = typ
            if op == "const":
                self.consts[lhs] = extra
                continue
            ct = _CTYPE[typ]
            tgt = "f64" if typ in ("w", "f64") else typ
            sfx = "f" if tgt == "f32" else "d"
            if op == "divf":
                expr = self.divide(self.conv(args[0], tgt), args[1], tgt)
            elif op in ("addf", "subf", "mulf"):
                fn = {"addf": "add", "subf": "sub", "mulf": "mul"}[op]
                expr = f"__{sfx}{fn}_rn({self.conv(args[0], tgt)}, {self.conv(args[1], tgt)})"
            elif op == "cast":
                expr = self.conv(args[0], tgt)
            elif op == "negf":
                expr = f"-({self.conv(args[0], tgt)})"
            elif op == "absf":
                expr = f"{'fabsf' if tgt == 'f32' else 'fabs'}({self.conv(args[0], tgt)})"
            elif op == "sqrt":
                expr = f"csd::sqrt_rn({self.conv(args[0], tgt)})"
            elif op in ("maxf", "minf"):
                fn = "csd_max" if op == "maxf" else "csd_min"
                expr = f"{fn}({self.conv(args[0], tgt)}, {self.conv(args[1], tgt)})"
            elif op.startswith("cmp."):
                pred = op.split(".", 1)[1]
                sym = {"oeq": "==", "ogt": ">", "oge": ">=", "olt": "<", "ole": "<=",
                       "one": "!=", "une": "!="}[pred]
                cmp_t = extra or "f64"
                a, b = self.conv(args[0], cmp_t), self.conv(args[1], cmp_t)
                if pred == "one":  # ordered not-equal: false on NaN
                    expr = f"(({a}) < ({b}) || ({a}) > ({b}))"
                else:
                    expr = f"(({a}) {sym} ({b}))"
            elif op == "select":
                c = self.name(args[0]) if self.types[args[0]] in ("b", "wb") else self.conv(args[0], "f64")
                expr = f"({c} ? {self.conv(args[1], tgt)} : {self.conv(args[2], tgt)})"
            else:
                raise ValueError(f"unknown SSA op {op!r}")
            self.lines.append(f"const {ct} {self.name(lhs)} = {expr};")
        return self.returns

    def result_as(self, v: str, store_t: str) -> str:
        t = self.types[v]
        if t in ("b", "wb"):
            return f"({store_t})({self.name(v)} ? 1 : 0)"
        if t == "w" and v in self.consts:
            return hex_literal(self.consts[v], store_t)
        return f"({store_t}){self.name(v)}"


def _pos_name(cid: int, pos) -> str:
    if pos is None:
        return f"c{cid}"
    return "c%d_%s" % (cid, "_".join(("m%d" % -p) if p < 0 else str(p) for p in pos))


class _ShiftClasses:
    """Values of the body up to a shift along Y and X.

    A value's class is its expression tree with every access's Y and X
    offsets made relative to the smallest Y and the smallest X offset in the
    tree (``(my, mx)``); the value at the thread's point ``(j, k)`` (row j of
    the unit, point k of the row) is then its class at absolute position
    ``(j + my, k + mx)``.  Two values of one class at one position are the
    same expression of the same staged cells, so a thread computes each
    (class, position) once: a flux at the face between points k and k+1
    serves as the east flux of k and the west flux of k+1, and a strip of
    row y + 1 read at offset dy serves row y at offset dy + 1.  Every value is
    still computed by the same round-to-nearest operations on the same
    operands, so results are bit-identical to evaluating each point alone.
    """

    def __init__(self):
        self.ids: dict = {}

    def intern(self, key) -> int:
        cid = self.ids.get(key)
        if cid is None:
            cid = self.ids[key] = len(self.ids)
        return cid


def _shared_divisors(ssa: list, accesses: list, points: int) -> frozenset:
    """Scalar parameters that an FP64 body of ``points`` points divides by
    often enough for a kept reciprocal to pay: twice per point.  Footprints of
    more than 16 loads are at the register limit already and keep full
    divisions.  B200, full -> shared: four quotients by dx per point (diffusion,
    4096^2) 114 -> 99 us, two 68 -> 63, one 68 -> 68; shallow water with six,
    RK2 batch, 12.3 -> 10.5 ms; four-field Euler fluxes (20 loads), RK2 step on
    2048^2, 601 -> 633 us."""
    per_field: dict = {}
    for f, *offs in accesses:
        per_field.setdefault(f, []).append(any(offs))
    if sum(len(v) for v in per_field.values() if any(v)) > 16:
        return frozenset()
    count: dict = {}
    for raw in ssa:
        _, op, args, _, _ = _parse_line(raw)
        if op == "divf" and args[1][0] == "s" and args[1][1:].isdigit():
            count[args[1]] = count.get(args[1], 0) + 1
    return frozenset(s for s, n in count.items() if n >= 2 * points)


def emit_body(kernel: KernelOp, vec: int | None = None, suffix: str = "",
              members: list | None = None) -> str:
    """Device functor ``Body_<name><suffix>`` for the kernel's stencil
    body(ies): ``vec`` points per unit (default: the kernel's own), with
    ``members`` as further member declarations."""
    name = kernel.kernel_name.data + suffix
    ndim = kernel.ndim.data
    dtype = kernel.dtype.data
    field_t = "f32" if dtype in ("float32", "fp32") else "f64"
    store_t = "float" if field_t == "f32" else "double"
    params = engine_params(kernel)
    # X points per unit (engine Cfg::VEC; 16 bytes unless widened) and Y rows
    # per thread (engine Cfg::RPY)
    rpy = params["RPY"] if vec is None else 1
    vec = vec or params["VEC"]
    accesses = [tuple(a.data for a in acc) for acc in kernel.accesses.data]
    acc_info = [_internal_offsets(ndim, offs) + (f,) for f, *offs in accesses]  # (dz, dy, dx, f)
    # strip groups: (field, dz, dy of the unit's row 0) -> X range, over all rows
    groups: dict[tuple, list] = {}
    for dz, dy, dx, f in acc_info:
        for j in range(rpy):
            groups.setdefault((f, dz, dy + j), []).append(dx)
    gkeys = list(groups)
    gindex = {key: gi for gi, key in enumerate(gkeys)}
    # small bodies let the engine unroll a stage's units (their coordinates
    # fold into per-thread constants); wide ones would keep several units'
    # strips live at once and spill
    body_lines = sum(len(prog.data) for prog in kernel.ssa_body.data)
    unroll = 4 if (len(gkeys) <= 8 and rpy == 1 and body_lines <= 48) else 0
    out = [f"struct Body_{name} {{",
           f"  static constexpr int UNROLL = {unroll};",
           *[f"  {m}" for m in members or []],
           "  template <class C, class View>",
           "  __device__ __forceinline__ static void compute(const View& t, int r, int y,",
           "                                                 int x, csd::OutPack<typename C::T, "
           "C::NOUT, C::VEC * C::RPY>& o) {",
           f"    static_assert(C::VEC == {vec} && C::RPY == {rpy}, "
           f"\"body emitted for {vec} points x {rpy} rows per thread\");"]
    for gi, key in enumerate(gkeys):
        f, dz, dy = key
        lo, hi = min(groups[key]), max(groups[key])
        out.append(f"    const auto st{gi} = t.template strip<{f}, {dz}, {dy}, {lo}, {hi}>(r, y, x);")
    access_types = {}
    n_scal = kernel.scalar_count.data if kernel.scalar_count is not None else 0
    n_dyn = kernel.dyn_count.data if kernel.dyn_count is not None else 0
    for k in range(n_scal):
        out.append(f"    const double s{k} = t.scalar({k});")
        access_types[f"s{k}"] = "w"
    for k in range(n_dyn):
        out.append(f"    const double d{k} = t.dynamic({k});")
        access_types[f"d{k}"] = "w"

    # classes of every SSA value of every member (members share classes, so a
    # value two fused members both compute is computed once too)
    classes = _ShiftClasses()
    members = []
    for prog in kernel.ssa_body.data:
        info: dict = {}        # SSA name -> (class id, (my, mx) or None)
        lines, rets = [], []
        for raw in (x.data for x in prog):
            lhs, op, args, typ, extra = _parse_line(raw)
            if op == "return":
                rets.append((args[0], extra))
                continue
            if op == "const":
                info[lhs] = (classes.intern(("const", typ, repr(extra))), None)
                lines.append((lhs, op, [], typ, extra))
                continue
            parts = []
            for a in args:
                if a[0] == "a" and a[1:].isdigit():
                    dz, dy, dx, f = acc_info[int(a[1:])]
                    parts.append((classes.intern(("leaf", f, dz)), (dy, dx)))
                elif a[0] in "sd" and a[1:].isdigit():
                    parts.append((classes.intern(("scalar", a)), None))
                else:
                    parts.append(info[a])
            pos = [m for _, m in parts if m is not None]
            mn = (min(m[0] for m in pos), min(m[1] for m in pos)) if pos else None
            key = (op, typ, extra, tuple(
                (c, None if m is None else (m[0] - mn[0], m[1] - mn[1])) for c, m in parts))
            info[lhs] = (classes.intern(key), mn)
            lines.append((lhs, op, args, typ, extra))
        members.append((info, lines, rets))

    def rename(a: str, info: dict, j: int, k: int) -> str:
        if a[0] == "a" and a[1:].isdigit():
            dz, dy, dx, f = acc_info[int(a[1:])]
            key = (f, dz, dy + j)
            gi = gindex[key]
            idx = k + dx - min(groups[key])
            leaf = f"L{gi}_{idx}"
            if leaf not in access_types:
                access_types[leaf] = field_t
                out.append(f"    const {store_t} q_{leaf} = st{gi}.v[{idx}];")
            return leaf
        if a[0] in "sd" and a[1:].isdigit():
            return a
        cid, mn = info[a]
        return _pos_name(cid, None if mn is None else (j + mn[0], k + mn[1]))

    emitted: set = set()
    ssa: list[str] = []
    stores = []
    for j in range(rpy):
        for k in range(vec):
            for m, (info, lines, rets) in enumerate(members):
                for lhs, op, args, typ, extra in lines:
                    nm = rename(lhs, info, j, k)
                    if nm in emitted:
                        continue
                    emitted.add(nm)
                    if op == "const":
                        ssa.append(f"{nm} = const {extra!r} : {typ}")
                    else:
                        tail = f" @{extra}" if extra is not None else ""
                        ssa.append(f"{nm} = {op} {', '.join(rename(a, info, j, k) for a in args)}"
                                   f"{tail} : {typ}")
                for res, idx in rets:
                    stores.append((m if idx is None else idx, j * vec + k, rename(res, info, j, k)))
    em = _BodyEmitter("q_", _shared_divisors(ssa, accesses, vec * rpy) if field_t == "f64" else ())
    em.emit(ssa, access_types)
    for line in em.divisors + em.lines:
        out.append("    " + line)
    for slot, e, res in stores:
        out.append(f"    o.v[{slot}][{e}] = {em.result_as(res, store_t)};")
    out.append("  }")
    out.append("};")
    return "\n".join(out)


DIRECT_THREADS = 256


def direct_columns(kernel: KernelOp) -> dict:
    """The columns a direct kernel keeps per point (engine.cuh ``DirectCfg``):
    distinct ``(field, dy, dx)`` with the range of dz the body reads there."""
    ndim = kernel.ndim.data
    cols: dict[tuple, list] = {}
    for f, *offs in (tuple(a.data for a in acc) for acc in kernel.accesses.data):
        dz, dy, dx = _internal_offsets(ndim, offs)
        cols.setdefault((f, dy, dx), []).append(dz)
    return {k: (min(v), max(v)) for k, v in sorted(cols.items())}


def direct_plan(kernel: KernelOp) -> tuple:
    """``(points per lane, blocks per SM)`` of the kernel's direct form, or
    ``(0, 0)`` where it has none: fused boundary fills, chains and bricks keep
    the ring, and so do long bodies, which share values between neighbouring
    points, and columns that do not fit the registers.

    Four points per lane pay where the columns and their next plane leave
    three blocks per SM (7-point 301 x 411 x 523, FP32 / FP64 us: four points
    130 / 212, two 145 / 240, one 188 / 263; the ring's per-element copies 402
    / 458).  Longer bodies take two (RK4 stage of a radius-2 operator, 1537 x
    2049 FP64: 25 us, four points 35; 27-point box 301 x 311 x 323 FP64: 185,
    one point 242, the ring 274)."""
    p = engine_params(kernel)
    lines = sum(len(prog.data) for prog in kernel.ssa_body.data)
    if p["BRICK"] or p["TEMPORAL"] != 1 or p["BC"] != BC_CODES["none"] or lines > 100:
        return (0, 0)
    words = sum(hi - lo + 2 for lo, hi in direct_columns(kernel).values()) * p["dtype_bytes"] // 4
    points, blocks = ((4, 3) if words <= 24 and lines <= 16 else (2, 2) if words <= 72 else
                      (1, 1) if words <= 144 else (0, 0))
    return (points, p["OCCUPANCY"] or blocks) if points else (0, 0)


def _table(name: str, args: str, rows: dict) -> str:
    """A constexpr device lookup ``name(args)`` over ``rows`` {condition: value}."""
    expr = "".join(f"{cond} ? {value} : " for cond, value in rows.items())
    return f"__host__ __device__ static constexpr int {name}({args}) {{ return {expr}-1; }}"


def _direct_members(kernel: KernelOp) -> list:
    """Column and group tables of a direct body.  A group is the columns
    loaded through one row pointer (field, dy, leading dz)."""
    cols = direct_columns(kernel)
    groups: list = []
    for (f, dy, dx), (lo, hi) in cols.items():
        if (f, dy, hi) not in groups:
            groups.append((f, dy, hi))
    cl = list(cols.items())

    def by_col(fn):
        return {f"c == {i}": fn(*cl[i][0], *cl[i][1]) for i in range(len(cl))}

    def by_grp(fn):
        return {f"q == {i}": fn(*g) for i, g in enumerate(groups)}

    return [
        f"static constexpr int NCOL = {len(cl)}, NGRP = {len(groups)}, "
        f"WIN = {max(hi - lo + 1 for lo, hi in cols.values())};",
        _table("col", "int f, int dy, int dx",
               {f"f == {f} && dy == {dy} && dx == {dx}": i
                for i, ((f, dy, dx), _) in enumerate(cl)}),
        _table("col_dx", "int c", by_col(lambda f, dy, dx, lo, hi: dx)),
        _table("col_hi", "int c", by_col(lambda f, dy, dx, lo, hi: hi)),
        _table("col_len", "int c", by_col(lambda f, dy, dx, lo, hi: hi - lo + 1)),
        _table("col_grp", "int c", by_col(lambda f, dy, dx, lo, hi: groups.index((f, dy, hi)))),
        _table("grp_f", "int q", by_grp(lambda f, dy, hi: f)),
        _table("grp_dy", "int q", by_grp(lambda f, dy, hi: dy)),
        _table("grp_hi", "int q", by_grp(lambda f, dy, hi: hi)),
        f"__host__ __device__ static constexpr bool rewritten(int f) "
        f"{{ return {engine_params(kernel)['REWRITTEN']} >> f & 1; }}",
    ]


def _emit_direct(kernel: KernelOp) -> list:
    """The ``<name>_direct`` kernel and its descriptor (rows of any pitch)."""
    name = kernel.kernel_name.data
    p = engine_params(kernel)
    points, min_blocks = direct_plan(kernel)
    c = f"Cfg_{name}_direct"
    return [
        emit_body(kernel, 1, "_direct", _direct_members(kernel)),
        f"typedef csd::DirectCfg<{p['T']}, {p['NIN']}, {p['NOUT']}, {p['RZ']}, {p['RY']}, "
        f"{p['RX']}, {DIRECT_THREADS}, {points}, {p['REDUCE']}, {p['ndim']}> {c};",
        f'extern "C" __global__ void __launch_bounds__({DIRECT_THREADS}, {min_blocks})',
        f"{name}_direct(const __grid_constant__ csd_params p) {{",
        f"  csd::direct_step<{c}, Body_{name}_direct>(p);",
        "}",
        _descriptor(f"{name}_direct_desc", c, p, 0, min_blocks, 0),
        "",
    ]


def _descriptor(symbol: str, c: str, p: dict, zchunk: int, min_blocks: int,
                brick_tma: int, smem: str | None = None) -> str:
    """``csd_kernel_desc`` of configuration type ``c``."""
    nout = "0" if p["REDUCE"] else f"{c}::NOUT"
    return "\n".join([
        f'extern "C" __device__ const csd_kernel_desc {symbol} = {{',
        f"  CSD_DESC_MAGIC, {p['ndim']}, {c}::NIN, {nout}, (int)sizeof({c}::T),",
        f"  {c}::RZ * {c}::TEMPORAL, {c}::RY * {c}::TEMPORAL, {c}::RX * {c}::TEMPORAL,",
        f"  {c}::ROWS, {c}::TY, {c}::TX, {c}::VEC, {c}::NT, {c}::STAGES, {c}::NSLOT,",
        f"  {c}::HC * {c}::TEMPORAL, {c}::PADL, {c}::BOXW, {c}::BOXH, "
        f"{smem or f'{c}::SMEM_BYTES'},",
        f"  {zchunk}, {c}::TEMPORAL, {c}::BC, {min_blocks}, {c}::ALIGN,",
        f"  {p['NSCAL']}, {p['NDYN']}, {p['REDUCE']}, {c}::BRICK_SHIFT, {brick_tma}}};"])


def _internal_radius(ndim: int, radius) -> tuple[int, int, int]:
    r = list(radius)
    if ndim == 3:
        return (r[0], r[1], r[2])
    if ndim == 2:
        return (r[0], 0, r[1])
    return (0, 0, r[0])


def engine_params(kernel: KernelOp, ring: bool = False) -> dict:
    """Template parameters of the engine instance described by *kernel*
    (``ring``: of a register chain's ring form)."""
    ndim = kernel.ndim.data
    dtype = kernel.dtype.data
    tile = [a.data for a in kernel.tile_shape.data]
    hints = {}
    if kernel.kernel_hints is not None:
        items = [a.data for a in kernel.kernel_hints.data]
        hints = {k: eval(v, {}) for k, v in zip(items[0::2], items[1::2])}  # repr'd ints
    if ring:
        hints.pop("register_chain", None)
        hints.pop("chain_rows", None)
    if ndim == 3:
        rows, ty, tx = tile
    elif ndim == 2:
        rows, tx = tile
        ty = 1
    else:
        (tx,) = tile
        rows, ty = 1, 1
    rz, ry, rx = _internal_radius(ndim, [a.data for a in kernel.radius.data])
    nout = sum(max(1, sum(1 for s in prog if s.data.startswith("return")))
               for prog in kernel.ssa_body.data)
    nin = len(kernel.input_names.data)
    return {
        "T": "float" if dtype in ("float32", "fp32") else "double",
        "dtype_bytes": 4 if dtype in ("float32", "fp32") else 8,
        "NIN": nin, "NOUT": nout, "RZ": rz, "RY": ry, "RX": rx, "ROWS": rows, "TY": ty, "TX": tx,
        "NT": int(hints.get("threads", 256)), "STAGES": int(hints.get("stages", 1)),
        "TEMPORAL": kernel.temporal_steps.data if kernel.temporal_steps is not None else 1,
        "BC": BC_CODES[kernel.boundary_mode.data if kernel.boundary_mode is not None else "none"],
        "MINB": int(hints.get("min_blocks", 1)), "ZCHUNK": (int(hints.get("zchunk", 0)) if int(hints.get("zchunk", 0)) > 0
                   else -int(hints.get("waves", 1)) if int(hints.get("waves", 1)) > 1 else 0),
        "ndim": ndim,
        "NSCAL": kernel.scalar_count.data if kernel.scalar_count is not None else 0,
        "NDYN": kernel.dyn_count.data if kernel.dyn_count is not None else 0,
        "REDUCE": kernel.reduce_max.data if kernel.reduce_max is not None else 0,
        "BRICK": _brick_code(kernel, ndim),
        "RPY": int(hints.get("chain_rows", 0) or hints.get("rpy", 1)),
        "CHAIN_WARPS": int(hints.get("chain_warps", 4)),   # warps per block of a register chain
        # inputs (bit f: field f) that a launch may give as outputs too
        "REWRITTEN": int(hints.get("rewritten", 0)),
        "OCCUPANCY": int(hints.get("occupancy", 0)),   # a caller's blocks per SM (0: none)
        # points per lane of a register chain (0: the ring engine)
        "CHAIN": int(hints.get("register_chain", 0)),
        # size from which the chain is the faster form (0: always)
        "RING_BELOW": int(hints.get("ring_below", 0)),
        "VEC": int(hints.get("register_chain", 0)
                   or hints.get("vec", 4 if dtype in ("float32", "fp32") else 2)),
    }


def brick_tma_eligible(p: dict) -> bool:
    """Whether a bricked kernel's TMA entry can stage bricks with tensor copies
    (engine.cuh ``Cfg::BTMA``): 3-D bricks, one Z row per chunk, one step, no
    periodic wrap, a tile height dividing the brick or a multiple of it and
    a tile width that is a whole number of bricks, bricks at least 16 bytes wide, at most 256
    bricks per staged row."""
    code = p["BRICK"]
    if not code or (code >> 4) != 3:
        return False
    b = 1 << (code & 15)
    esz = p["dtype_bytes"]
    balign = max(b, 128 // esz)
    padl = -(-p["RX"] // b) * b
    boxw = -(-(padl + p["TX"] + p["RX"]) // balign) * balign
    return (p["ROWS"] == 1 and p["TEMPORAL"] == 1 and p["BC"] != BC_CODES["periodic"]
            and (b % p["TY"] == 0 or p["TY"] % b == 0) and p["TX"] % b == 0 and (b * esz) % 16 == 0
            and boxw // b <= 256)


def _brick_code(kernel: KernelOp, ndim: int) -> int:
    """(ndim << 4) | log2(brick size) for a bricked-layout kernel, else 0."""
    if kernel.layout is None or kernel.layout.data != "bricked":
        return 0
    b = kernel.brick_size.data if kernel.brick_size is not None else 0
    if b < 4 or b > 64 or (b & (b - 1)):
        raise ValueError(f"brick size must be a power of two in [4, 64], got {b}")
    return (ndim << 4) | (b.bit_length() - 1)


def _emit_engine(name: str, p: dict) -> list:
    """The ``<name>_tma`` and ``<name>_ldg`` kernels and their descriptor."""
    parts = []
    brick_tma = brick_tma_eligible(p)
    for suffix, loader in (("tma", "CSD_LOADER_TMA"), ("ldg", "CSD_LOADER_LDG")):
        if p["BRICK"] and not brick_tma:
            loader = "CSD_LOADER_LDG"   # bricked fields the TMA boxes cannot stage
        entry, nt, minb = "stream_engine", p["NT"], p["MINB"]
        cfg = (f"csd::Cfg<{p['T']}, {p['NIN']}, {p['NOUT']}, {p['RZ']}, {p['RY']}, {p['RX']}, "
               f"{p['ROWS']}, {p['TY']}, {p['TX']}, {p['NT']}, {p['STAGES']}, {p['TEMPORAL']}, "
               f"{loader}, {p['BC']}, {p['REDUCE']}, {p['BRICK']}, {p['RPY']}, {p['VEC']}>")
        if p["CHAIN"]:
            entry, nt, minb = "register_chain", 32 * p["CHAIN_WARPS"], 1
            cfg = (f"csd::ChainCfg<{p['T']}, {p['NIN']}, {p['NOUT']}, {p['RZ']}, {p['RX']}, "
                   f"{nt}, {p['TEMPORAL']}, {loader}, {p['VEC']}>")
            if p["ndim"] == 3:
                entry = "plane_chain"
                cfg = (f"csd::PlaneChainCfg<{p['T']}, {p['NIN']}, {p['NOUT']}, {p['RZ']}, "
                       f"{p['RY']}, {p['RX']}, {nt}, {p['TEMPORAL']}, {loader}, {p['VEC']}, "
                       f"{p['RPY']}>")
        parts.append(f"typedef {cfg} Cfg_{name}_{suffix};")
        # chains have kernels of their own for batches
        for form, infix, last in (((0, "", ", false"), (3, "batch_", ", true")) if p["CHAIN"] else
                                  ((0, "", ""),)):
            if p["CHAIN"]:
                parts.append(f"#if CSD_HAS({form})")
            parts.append(f'extern "C" __global__ void __launch_bounds__({nt}, {minb})')
            parts.append(f"{name}_{infix}{suffix}(const __grid_constant__ csd_params p) {{")
            parts.append(f"  csd::{entry}<Cfg_{name}_{suffix}, Body_{name}{last}>(p);")
            parts.append("}")
            if p["CHAIN"]:
                parts.append("#endif")
    if p["CHAIN"]:
        parts += ["#if CSD_HAS(0)", f'extern "C" __device__ const int {name}_batch_apart = 1;']
    c = f"Cfg_{name}_tma"
    # both entries launch with one shared-memory size: the larger one
    smem = (f"({c}::SMEM_BYTES > Cfg_{name}_ldg::SMEM_BYTES ? {c}::SMEM_BYTES : "
            f"Cfg_{name}_ldg::SMEM_BYTES)")
    parts.append(_descriptor(f"{name}_desc", c, p, p["ZCHUNK"], p["MINB"],
                             1 if brick_tma else 0, smem))
    if p["CHAIN"]:
        parts.append("#endif")
    parts.append("")
    return parts


def source_forms(source: str, name: str) -> tuple:
    """Forms of kernel ``name`` beside its own that a generated source holds."""
    return tuple(f for f, mark in ((1, f"{name}_direct_desc = {{"), (2, f"{name}_ring_desc = {{"),
                                   (3, f"{name}_batch_apart = ")) if f" {mark}" in source)


def emit_cuda(module: ModuleOp, preamble: bool = True) -> str:
    """CUDA translation unit for the kernel(s) in a D3 module (``preamble=False``
    gives just the kernels, to append to another unit)."""
    kernels = [op for op in module.body.block.ops if isinstance(op, KernelOp)]
    if not kernels:
        raise ValueError("No KernelOp found in target IR module")
    parts = ["// Generated B200 stencil kernel(s). Do not edit.",
             "// Forms: 0 the kernels themselves, 1 for unaligned rows, 2 rings of register",
             "// chains, 3 batches of register chains; all of them unless CSD_FORM names one.",
             "#ifdef CSD_FORM", "#define CSD_HAS(form) (CSD_FORM == (form))", "#else",
             "#define CSD_HAS(form) 1", "#endif",
             '#include "csd/engine.cuh"', "",
             "__device__ __forceinline__ double csd_max(double a, double b) "
             "{ return (a != a || a > b) ? a : b; }",
             "__device__ __forceinline__ double csd_min(double a, double b) "
             "{ return (a != a || a < b) ? a : b; }",
             "__device__ __forceinline__ float csd_max(float a, float b) "
             "{ return (a != a || a > b) ? a : b; }",
             "__device__ __forceinline__ float csd_min(float a, float b) "
             "{ return (a != a || a < b) ? a : b; }", ""]
    if not preamble:
        parts = []
    for kernel in kernels:
        name = kernel.kernel_name.data
        p = engine_params(kernel)
        parts.append(f"// expression: {kernel.expression.data}")
        parts.append("#if CSD_HAS(0) || CSD_HAS(3)" if p["CHAIN"] else "#if CSD_HAS(0)")
        parts.append(emit_body(kernel))
        parts.append("")
        parts.extend(_emit_engine(name, p))
        parts.append("#endif")
        if p["CHAIN"] and p["RING_BELOW"] > 0:
            # the same steps by the shared-memory rings, for smaller arrays
            q = engine_params(kernel, ring=True)
            parts += ["#if CSD_HAS(0)", f'extern "C" __device__ const long long {name}_ring_below = '
                      f'{p["RING_BELOW"]};', "#endif", "#if CSD_HAS(2)"]
            parts.append(emit_body(kernel, q["VEC"], "_ring"))
            parts.append("")
            parts.extend(_emit_engine(f"{name}_ring", q))
            parts.append("#endif")
        if direct_plan(kernel)[0]:
            if p["REWRITTEN"]:      # (read before the direct form is there)
                parts += ["#if CSD_HAS(0)", f'extern "C" __device__ const unsigned '
                          f'{name}_direct_rewrites = {p["REWRITTEN"]};', "#endif"]
            parts.append("#if CSD_HAS(1)")
            parts.extend(_emit_direct(kernel))
            parts.append("#endif")
        parts.append("")
    return "\n".join(parts) + "\n"


__all__ = ["emit_cuda", "source_forms", "emit_body", "engine_params", "hex_literal", "brick_tma_eligible"]
