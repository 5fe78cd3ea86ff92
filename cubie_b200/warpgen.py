"""Code generation for the warp-per-system path (large systems).

For a system with many states, one warp integrates one run: lane ``l``
holds components ``l, l + 32, l + 64, ...`` of every state-sized vector, and
the right-hand side and the Jacobian-vector product are evaluated by all 32
lanes together from a copy of the state in shared memory.

A straight-line, component-by-component translation would make every lane
execute different code.  Instead the expressions are grouped into
*classes*: two components belong to the same class when their expressions
are the same up to which states, parameters and drivers they read (the
interior compartments of a cable, every gate of the same kind, ...).  A
class is emitted once as a function of its slot values; lane ``l`` then
evaluates members ``l, l + 32, ...`` of the class, gathering each member's
slots from shared memory through index tables (or through an affine formula
``index = a * member + b`` when the indices follow one, which is the common
case and needs no table).  All lanes run the same instructions; only the
member count of a class decides how many lanes are busy.

The Jacobian-vector product ``(J v)_i = sum_k df_i/dy_k v_k`` is generated
the same way, with the components of ``v`` as a fourth kind of slot.
"""

from __future__ import annotations

from dataclasses import dataclass, field
from typing import Dict, List, Sequence, Tuple

import sympy as sp

from .codegen import FlopCount, _CudaPrinter, count_ops
from .symbolic import TIME, SymbolicODE

KINDS = ("y", "v", "p", "d")


@dataclass
class ExprClass:
    """One group of isomorphic component expressions."""

    template: sp.Expr                    # expression in slot placeholders
    slots: List[Tuple[str, int]]         # (kind, slot number) in placeholder order
    members: List[int] = field(default_factory=list)          # output component of each member
    indices: List[List[int]] = field(default_factory=list)    # per member, the index of each slot


def _placeholder(kind: str, k: int) -> sp.Symbol:
    return sp.Symbol(f"_{kind}{k}", real=True)


def _canonical(expr: sp.Expr, kind_of: Dict[sp.Symbol, Tuple[str, int]]) -> Tuple[sp.Expr, List[Tuple[str, int]]]:
    """Replace the states, v components, parameters and drivers in ``expr``
    by placeholders numbered per kind in order of first appearance (a
    preorder walk; repeated twice so the ordering no longer depends on the
    original names).  Returns the template and, per placeholder, the
    original (kind, index)."""
    cur = expr
    binding: Dict[sp.Symbol, Tuple[str, int]] = {}
    for _ in range(2):
        order: List[sp.Symbol] = []
        for node in sp.preorder_traversal(cur):
            if isinstance(node, sp.Symbol) and node not in order and (node in kind_of or node in binding):
                order.append(node)
        counters = {k: 0 for k in KINDS}
        new_binding = {}
        rename = {}
        for s in order:
            kind, idx = binding[s] if s in binding else kind_of[s]
            ph = _placeholder(kind, counters[kind])
            counters[kind] += 1
            rename[s] = ph
            new_binding[ph] = (kind, idx)
        cur = cur.xreplace(rename)
        binding = new_binding
    slots = [binding[ph] for ph in sorted(binding, key=lambda s: (KINDS.index(s.name[1]), int(s.name[2:])))]
    return cur, slots


def group_classes(exprs: Sequence[sp.Expr], kind_of: Dict[sp.Symbol, Tuple[str, int]]) -> List[ExprClass]:
    classes: Dict[str, ExprClass] = {}
    order: List[str] = []
    for i, e in enumerate(exprs):
        tmpl, slots = _canonical(sp.sympify(e), kind_of)
        key = sp.srepr(tmpl)
        if key not in classes:
            ph = sorted(tmpl.free_symbols & {_placeholder(k, j) for k in KINDS for j in range(len(slots) + 1)},
                        key=lambda s: (KINDS.index(s.name[1]), int(s.name[2:])))
            classes[key] = ExprClass(template=tmpl, slots=[(s.name[1], int(s.name[2:])) for s in ph])
            order.append(key)
        c = classes[key]
        c.members.append(i)
        c.indices.append([idx for (_, idx) in slots])
    return [classes[k] for k in order]


def _times(fc: FlopCount, k: int) -> FlopCount:
    """The operation count of ``k`` evaluations of one class body."""
    return FlopCount(fc.add * k, fc.mul * k, fc.div * k, fc.special * k)


def _affine(values: List[int]):
    """(a, b) with values[m] == a * m + b for every m, or None."""
    if len(values) == 1:
        return 0, values[0]
    a = values[1] - values[0]
    b = values[0]
    if all(v == a * m + b for m, v in enumerate(values)):
        return a, b
    return None


@dataclass
class WarpSystemCode:
    source: str
    n_classes_f: int
    n_classes_jv: int
    flops: Dict[str, FlopCount]
    nnz: int = 0                 # cached Jacobian coefficients per run (0: J v stays matrix-free)
    n_classes_fj: int = 0
    register_slots: int = 0      # register form: components and Jacobian coefficients per lane (0: none)
    register_coefs: int = 0


# Largest cached Jacobian (coefficients per run) the generator emits: one
# warp keeps them in shared memory, 4 bytes each in FP32.
CACHED_JAC_MAX = 2048


def _emit_classes(name: str, classes: List[ExprClass], with_v: bool, tables: List[str]) -> Tuple[str, FlopCount]:
    """A device function evaluating every class for the calling lane."""
    lines = []
    fc = FlopCount()
    sig = (f"    template <class R> static __device__ CBX_NOINLINE void {name}(const R* __restrict__ ys, "
           + ("const R* __restrict__ vs, " if with_v else "")
           + "const R* __restrict__ ps, const R* __restrict__ ds, R t, R* __restrict__ out, int lane)")
    lines.append(sig)
    lines.append("    {")
    lines.append("        (void)ys; (void)ps; (void)ds; (void)t;" + (" (void)vs;" if with_v else ""))
    for ci, c in enumerate(classes):
        nm = len(c.members)
        slot_syms = [_placeholder(k, j) for (k, j) in c.slots]
        sym_map = {TIME: "t"}
        for s in slot_syms:
            sym_map[s] = f"s_{s.name[1:]}"
        lines.append(f"        // class {ci}: {nm} member(s)")
        # kept as a loop: unrolled over a lane's members the class code
        # grew the kernel until instruction fetch bounded it
        lines.append("        #pragma unroll 1")
        lines.append(f"        for (int m = lane; m < {nm}; m += 32) {{")
        # output index
        aff = _affine(c.members)
        if aff is not None:
            lines.append(f"            const int o = {aff[0]} * m + {aff[1]};")
        else:
            tname = f"{name}_c{ci}_out"
            tables.append(f"    static __device__ const unsigned short {tname}[{nm}] = "
                          f"{{{', '.join(str(v) for v in c.members)}}};")
            lines.append(f"            const int o = {tname}[m];")
        for q, (kind, j) in enumerate(c.slots):
            col = [row[q] for row in c.indices]
            src = {"y": "ys", "v": "vs", "p": "ps", "d": "ds"}[kind]
            aff = _affine(col)
            if aff is not None:
                idx = f"{aff[0]} * m + {aff[1]}" if aff[0] != 0 else f"{aff[1]}"
            else:
                tname = f"{name}_c{ci}_s{q}"
                tables.append(f"    static __device__ const unsigned short {tname}[{nm}] = "
                              f"{{{', '.join(str(v) for v in col)}}};")
                idx = f"{tname}[m]"
            lines.append(f"            const R s_{kind}{j} = {src}[{idx}];")
        printer = _CudaPrinter(sym_map)
        reps, reduced = sp.cse([c.template], symbols=sp.numbered_symbols("_t"), optimizations="basic")
        for s, e in reps:
            lines.append(f"            const R {s} = {printer.doprint(e)};")
            fc = fc + _times(count_ops(e), nm)
        lines.append(f"            out[o] = {printer.doprint(reduced[0])};")
        fc = fc + _times(count_ops(reduced[0]), nm)
        lines.append("        }")
    lines.append("    }")
    return "\n".join(lines), fc


def _index_expr(name: str, ci: int, q: int, values: List[int], tables: List[str]) -> str:
    aff = _affine(values)
    if aff is not None:
        return f"{aff[0]} * m + {aff[1]}" if aff[0] != 0 else f"{aff[1]}"
    tname = f"{name}_c{ci}_s{q}"
    tables.append(f"    static __device__ const unsigned short {tname}[{len(values)}] = "
                  f"{{{', '.join(str(v) for v in values)}}};")
    return f"{tname}[m]"


def _emit_cached_jacobian(classes: List[ExprClass], tables: List[str]):
    """``fj_lanes`` (f and the Jacobian's nonzero coefficients at one state,
    in one pass that shares the subexpressions of both) and ``jmv_cached``
    (J v from those coefficients) for classes of the joint expression
    (f_i, (J v)_i).  A class of M members whose (J v) template reads r
    components of v stores its coefficients at
    ``jac[base + j * M + m]`` (slot j, member m), so the lanes of a warp
    read and write consecutive words."""
    fj = ["    template <class R> static __device__ CBX_NOINLINE void fj_lanes(const R* __restrict__ ys, "
          "const R* __restrict__ ps, const R* __restrict__ ds, R t, R* __restrict__ out, R* __restrict__ jac, "
          "int lane)", "    {", "        (void)ys; (void)ps; (void)ds; (void)t; (void)jac;"]
    jm = ["    template <class R> static __device__ CBX_NOINLINE void jmv_cached(const R* __restrict__ vs, "
          "const R* __restrict__ jac, R* __restrict__ out, int lane)", "    {", "        (void)jac; (void)vs;"]
    fl_fj, fl_jm = FlopCount(), FlopCount()
    base = 0
    for ci, c in enumerate(classes):
        f_t, jv_t = c.template.args
        nm = len(c.members)
        slot_syms = [_placeholder(k, j) for (k, j) in c.slots]
        v_syms = [ph for ph in slot_syms if ph.name[1] == "v"]
        coefs = [sp.diff(jv_t, v) for v in v_syms]
        if any(v in cf.free_symbols for cf in coefs for v in v_syms):
            raise ValueError("Jacobian-vector template is not linear in v")
        sym_map = {TIME: "t"}
        for sy in slot_syms:
            sym_map[sy] = f"s_{sy.name[1:]}"
        printer = _CudaPrinter(sym_map)
        out_idx = _index_expr("fj", ci, 99, c.members, tables)
        head = [f"        // class {ci}: {nm} member(s), {len(v_syms)} coefficient(s) each",
                "        #pragma unroll 1",
                f"        for (int m = lane; m < {nm}; m += 32) {{", f"            const int o = {out_idx};"]
        fj += head
        jm += head
        for q, (kind, j) in enumerate(c.slots):
            col = [row[q] for row in c.indices]
            idx = _index_expr("cj", ci, q, col, tables)
            src = {"y": "ys", "v": "vs", "p": "ps", "d": "ds"}[kind]
            if kind == "v":
                jm.append(f"            const R s_{kind}{j} = {src}[{idx}];")
            else:
                fj.append(f"            const R s_{kind}{j} = {src}[{idx}];")
        reps, reduced = sp.cse([f_t, *coefs], symbols=sp.numbered_symbols("_t"), optimizations="basic")
        for sy, e in reps:
            fj.append(f"            const R {sy} = {printer.doprint(e)};")
            fl_fj = fl_fj + _times(count_ops(e), nm)
        fj.append(f"            out[o] = {printer.doprint(reduced[0])};")
        for k, e in enumerate(reduced):
            fl_fj = fl_fj + _times(count_ops(e), nm)
        for j, e in enumerate(reduced[1:]):
            fj.append(f"            jac[{base + j * nm} + m] = {printer.doprint(e)};")
        terms = [f"jac[{base + j * nm} + m] * {printer.doprint(v)}" for j, v in enumerate(v_syms)]
        jm.append(f"            out[o] = {' + '.join(terms) if terms else 'R(0)'};")
        fl_jm = fl_jm + FlopCount(add=max(len(terms) - 1, 0) * nm, mul=len(terms) * nm)
        fj.append("        }")
        jm.append("        }")
        base += nm * len(v_syms)
    fj.append("    }")
    jm.append("    }")
    return "\n".join(fj), "\n".join(jm), base, fl_fj, fl_jm


# Largest register form the generator emits (see ``_register_plan``).  The
# device code decides by its working precision whether the lanes can hold it.
REGISTER_MAX_SLOTS = 16      # vector components per lane (512 states)
REGISTER_MAX_COEFS = 64      # Jacobian coefficients per lane
REGISTER_MAX_GATHERS = 40    # exchanged values per J v


@dataclass
class RegisterBody:
    """One class evaluated for one slot by the lanes ``lanes``."""

    cls: int
    slot: int
    lanes: List[int]
    offsets: List[int]           # per placeholder: distance of the place read (y, v), index (p, d)


@dataclass
class LaneMap:
    """Where the components live: lane ``l`` holds component
    ``base[k] + stride l`` in slot ``k`` when ``l < count[k]``; place
    ``32 k + l`` is that component's, ``place[c]`` component ``c``'s."""

    place: List[int]
    base: List[int]
    count: List[int]
    stride: int


def _lane_maps(n: int) -> List[LaneMap]:
    """Candidate layouts: the components in a row, and for every way to see
    them as ``g`` variables of ``q`` cells (grouped by variable, or
    interleaved cell by cell) each variable from lane 0 of slots of its own,
    so that a cell's variables share a lane."""
    maps = [LaneMap(list(range(n)), [32 * k for k in range((n + 31) // 32)],
                    [min(32, n - 32 * k) for k in range((n + 31) // 32)], 1)]
    for g in range(2, REGISTER_MAX_SLOTS + 1):
        if n % g:
            continue
        q = n // g
        per = (q + 31) // 32                       # slots per variable
        cells = [32 * k for k in range(per)]
        count = [min(32, q - j) for j in cells]
        if q % 32:
            maps.append(LaneMap([c // q * 32 * per + c % q for c in range(n)],
                                [v * q + j for v in range(g) for j in cells], count * g, 1))
        maps.append(LaneMap([c % g * 32 * per + c // g for c in range(n)],
                            [j * g + v for v in range(g) for j in cells], count * g, g))
    return [m for m in maps if len(m.base) <= REGISTER_MAX_SLOTS]


@dataclass
class RegisterPlan:
    lanes: LaneMap
    bodies_f: List[RegisterBody]                      # f alone
    bodies_fj: List[RegisterBody]                     # f and the Jacobian's coefficients
    gathers: List[Tuple[int, int, int]]               # (slot, shift, mode) of every exchanged value
    gather_of: Dict[Tuple[int, int], int]             # (slot, offset) -> exchange, absent when the lane holds it
    coefs: Dict[Tuple[int, int], int]                 # (slot, offset) -> coefficient


def _register_bodies(classes: List[ExprClass], place: List[int]) -> List[RegisterBody]:
    bodies: Dict[tuple, RegisterBody] = {}
    for ci, c in enumerate(classes):
        for row, comp in zip(c.indices, c.members):
            at = place[comp]
            offs = [place[idx] - at if kind in "yv" else idx for (kind, _), idx in zip(c.slots, row)]
            b = bodies.setdefault((at // 32, ci, tuple(offs)), RegisterBody(ci, at // 32, [], offs))
            b.lanes.append(at % 32)
    return [bodies[k] for k in sorted(bodies, key=lambda k: (k[0], bodies[k].lanes[0], k[1]))]


def _merged_order(sequences: List[List[int]]) -> List[int]:
    """The distinct items of ``sequences`` in an order that keeps every
    sequence's own (first-seen order where they contradict each other)."""
    items = list(dict.fromkeys(d for seq in sequences for d in seq))
    before: Dict[int, set] = {d: set() for d in items}
    for seq in sequences:
        for a, b in zip(seq, seq[1:]):
            before[b].add(a)
    out: List[int] = []
    while len(out) < len(items):
        left = [d for d in items if d not in out]
        out.append(next((d for d in left if before[d] <= set(out)), left[0]))
    return out


def _body_cost(c: ExprClass) -> int:
    """Issue slots of one evaluation, roughly: a division or a special
    function is a handful of instructions."""
    ops = count_ops(c.template)
    return ops.add + ops.mul + 8 * (ops.div + ops.special)


def _plan_cost(plan: RegisterPlan, classes_f: List[ExprClass], classes_fj: List[ExprClass]) -> int:
    """Issue slots of one stage solve, roughly: every body runs once for f and
    once for f and J whatever its number of lanes, one Krylov iteration takes
    six J v's (a select and a shuffle per exchange, a multiply-add per
    coefficient) and about a hundred slots of vector work per component."""
    return (sum(_body_cost(classes_f[b.cls]) for b in plan.bodies_f)
            + 2 * sum(_body_cost(classes_fj[b.cls]) for b in plan.bodies_fj)
            + 18 * len(plan.gathers) + 8 * len(plan.coefs) + 110 * len(plan.lanes.base))


def _register_plan(n: int, classes_f: List[ExprClass], classes_fj: List[ExprClass]):
    """The cheapest register form over the candidate layouts, or None.

    A 76-state cable (four variables of 19 compartments) packed in a row
    shares its slots between variables, and a slot's classes run one after
    the other; with a slot per variable each class runs once and a
    compartment's variables need no exchange.  Measured, in a row against
    the chosen layout (80 steps): 76 states x 5,003 runs 3.24 -> 2.60 ms, 96 x
    4,000 2.36 -> 2.06, 124 x 3,000 2.40 -> 1.82; at 64, 160 and 192 states the
    row is the cheaper one and stays."""
    plans = [p for p in (_plan_layout(m, classes_f, classes_fj) for m in _lane_maps(n)) if p is not None]
    return min(plans, key=lambda p: _plan_cost(p, classes_f, classes_fj), default=None)


def _plan_layout(lanes: LaneMap, classes_f: List[ExprClass], classes_fj: List[ExprClass]):
    """How a warp evaluates ``classes_f`` (of f_i) and ``classes_fj`` (of the
    joint expression (f_i, (J v)_i)) with every vector spread over its lanes'
    registers, or None when it cannot.

    When the place an expression reads lies at a constant offset ``d`` from
    the place it computes (neighbours on a line, the same compartment's other
    variables), the read is a rotation of the vector by ``d``: with
    ``d = 32 q + s`` lane ``l`` needs slot ``k + q`` (or ``k + q + 1`` past the
    end of the warp) of lane ``(l + s) % 32``.  Every source lane serves
    exactly one lane, so it first selects the slot it is asked for and one
    shuffle moves it; ``s = 0`` needs neither.  Members of a class that read
    at different offsets become separate bodies.

    A gather's mode: 0 selects between the two slots, 1 only the first is
    ever read, 2 only the second."""
    slots = len(lanes.base)
    bodies_f = _register_bodies(classes_f, lanes.place)
    bodies_fj = _register_bodies(classes_fj, lanes.place)
    if slots > REGISTER_MAX_SLOTS or max(len(bodies_f), len(bodies_fj)) > 3 * slots + 4:
        return None
    need: Dict[Tuple[int, int], set] = {}             # (slot + q, s) -> {False: first slot read, True: second}
    gather_keys: Dict[Tuple[int, int], Tuple[int, int]] = {}
    coefs: Dict[Tuple[int, int], int] = {}
    for classes, bodies in ((classes_f, bodies_f), (classes_fj, bodies_fj)):
        for b in bodies:
            for (kind, _), d in zip(classes[b.cls].slots, b.offsets):
                if kind not in "yv":
                    continue
                q, s = divmod(d, 32)
                if s:
                    gather_keys[(b.slot, d)] = (b.slot + q, s)
                    need.setdefault((b.slot + q, s), set()).update(l + s >= 32 for l in b.lanes)
    # each row sums its terms in its own class's order (zero coefficients of
    # the slot's other classes in between), so a J v rounds as the
    # shared-memory form's does
    for k in range(slots):
        rows = [[d for (kind, _), d in zip(classes_fj[b.cls].slots, b.offsets) if kind == "v"]
                for b in bodies_fj if b.slot == k]
        for d in _merged_order(rows):
            coefs[(k, d)] = len(coefs)
    if len(coefs) > REGISTER_MAX_COEFS or len(need) > REGISTER_MAX_GATHERS:
        return None
    order = sorted(need)
    gathers = [(k, s, 0 if len(need[(k, s)]) == 2 else (2 if True in need[(k, s)] else 1)) for k, s in order]
    gather_of = {key: order.index(ks) for key, ks in gather_keys.items()}
    return RegisterPlan(lanes, bodies_f, bodies_fj, gathers, gather_of, coefs)


def _lane_condition(lanes: List[int]) -> str:
    """Condition on ``lane`` for ``lanes`` of a slot ("" when every lane)."""
    if len(lanes) == 32:
        return ""
    lo, hi = min(lanes), max(lanes)
    if len(lanes) == hi - lo + 1:
        if lo == hi:
            return f"lane == {lo}"
        if lo == 0:
            return f"lane < {hi + 1}"
        return f"lane >= {lo}" if hi == 31 else f"(lane >= {lo} && lane < {hi + 1})"
    return f"((0x{sum(1 << l for l in lanes):x}u >> lane) & 1u)"


def _emit_register_lanes(classes_f: List[ExprClass], classes_fj: List[ExprClass], plan: RegisterPlan) -> str:
    """The per-lane functions of the register form.  ``y`` / ``v`` are the
    lane's slots, ``g`` the exchanged values in the plan's order, ``J`` the
    lane's Jacobian coefficients (zero where a lane's row has none)."""
    slots = len(plan.lanes.base)

    def read(vec: str, slot: int, d: int) -> str:
        q, s = divmod(d, 32)
        return f"{vec}[{slot + q}]" if s == 0 else f"g[{plan.gather_of[(slot, d)]}]"

    def body_lines(b: RegisterBody, with_j: bool) -> List[str]:
        c = (classes_fj if with_j else classes_f)[b.cls]
        f_t, jv_t = c.template.args if with_j else (c.template, sp.Integer(0))
        sym_map = {TIME: "t"}
        lines = []
        v_syms = []
        for (kind, j), d in zip(c.slots, b.offsets):
            ph = _placeholder(kind, j)
            if kind == "v":
                v_syms.append((ph, d))
                continue
            sym_map[ph] = (read("y", b.slot, d) if kind == "y" else f"{'ps' if kind == 'p' else 'ds'}[{d}]")
        coefs = [sp.diff(jv_t, v) for v, _ in v_syms]
        if any(v in cf.free_symbols for cf in coefs for v, _ in v_syms):
            raise ValueError("Jacobian-vector template is not linear in v")
        printer = _CudaPrinter(sym_map)
        reps, reduced = sp.cse([f_t, *coefs], symbols=sp.numbered_symbols("_t"), optimizations="basic")
        for sy, e in reps:
            lines.append(f"const R {sy} = {printer.doprint(e)};")
        lines.append(f"f[{b.slot}] = {printer.doprint(reduced[0])};")
        for (_, d), e in zip(v_syms, reduced[1:]):
            lines.append(f"J[{plan.coefs[(b.slot, d)]}] = {printer.doprint(e)};")
        return lines

    def evaluate(name: str, with_j: bool) -> List[str]:
        out = [f"    template <class R> static __device__ __forceinline__ void {name}(const R* y, const R* g, "
               f"const R* __restrict__ ps, const R* ds, R t, int lane, R* f{', R* J' if with_j else ''})", "    {",
               "        (void)y; (void)g; (void)ps; (void)ds; (void)t; (void)lane;"]
        bodies = plan.bodies_fj if with_j else plan.bodies_f
        covered: Dict[int, int] = {}
        for b in bodies:
            covered[b.slot] = max(covered.get(b.slot, 0), len(b.lanes))
        for k in range(slots):
            if covered.get(k, 0) < 32:
                out.append(f"        f[{k}] = R(0);")
        if with_j:
            for (k, _), i in plan.coefs.items():
                if covered.get(k, 0) < 32:
                    out.append(f"        J[{i}] = R(0);")
        for b in bodies:
            cond = _lane_condition(b.lanes)
            out.append(f"        {'if (' + cond + ') ' if cond else ''}{{")
            out += ["            " + ln for ln in body_lines(b, with_j)]
            out.append("        }")
        return out + ["    }"]

    jm = ["    template <class R> static __device__ __forceinline__ void jmv_reg(const R* v, const R* g, const R* J, "
          "R* out)", "    {", "        (void)v; (void)g; (void)J;"]
    for k in range(slots):
        terms = [f"J[{i}] * {read('v', kk, d)}" for (kk, d), i in plan.coefs.items() if kk == k]
        jm.append(f"        out[{k}] = {' + '.join(terms) if terms else 'R(0)'};")
    jm.append("    }")
    tables = []
    for fn, vals in (("slot_base", plan.lanes.base), ("slot_count", plan.lanes.count),
                     *((name, [g[q] for g in plan.gathers]) for q, name in enumerate(("g_slot", "g_shift", "g_mode")))):
        vals = [str(v) for v in vals] or ["0"]
        tables.append(f"    static __device__ constexpr int {fn}(int i) {{ constexpr int v[{len(vals)}] = "
                      f"{{{', '.join(vals)}}}; return v[i]; }}")
    return "\n".join([f"    static constexpr int SLOTS = {slots}, LANE_STRIDE = {plan.lanes.stride};",
                      f"    static constexpr int NC = {len(plan.coefs)};   // coefficients per lane",
                      f"    static constexpr int NG = {len(plan.gathers)};   // exchanged values per lane",
                      *tables, *evaluate("f_reg", False), *evaluate("fj_reg", True), *jm])


def generate_warp_system(system: SymbolicODE, struct_name: str = "WarpSystem") -> WarpSystemCode:
    """Class-grouped right-hand side and Jacobian-vector product."""
    n = system.num_states
    ys = list(system.state_symbols)
    kind_of: Dict[sp.Symbol, Tuple[str, int]] = {}
    for i, s in enumerate(ys):
        kind_of[s] = ("y", i)
    for i, s in enumerate(system.parameter_symbols):
        kind_of[s] = ("p", i)
    for i, s in enumerate(system.driver_symbols):
        kind_of[s] = ("d", i)
    vs = [sp.Symbol(f"_vcomp{i:06d}", real=True) for i in range(n)]  # padded: name order = index order
    kind_v = dict(kind_of)
    for i, s in enumerate(vs):
        kind_v[s] = ("v", i)
    f = system.rhs_expressions()
    J = system.jacobian()
    jv = []
    for i in range(n):
        terms = [J[i, k] * vs[k] for k in range(n) if J[i, k] != 0]
        jv.append(sp.Add(*terms) if terms else sp.Integer(0))
    cf = group_classes(f, kind_of)
    cj = group_classes(jv, kind_v)
    tables: List[str] = []
    body_f, fl_f = _emit_classes("dxdt_lanes", cf, False, tables)
    body_j, fl_j = _emit_classes("jmv_lanes", cj, True, tables)
    flops = {"dxdt": fl_f, "jmv": fl_j}
    # J cached at each linearisation: its nonzero coefficients evaluated
    # together with f, then every J v is a short sum over shared memory
    nnz = sum(1 for i in range(n) for k in range(n) if J[i, k] != 0)
    cached, n_fj = [], 0
    register, slots, coefs = "    static constexpr int NC = 0, NG = 0, SLOTS = 0;", 0, 0
    if 0 < nnz <= CACHED_JAC_MAX:
        cfj = group_classes([sp.Tuple(f[i], jv[i]) for i in range(n)], kind_v)
        body_fj, body_jc, stored, fl_fj, fl_jc = _emit_cached_jacobian(cfj, tables)
        cached = [body_fj, body_jc]
        plan = _register_plan(n, cf, cfj)
        if plan is not None:
            register = _emit_register_lanes(cf, cfj, plan)
            slots, coefs = len(plan.lanes.base), len(plan.coefs)
        n_fj = len(cfj)
        nnz = stored
        flops.update({"fj": fl_fj, "jmv_cached": fl_jc})
    else:
        nnz = 0
    src = [*(t.strip() for t in tables),
           f"struct {struct_name} {{",
           f"    static constexpr int N = {n};",
           f"    static constexpr int NP = {system.num_parameters};",
           f"    static constexpr int ND = {system.num_drivers};",
           f"    static constexpr int NNZ = {nnz};",
           register,
           body_f,
           body_j,
           *cached,
           "};"]
    return WarpSystemCode(source="\n".join(src), n_classes_f=len(cf), n_classes_jv=len(cj),
                          flops=flops, nnz=nnz, n_classes_fj=n_fj, register_slots=slots, register_coefs=coefs)
