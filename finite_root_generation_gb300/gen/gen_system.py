"""Generate the CSE'd straight-line evaluation of the Stephenson II loop-closure
system, its Jacobian nonzeros and its t-derivative, for the CUDA tracker.

The system is FSYS of the reference (htpykinematics.cu:8-126): for each j = 1..7 three
equations (rows j-1, j+6, j+13) in the 22 homogeneous unknowns
Z = [A,B,C,D,F,G,H, Ac..Hc, U1..U7, Z0] and the 30 parameters
q = [P0..P7, Pc0..Pc7, Q1..Q7, Qc1..Qc7]. Equation j involves only U_j among the U's, so
one "group" evaluation per j yields F (3 values), dF/dZ (8 + 6 + 16 nonzeros, the
sparsity of JVAR, htpykinematics.cu:129-1129) and dF/dt = dF/dq . dq/dt (the t
column of JH, htpysupport.cu:113-121) in one pass.

The equations are restated here symbolically and differentiated by sympy; the
reciprocals 1/U, 1/(F-B), 1/(H-C), 1/(Fc-Bc), 1/(Hc-Cc) are carried as symbols with
their own chain rule so that the emitted code has no division. Quantities that do
not depend on j are hoisted into a per-point "shared" block.

Output: ../csrc/frg_system_gen.cuh (committed; regenerate with
``python finite_root_generation_gb300/gen/gen_system.py``). The script also prints
the operation counts used for the roofline's algorithmic FLOPs per evaluation.
"""
from __future__ import annotations

import ast
import os
import re

import numpy as np
import sympy as sp

HERE = os.path.dirname(os.path.abspath(__file__))
OUT = os.path.join(HERE, "..", "csrc", "frg_system_gen.cuh")

# ---- symbols -----------------------------------------------------------------
A, B, C, D, F, G, H = sp.symbols("A B C D F G H")
Ac, Bc, Cc, Dc, Fc, Gc, Hc = sp.symbols("Ac Bc Cc Dc Fc Gc Hc")
U, z = sp.symbols("U z")
P0, Pc0, Pj, Pcj, Qj, Qcj = sp.symbols("P0 Pc0 Pj Pcj Qj Qcj")
dP0, dPc0, dPj, dPcj, dQj, dQcj = sp.symbols("dP0 dPc0 dPj dPcj dQj dQcj")
# reciprocals carried as symbols
iU, e1, e2, ec1, ec2 = sp.symbols("iU e1 e2 ec1 ec2")

VARS = [A, B, C, D, F, G, H, Ac, Bc, Cc, Dc, Fc, Gc, Hc, U, z]
PARAMS = [(P0, dP0), (Pc0, dPc0), (Pj, dPj), (Pcj, dPcj), (Qj, dQj), (Qcj, dQcj)]
# d(reciprocal)/d(var) rules
RECIP = {
    iU: {U: -iU**2},
    e1: {F: -e1**2, B: e1**2},
    e2: {H: -e2**2, C: e2**2},
    ec1: {Fc: -ec1**2, Bc: ec1**2},
    ec2: {Hc: -ec2**2, Cc: ec2**2},
}


def total_diff(expr, v):
    d = sp.diff(expr, v)
    for r, rules in RECIP.items():
        if v in rules:
            d += sp.diff(expr, r) * rules[v]
    return sp.expand(d) if False else d


# ---- the three equation families (htpykinematics.cu:36-122) -------------------
p, pc, p0, pc0 = Pj * z, Pcj * z, P0 * z, Pc0 * z
a, ac = C - A, Cc - Ac
S = Pj * Pcj + P0 * Pc0
m = pc - Ac - ac * Qcj
n = p - A - a * Qj
fI = (-S * z**3 + ac * Qcj * z * (p - A) + Ac * z * (a + p) + Hc * z * (p0 - C) + a * Qj * z * (pc - Ac)
      + A * z * (ac + pc) + U * (p0 - H) * m + H * z * (pc0 - Cc) + z**2 * n * (pc0 - Hc) * iU)
fII = (z**2 * (Bc * Pj + B * Pcj) - S * z**3 + Fc * z * (p0 - B) + U * (p0 - F) * (pc - Bc)
       + F * z * (pc0 - Bc) + z**2 * (p - B) * (pc0 - Fc) * iU)
X = (A - B) + a * Qj - (D - B) * (p - B) * e1 + (G - C) * n * e2
Xc = (Ac - Bc) + ac * Qcj - (Dc - Bc) * (pc - Bc) * ec1 + (Gc - Cc) * m * ec2
W = -(D - B) * (p0 - F) * e1 + (G - C) * (p0 - H) * e2
Wc = -(Dc - Bc) * (pc0 - Fc) * ec1 + (Gc - Cc) * (pc0 - Hc) * ec2
fIII = (G - D) * (Gc - Dc) * z - z * X * Xc + U * W * Xc + z**2 * X * Wc * iU - z * W * Wc

FAMILIES = [
    ("I", fI, [A, C, H, Ac, Cc, Hc, U, z]),
    ("II", fII, [B, F, Bc, Fc, U, z]),
    ("III", fIII, [A, B, C, D, F, G, H, Ac, Bc, Cc, Dc, Fc, Gc, Hc, U, z]),
]
# column of each variable in Z (U -> 13 + j)
COL = {A: 0, B: 1, C: 2, D: 3, F: 4, G: 5, H: 6, Ac: 7, Bc: 8, Cc: 9, Dc: 10, Fc: 11, Gc: 12, Hc: 13,
       U: -1, z: 21}

# j-independent inputs the group code reads from the shared block
SHARED = {
    "z2": z**2, "z3": z**3, "p0": P0 * z, "pc0": Pc0 * z, "S0": P0 * Pc0,
    "k1": D - B, "k2": G - C, "kc1": Dc - Bc, "kc2": Gc - Cc,
    "GD": (G - D) * (Gc - Dc),
}


def outputs():
    outs = []
    names = []
    for fam, f, vars_ in FAMILIES:
        outs.append(f)
        names.append(("f", fam, None))
        for v in vars_:
            outs.append(total_diff(f, v))
            names.append(("j", fam, v))
        tcol = sum(total_diff(f, prm) * dprm for prm, dprm in PARAMS)
        outs.append(tcol)
        names.append(("t", fam, None))
    return names, outs


def count_ops(exprs):
    """(complex muls, complex adds, scalar*complex) of straight-line code."""
    cm = ca = sm = 0
    for e in exprs:
        for node in sp.preorder_traversal(e):
            if isinstance(node, sp.Mul):
                num = [a for a in node.args if a.is_Number]
                sym = [a for a in node.args if not a.is_Number]
                k = len(sym)
                cm += max(k - 1, 0)
                if num and num[0] not in (1, -1):
                    sm += 1
            elif isinstance(node, sp.Add):
                ca += len(node.args) - 1
            elif isinstance(node, sp.Pow):
                ex = int(node.exp)
                cm += abs(ex) - 1
    return cm, ca, sm


class Printer:
    def __init__(self):
        self.lines = []

    def expr(self, e) -> str:
        if e.is_Symbol:
            return e.name
        if e.is_Number:
            return f"cx<T>(T({float(e)!r}))"
        if isinstance(e, sp.Pow):
            base = self.expr(e.args[0])
            ex = int(e.args[1])
            assert ex >= 2, e
            return "(" + "*".join([base] * ex) + ")"
        if isinstance(e, sp.Mul):
            coeff, rest = e.as_coeff_Mul()
            factors = sp.Mul.make_args(rest)
            body = "*".join(self.expr(f) if not isinstance(f, sp.Add) else "(" + self.expr(f) + ")" for f in factors)
            if coeff == 1:
                return body
            if coeff == -1:
                return f"(-({body}))"
            return f"(T({float(coeff)!r})*({body}))"
        if isinstance(e, sp.Add):
            terms = list(sp.Add.make_args(e))
            out = ""
            for i, t in enumerate(terms):
                coeff, rest = t.as_coeff_Mul()
                if coeff.is_negative:
                    tt = self.expr(-t)
                    out += f" - {tt}" if i else f"(-{tt})"
                else:
                    tt = self.expr(t)
                    out += f" + {tt}" if i else tt
            return out
        raise TypeError(type(e), e)


# ---- the evaluation split over a block's four warps -------------------------------
# Quantities that a path's own warp computes once per step and every slice reads. Each
# has a plain form (side 0) and its conjugate partner (side 1), computed by the same
# instructions on different lanes; `pj` marks those that differ per group. The printed
# forms are what the kernel's preparation evaluates: the generator checks them.
HOISTED = [
    # name, per group, side 0 (symbol form), side 1
    ("pz", False, "P0*z", "Pc0*z"),
    ("fp", False, "F - pz0", "Fc - pz1"),
    ("hp", False, "H - pz0", "Hc - pz1"),
    ("bd", False, "B - D", "Bc - Dc"),
    ("ebd", False, "e1*bd0", "ec1*bd1"),
    ("cg", False, "C - G", "Cc - Gc"),
    ("ecg", False, "e2*cg0", "ec2*cg1"),
    ("v", False, "fp0*ebd0 - hp0*ecg0", "fp1*ebd1 - hp1*ecg1"),
    ("ac", False, "A - C", "Ac - Cc"),
    ("pjz", True, "Pj*z", "Pcj*z"),
    ("ap", True, "A - pjz0", "Ac - pjz1"),
    ("bp", True, "B - pjz0", "Bc - pjz1"),
    ("qa", True, "Qj*ac0", "Qcj*ac1"),
    ("aq", True, "ap0 - qa0", "ap1 - qa1"),
    ("eaq", True, "e2*aq0", "ec2*aq1"),
    ("w", True, "B - A + qa0 + bp0*ebd0 - cg0*eaq0", "Bc - Ac + qa1 + bp1*ebd1 - cg1*eaq1"),
]
# the equations-alone form's own order of the same sum
RESIDUAL_FORMS = {"w": ("B + qa0 - A + bp0*ebd0 - ecg0*aq0", "Bc + qa1 - Ac + bp1*ebd1 - ecg1*aq1")}
# Which warp evaluates which outputs: 4 parts of equal cost (492 real FMA-pipe operations
# each, found by a local search over the outputs' closures; the whole group is 1,770).
EVAL_SLICES = [
    ["dI[5]", "dIII[1]", "dIII[2]", "dIII[3]", "dIII[4]", "dIII[5]", "dIII[6]", "dIII[15]"],
    ["fI", "dI[0]", "dI[1]", "dI[2]", "dI[6]", "tI", "fII", "dII[0]", "dII[1]", "dII[4]", "tII", "dIII[14]"],
    ["fIII", "dIII[0]", "dIII[7]", "dIII[8]", "dIII[9]", "dIII[11]", "tIII"],
    ["dI[3]", "dI[4]", "dI[7]", "dII[2]", "dII[3]", "dII[5]", "dIII[10]", "dIII[12]", "dIII[13]"],
]
# column of each derivative slot in the group's row: links 0..13, Z0 14, t 15, U_j 16, F 17
ROW_COLS = {"I": [0, 2, 6, 7, 9, 13, 16, 14], "II": [1, 4, 8, 11, 16, 14], "III": list(range(14)) + [16, 14]}


def hoisted_symbols(repl, pr, other={}):
    """{temporary's name: hoisted quantity} of the temporaries that have a hoisted quantity's
    value, after checking in single precision on random inputs that both forms round alike
    (a - b, a + (-b) and -((-a) + b) do; another order of a sum does not)."""
    base = {n: sp.Symbol(n) for n in ("z e1 e2 ec1 ec2 P0 Pc0 Pj Pcj Qj Qcj A B C D F G H "
                                      "Ac Bc Cc Dc Fc Gc Hc").split()}
    forms = {f"{name}{side}": other.get(name, (f0, f1))[side] for name, _, f0, f1 in HOISTED for side in (0, 1)}
    values = {}
    for key, form in forms.items():
        values[key] = sp.sympify(form, locals={**base, **values})
    full, found = {}, {}
    for s_, e in repl:
        full[s_] = sp.expand(e.subs(full))
        for key, val in values.items():
            if sp.expand(full[s_] - val) == 0:
                found[s_.name] = key
    rng = np.random.default_rng(1)
    names = set(base) | {y.name for _, e in repl for y in e.free_symbols}
    for _ in range(200):
        env = {n: np.complex64(complex(*rng.normal(size=2))) for n in sorted(names)}
        env.update(cx=lambda v: v, T=np.float32)
        for key, form in forms.items():
            env[key] = eval(form, {}, env)
        for s_, e in repl:
            env[s_.name] = eval(pr.expr(e).replace("cx<T>", "cx"), {}, env)
            if s_.name in found:
                assert env[s_.name] == env[found[s_.name]], (s_.name, found[s_.name])
    return found


def slice_lines(repl, wanted, found, loads, pr):
    """Straight-line code of the outputs `wanted` (expr, statement) from the hoisted quantities."""
    defs = {s_.name: e for s_, e in repl}
    need, stack = set(), [x.name for e, _ in wanted for x in e.free_symbols]
    used = set()
    while stack:
        x = stack.pop()
        if x in found or x not in defs:
            used.add(x)
        elif x not in need:
            need.add(x)
            stack += [y.name for y in defs[x].free_symbols]
    out = [f"    const CX {x}({loads(x, found.get(x))});" for x in sorted(used)]
    # a real multiple stays unevaluated where CX has a type for it, to round as the fused form
    scaled = {s_ for s_, e in repl if abs(e.as_coeff_Mul()[0]) != 1 and e.as_coeff_Mul()[0].is_Number}
    out += [f"    const {'auto' if s_ in scaled else 'CX'} {s_} = {pr.expr(e)};" for s_, e in repl if s_.name in need]
    out += ["    " + st.format(pr.expr(e)) for e, st in wanted]
    return [ln.replace("cx<T>(T(", "CX(T(") for ln in out]


INDEP = [h[0] for h in HOISTED if not h[1]]
PERJ = [h[0] for h in HOISTED if h[1]]


def load_of(x, key):
    """Where a slice reads the value named x (a hoisted quantity `key` if it is one)."""
    links = ["A", "B", "C", "D", "F", "G", "H", "Ac", "Bc", "Cc", "Dc", "Fc", "Gc", "Hc"]
    if key:
        name, side = key[:-1], key[-1]
        if name in INDEP:
            return f"in.sa[{side}][FRG_IN_{name.upper()}]"
        return f"in.sb[{side}][FRG_IN_{name.upper()}][j - 1]"
    if x in links:
        return f"Y[{links.index(x)}]"
    q = {"P0": "0", "Pc0": "8", "Pj": "j", "Pcj": "8 + j", "Qj": "15 + j", "Qcj": "22 + j"}
    e = {"e1": "0", "e2": "1", "ec1": "2", "ec2": "3"}
    if x in q:
        return f"in.q[{q[x]}]"
    if x[0] == "d" and x[1:] in q:
        return f"dq[{q[x[1:]]}]"
    if x in e:
        return f"in.e[{e[x]}]"
    return {"z": "Y[21]", "z2": "in.z2", "z3": "in.z3", "U": "Y[13 + j]", "iU": "in.iU[j - 1]"}[x]


def operand_of(x, key):
    """(segment, index, 1 if one per group) of the value named x: segment 0 the point, 1 FrgEvalIn."""
    load = load_of(x, key)
    index = [eval(i, {"j": 1, **{f"FRG_IN_{n.upper()}": (INDEP + PERJ).index(n) - (len(INDEP) if n in PERJ else 0)
                                 for n in INDEP + PERJ}}) for i in re.findall(r"\[(.*?)\]", load)]
    if load.startswith("Y"):
        return 0, index[0], int("j" in load)
    start = {"z2": 0, "z3": 1, "e": 2, "q": 6, "iU": 38, "sa": 46, "sb": 46 + 2 * len(INDEP)}
    name = re.match(r"in\.(\w+)", load).group(1)
    flat = {"sa": lambda s_, k: s_ * len(INDEP) + k, "sb": lambda s_, k, g: (s_ * len(PERJ) + k) * 8 + g}
    return 1, start[name] + flat.get(name, lambda k=0: k)(*index), int("j" in load)


# name and side -> form, as the residual has it
HOISTED_FORMS = {f"{name}{side}": (RESIDUAL_FORMS.get(name, forms))[side]
                 for name, _, *forms in HOISTED for side in (0, 1)}


class ResidualTape:
    """Equations of some groups as a schedule of complex operations for a warp: pairs of lanes
    (one per real component) take one operation each, so a step is up to WIDTH products or
    sums that do not depend on each other. Operations, operand order and association are the
    printed code's, an operation common to several groups is done once; a minus sign travels
    with a value's use ((-a) b = -(a b) and (-a) + b = -(a - b) round alike). A value lives in
    a temporary until its last use; a step writes none that it reads."""

    WIDTH = 16

    def __init__(self, repl, reduced, found, items, products):
        self.defs, self.found = {s_.name: d for s_, d in repl}, found
        self.ops, self.memo = [], {}
        self.outs = []  # (equation, group, operation, sign)
        for eq, g in items:
            self.seen = {}
            ref, sign = self.expr(reduced[eq], g)
            self.outs.append((eq, g, ref[1], sign))
        self.schedule(products)

    def value(self, name, g):
        """A prepared value, or a hoisted quantity from the form that eval_prep evaluates."""
        if name == "z2" or name == "z3":
            return self.op("mul", self.value("z" if name == "z2" else "z2", g), self.value("z", g))
        key = self.found.get(name, name)
        form = HOISTED_FORMS.get(key)
        if form is None:
            seg, index, per_group = operand_of(name, None)
            return "v", (seg, index + g * per_group)

        def walk(e):
            if isinstance(e, ast.Name):
                return self.value(e.id, g)
            kind = "mul" if isinstance(e.op, ast.Mult) else "add"
            return self.op(kind, walk(e.left), walk(e.right), int(isinstance(e.op, ast.Sub)))

        return walk(ast.parse(form, mode="eval").body)

    def op(self, kind, x, y, sub=0):
        key = (kind, x, y, sub)
        if key not in self.memo:
            self.memo[key] = ("n", len(self.ops))
            self.ops.append(key)
        return self.memo[key]

    def expr(self, e, g):
        if e.is_Symbol:
            if e.name in self.found or e.name not in self.defs:
                return self.value(e.name, g), 1
            if e.name not in self.seen:
                self.seen[e.name] = self.expr(self.defs[e.name], g)
            return self.seen[e.name]
        if isinstance(e, sp.Mul):
            coeff, rest = e.as_coeff_Mul()
            assert abs(coeff) == 1, e
            parts = [self.expr(f, g) for f in sp.Mul.make_args(rest)]
            out = parts[0]
            for v in parts[1:]:
                out = self.op("mul", out[0], v[0]), out[1] * v[1]
            return out[0], out[1] * int(coeff)
        assert isinstance(e, sp.Add), e
        out = None
        for t in sp.Add.make_args(e):
            v = self.expr(t, g)
            out = v if out is None else (self.op("add", out[0], v[0], int(out[1] != v[1])), out[1])
        return out

    def schedule(self, products):
        """From the last step back: each step takes operations of one kind whose users are all
        in later steps, those with the longest chain before them first. At least `products`
        ready products go before sums: a term is then computed shortly before it is added,
        and few temporaries are live."""
        n = len(self.ops)
        need = [{r[1] for r in o[1:3] if r[0] == "n"} for o in self.ops]
        users = [{k for k in range(n) if d in need[k]} for d in range(n)]
        depth = [0] * n
        for k in range(n):
            depth[k] = (3 if self.ops[k][0] == "mul" else 2) + max([depth[d] for d in need[k]], default=0)
        done, back = set(), []
        while len(done) < n:
            ready = sorted((k for k in range(n) if k not in done and users[k] <= done), key=lambda k: (-depth[k], -k))
            many = sum(self.ops[k][0] == "mul" for k in ready) >= products
            kind = "mul" if many else self.ops[ready[0]][0]
            pick = [k for k in ready if self.ops[k][0] == kind][:self.WIDTH]
            back.append(pick)
            done |= set(pick)
        keep = {k for _, _, k, _ in self.outs}
        free, self.where, self.steps = [], {}, []
        self.ntemps, ran = 0, set()
        for pick in reversed(back):
            for k in pick:
                if not free:
                    free.append(self.ntemps)
                    self.ntemps += 1
                self.where[k] = free.pop(0)
            self.steps.append([(self.ops[k][0] == "mul", self.ops[k][3], self.where[k],
                                *[r[1] if r[0] == "v" else (2, self.where[r[1]]) for r in self.ops[k][1:3]])
                               for k in pick])
            ran |= set(pick)
            free += sorted({self.where[d] for k in pick for d in need[k] if d not in keep and users[d] <= ran})


# A part's four warps: (equation, group) and the least number of ready products that go
# before sums; 17, 17, 17 and 13 steps (the last warp also takes the patch row), 207 temporaries
RESIDUAL_PARTS = [([(0, g) for g in range(4)] + [(1, g) for g in (2, 3)], 14),
                  ([(0, g) for g in range(4, 7)] + [(2, g) for g in (4, 5)], 12),
                  ([(2, g) for g in (0, 1, 2, 3, 6)], 8), ([(1, g) for g in (0, 1, 4, 5, 6)], 8)]


def residual_system():
    """The three equations alone: common subexpressions, equations, hoisted symbols."""
    f_outs = [o.subs(z**3, sp.Symbol("z3")).subs(z**2, sp.Symbol("z2")) for o in (fI, fII, fIII)]
    repl, reduced = sp.cse(f_outs, symbols=sp.numbered_symbols("y"), optimizations="basic")
    return repl, reduced, hoisted_symbols(repl, Printer(), RESIDUAL_FORMS)


def residual_tapes():
    repl, reduced, found = residual_system()
    return [ResidualTape(repl, reduced, found, items, products) for items, products in RESIDUAL_PARTS]


def emit_residual(lines, tapes):
    starts = [sum(len(t.steps) for t in tapes[:k]) for k in range(len(tapes) + 1)]
    temps = [sum(t.ntemps for t in tapes[:k]) for k in range(len(tapes) + 1)]
    seg = ["Y", "IN", "T"]
    lines += ["",
              "// The three equations at a point alone (their own common subexpressions) as schedules for a",
              "// part's four warps, residual_part in frg_team.cuh executes them. Warp k: steps START[k] ..",
              f"// START[k + 1] of {ResidualTape.WIDTH} words OP(result, a, b, b subtracted, product), values by",
              "// number in Y (the point), IN (FrgEvalIn) and T (temporaries; the last takes idle lanes' results), two steps",
              "// of padding at the end; then OUT(value, equation, group, negated), 7 per warp.",
              f"#define FRG_RESIDUAL_TEMPS {temps[-1] + 1}",
              f"#define FRG_RESIDUAL_START {{{', '.join(map(str, starts))}}}"]
    words = []
    for k, t in enumerate(tapes):
        for step in t.steps:
            for mul, sub, dst, a, b in step:
                ops = [f"{seg[s_]}({i + (temps[k] if s_ == 2 else 0)})" for s_, i in (a, b)]
                words.append(f"OP(T({temps[k] + dst}), {ops[0]}, {ops[1]}, {sub}, {int(mul)})")
            words += [f"OP(T({temps[-1]}), Y(0), Y(0), 0, {int(step[0][0])})"] * (t.WIDTH - len(step))
    words += ["0"] * (2 * ResidualTape.WIDTH)
    outs = []
    for k, t in enumerate(tapes):
        o = [f"OUT(T({temps[k] + t.where[n]}), {eq}, {g}, {int(s_ < 0)})" for eq, g, n, s_ in t.outs]
        outs += o + ["0xffff"] * (7 - len(o))
    for name, items in (("CODE(OP, Y, IN, T)", words), ("OUTS(OUT, T)", outs)):
        lines.append(f"#define FRG_RESIDUAL_{name} \\")
        row = "   "
        for i, w in enumerate(items):
            w += "," if i + 1 < len(items) else ""
            if len(row) + len(w) > 110:
                lines.append(row + " \\")
                row = "   "
            row += " " + w
        lines.append(row)


def emit_slices(lines, names, repl, reduced, pr):
    found = hoisted_symbols(repl, pr)
    by, slot = {}, {"I": 0, "II": 0, "III": 0}
    row = {"I": 0, "II": 1, "III": 2}
    for (kind, fam, v), e in zip(names, reduced):
        if kind in "ft":
            by[f"{kind}{fam}"] = (e, row[fam], 17 if kind == "f" else 15)
        else:
            by[f"d{fam}[{slot[fam]}]"] = (e, row[fam], ROW_COLS[fam][slot[fam]])
            slot[fam] += 1
    assert sorted(by) == sorted(n for s_ in EVAL_SLICES for n in s_)
    lines += ["",
              "// What one path's step needs besides its point: computed by the path's own warp, read by",
              "// the slices below. Side 0 holds a quantity's plain form, side 1 its conjugate partner.",
              "//   sa: " + ", ".join(INDEP) + "   (the same for every group)",
              "//   sb: " + ", ".join(PERJ) + "   (per group j)"]
    for name, pj, f0, _ in HOISTED:
        r = f"; for the residual alone {RESIDUAL_FORMS[name][0]}" if name in RESIDUAL_FORMS else ""
        lines.append(f"//   {name:4s} = {f0}{r}")
    for name in INDEP + PERJ:
        lines.append(f"#define FRG_IN_{name.upper()} {(INDEP + PERJ).index(name) - (len(INDEP) if name in PERJ else 0)}")
    lines += ["template <typename T>", "struct FrgEvalIn {",
              "  cx<T> z2, z3, e[4], q[32], iU[8];  // e: e1, e2, ec1, ec2; q(t); 1 / U_j at [j - 1]",
              f"  cx<T> sa[2][{len(INDEP)}], sb[2][{len(PERJ)}][8];", "};", "",
              "// One quarter of group j's evaluation (frg_group_eval's operations in its order): rows of",
              "// the group into M[(row * 18 + column) * 8 + g], columns 0..13 links, 14 Z0, 15 t, 16 U_j, 17 F.",
              "// CX: cx<T>, or a type with its operators whose values several lanes share.",
              "template <int SLICE, typename CX, typename T>",
              "__device__ __forceinline__ void frg_eval_slice(const cx<T>* Y, const FrgEvalIn<T>& in, const cx<T>* dq, int j,",
              "                                               int g, cx<T>* M) {"]
    for k, outs in enumerate(EVAL_SLICES):
        lines.append(f"  if constexpr (SLICE == {k}) {{")
        wanted = [(by[n][0], f"cx_put(M + {(by[n][1] * 18 + by[n][2]) * 8} + g, {{}});") for n in outs]
        lines += slice_lines(repl, wanted, found, load_of, pr)
        lines.append("  }")
    lines.append("}")
    emit_residual(lines, residual_tapes())


def main():
    names, outs = outputs()
    # hoist shared quantities: substitute them by symbols
    shared_syms = {k: sp.Symbol(k) for k in SHARED}
    rep = []
    for k, v in SHARED.items():
        rep.append((v, shared_syms[k]))
    outs = [o.subs(z**3, shared_syms["z3"]).subs(z**2, shared_syms["z2"]) for o in outs]
    repl, reduced = sp.cse(outs, symbols=sp.numbered_symbols("x"), optimizations="basic")
    cm, ca, sm = count_ops([r for _, r in repl] + reduced)
    pr = Printer()

    lines = []
    lines.append("// GENERATED by finite_root_generation_gb300/gen/gen_system.py -- do not edit.")
    lines.append("//")
    lines.append("// One j-group of the Stephenson II loop-closure system (reference FSYS,")
    lines.append("// htpykinematics.cu:36-122): the three equations (rows j-1, j+6, j+13), their")
    lines.append("// nonzero partial derivatives over Z (JVAR's sparsity, htpykinematics.cu:129-1129)")
    lines.append("// and the t-derivative dF/dq . dq/dt (JH's last column, htpysupport.cu:113-121).")
    lines.append(f"// Straight-line cost per group: {cm} complex mul, {ca} complex add/sub,")
    lines.append(f"// {sm} real-scalar x complex.")
    lines.append("#pragma once")
    lines.append("")
    lines.append(f"#define FRG_GEN_CMUL {cm}")
    lines.append(f"#define FRG_GEN_CADD {ca}")
    lines.append(f"#define FRG_GEN_SMUL {sm}")
    lines.append("")
    lines.append("// Output slots: fI, dI[8] over {A,C,H,Ac,Cc,Hc,U_j,Z0}, tI;")
    lines.append("//               fII, dII[6] over {B,F,Bc,Fc,U_j,Z0}, tII;")
    lines.append("//               fIII, dIII[16] over {A..H,Ac..Hc,U_j,Z0}, tIII.")
    lines.append("template <typename T>")
    lines.append("struct FrgGroupOut {")
    lines.append("  cx<T> fI, dI[8], tI;")
    lines.append("  cx<T> fII, dII[6], tII;")
    lines.append("  cx<T> fIII, dIII[16], tIII;")
    lines.append("};")
    lines.append("")
    lines.append("// Column in Z of each derivative slot (U_j's column is 13 + j, marked -1).")
    for fam, _, vars_ in FAMILIES:
        cols = ", ".join(str(COL[v]) for v in vars_)
        lines.append(f"#define FRG_COLS_{fam} {{{cols}}}")
    lines.append("")
    lines.append("template <typename T>")
    lines.append("__device__ __forceinline__ void frg_group_eval(")
    lines.append("    const cx<T> A, const cx<T> B, const cx<T> C, const cx<T> D, const cx<T> F, const cx<T> G,")
    lines.append("    const cx<T> H, const cx<T> Ac, const cx<T> Bc, const cx<T> Cc, const cx<T> Dc, const cx<T> Fc,")
    lines.append("    const cx<T> Gc, const cx<T> Hc, const cx<T> z,")
    lines.append("    const cx<T> e1, const cx<T> e2, const cx<T> ec1, const cx<T> ec2,")
    lines.append("    const cx<T> z2, const cx<T> z3,")
    lines.append("    const cx<T> P0, const cx<T> Pc0, const cx<T> dP0, const cx<T> dPc0,")
    lines.append("    const cx<T> U, const cx<T> iU, const cx<T> Pj, const cx<T> Pcj, const cx<T> Qj, const cx<T> Qcj,")
    lines.append("    const cx<T> dPj, const cx<T> dPcj, const cx<T> dQj, const cx<T> dQcj,")
    lines.append("    FrgGroupOut<T>& o) {")
    for s_, e in repl:
        lines.append(f"  const cx<T> {s_} = {pr.expr(e)};")
    slot = {"I": 0, "II": 0, "III": 0}
    for (kind, fam, v), e in zip(names, reduced):
        if kind == "f":
            lines.append(f"  o.f{fam} = {pr.expr(e)};")
        elif kind == "t":
            lines.append(f"  o.t{fam} = {pr.expr(e)};")
        else:
            lines.append(f"  o.d{fam}[{slot[fam]}] = {pr.expr(e)};")
            slot[fam] += 1
    lines.append("}")
    # ---- F only (the three equations), for the residuals next to FP32 Jacobians
    frepl, fred, _ = residual_system()
    fcm, fca, fsm = count_ops([r for _, r in frepl] + fred)
    lines.insert(8, f"// The three equations alone: {fcm} complex mul, {fca} complex add/sub, {fsm} real x complex.")
    emit_slices(lines, names, repl, reduced, pr)
    used = set()
    for _, e in repl:
        used |= {s.name for s in e.free_symbols}
    for e in reduced:
        used |= {s.name for s in e.free_symbols}
    with open(OUT, "w") as fh:
        fh.write("\n".join(lines) + "\n")
    print(f"wrote {OUT}: {len(repl)} temporaries; per group {cm} cmul, {ca} cadd, {sm} smul; "
          f"F only {fcm} cmul, {fca} cadd")
    print("free inputs used:", sorted(u for u in used if not u.startswith("x")))


if __name__ == "__main__":
    main()
