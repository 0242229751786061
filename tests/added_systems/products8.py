"""Eight quadrics in eight unknowns, each with sixteen products of its own (136 parameters)."""
import sympy as sp

NAME = "products8"
UNKNOWNS = list(sp.symbols("x0:8"))
_pairs = [(i, j) for i in range(8) for j in range(i, 8)]
_a = [sp.symbols(f"a{k}_0:16") for k in range(8)]
_c = list(sp.symbols("c0:8"))
PARAMS = [q for row in _a for q in row] + _c
EQUATIONS = [sum(_a[k][m] * UNKNOWNS[_pairs[(9 * k + m) % 36][0]] * UNKNOWNS[_pairs[(9 * k + m) % 36][1]]
                 for m in range(16)) + _c[k] for k in range(8)]
SOLVED = _c
