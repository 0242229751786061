"""Twelve sparse quadratic equations in twelve unknowns."""
import sympy as sp

NAME = "sparse12"
UNKNOWNS = list(sp.symbols("x0:12"))
PARAMS = list(sp.symbols("a0:12 b0:12 c0:12"))
_a, _b, _c = PARAMS[:12], PARAMS[12:24], PARAMS[24:]
EQUATIONS = [_a[i] * UNKNOWNS[i] * UNKNOWNS[(i + 1) % 12] + _b[i] * UNKNOWNS[(i + 5) % 12] + UNKNOWNS[i] + _c[i]
             for i in range(12)]
SOLVED = _c
