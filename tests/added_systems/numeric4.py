"""Four quadrics in four unknowns with coefficients that are numbers, 65 of them different."""
import sympy as sp

NAME = "numeric4"
UNKNOWNS = list(sp.symbols("x0:4"))
PARAMS = list(sp.symbols("c0:4"))
_monomials = [UNKNOWNS[i] * UNKNOWNS[j] for i in range(4) for j in range(i, 4)] + UNKNOWNS
EQUATIONS = [sum(sp.Rational((m + 2) ** (k + 2) % 97, 32) * t for m, t in enumerate(_monomials)) + PARAMS[k]
             for k in range(4)]
SOLVED = PARAMS
