"""Two cubics in two unknowns: their derivatives have the factor 3, which is not exact."""
import sympy as sp

NAME = "cubic2"
x, y = UNKNOWNS = list(sp.symbols("x y"))
a, b, c, d, e, f = PARAMS = list(sp.symbols("a b c d e f"))
EQUATIONS = [a * x**3 + b * x * y**2 + c * y + d, b * y**3 + e * x**2 * y + a * x + f]
SOLVED = [d, f]
