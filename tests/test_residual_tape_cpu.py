"""The refinement residual's schedules for a part's four warps (gen/gen_system.py
ResidualTape) against the printed expressions: executed step by step in single precision on
random inputs, every equation of every group must be equal bit for bit, no step may read
what it writes, and the parts' temporaries must not overlap."""
import re

import numpy as np
import pytest

pytest.importorskip("sympy")

from finite_root_generation_gb300.gen import gen_system as gs  # noqa: E402


@pytest.mark.parametrize("part", range(4))
def test_schedule_equals_printed_equations(part):
    tape, (items, _) = gs.residual_tapes()[part], gs.RESIDUAL_PARTS[part]
    repl, reduced, found = gs.residual_system()
    pr = gs.Printer()
    rng = np.random.default_rng(part)
    assert [o[:2] for o in tape.outs] == items
    for _ in range(20):
        def draw(n):
            return [np.complex64(complex(*rng.normal(size=2))) for _ in range(n)]

        mem = [draw(23), draw(46), [np.complex64(0)] * tape.ntemps]  # the point, prepared values
        want = {}
        for eq, g in items:
            env = {"T": np.float32, "cx": np.complex64}

            def value(name):
                if name in env:
                    return env[name]
                form = {"z2": "z*z", "z3": "z2*z"}.get(name) or gs.HOISTED_FORMS.get(found.get(name, name))
                if form:
                    env[name] = eval(form, {}, {x: value(x) for x in re.findall(r"[A-Za-z]\w*", form)})
                else:
                    seg, index, per_group = gs.operand_of(name, None)
                    env[name] = mem[seg][index + g * per_group]
                return env[name]

            defined = {s.name for s, _ in repl}
            for name in {s.name for e in [*reduced, *(d for _, d in repl)] for s in e.free_symbols}:
                if name in found or name not in defined:
                    value(name)
            for s, d in repl:
                if s.name not in found:
                    env[s.name] = eval(pr.expr(d), {}, env)
            want[eq, g] = np.complex64(eval(pr.expr(reduced[eq]), {}, env))
        for step in tape.steps:
            assert len(step) <= tape.WIDTH and len({mul for mul, *_ in step}) == 1
            written = {dst for _, _, dst, _, _ in step}
            assert len(written) == len(step)
            assert not written & {i for _, _, _, a, b in step for seg, i in (a, b) if seg == 2}
            new = []
            for mul, sub, dst, (sa, ia), (sb, ib) in step:
                a, b = mem[sa][ia], mem[sb][ib]
                new.append((dst, a * b if mul else (a - b if sub else a + b)))
            for dst, v in new:
                mem[2][dst] = v
        for eq, g, k, sign in tape.outs:
            got = mem[2][tape.where[k]]
            assert (got if sign > 0 else -got) == want[eq, g]
