"""The plug-in rows' schedule for a warp (gen/gen_plugins.py Tape) against the generated
straight-line code: executed step by step in single precision on random inputs, every row
entry and equation must be equal bit for bit (the same operations on the same operands),
and no step may read what it writes or exceed its 16 operations."""
import re

import numpy as np
import pytest

pytest.importorskip("sympy")

from finite_root_generation_gb300.gen import gen_plugins  # noqa: E402


@pytest.mark.parametrize("k", [0, 1], ids=["conic2", "burmester5"])
def test_schedule_equals_straight_line_code(k):
    mod = gen_plugins.load_plugins()[k]
    info = gen_plugins.analyse(mod)
    tape = gen_plugins.Tape(info)
    nz, npar = info["nv"] + 1, info["np"]
    code = "\n".join(gen_plugins.emit_rows(mod, info, "cuda")).replace("cx<T>", "cx")
    rng = np.random.default_rng(11)
    for _ in range(20):
        def draw(n):
            return [np.complex64(complex(*rng.normal(size=2))) for _ in range(n)]

        Y, q, dq = draw(nz), draw(npar), draw(npar)
        env = dict(Y=Y, q=q, dq=dq, T=np.float32, cx=np.complex64)
        for name, e in re.findall(r"const cx (\w+) = (.*?);", code):
            env[name] = eval(e, {}, env)
        want = [np.complex64(eval(e, {}, env)) for e in re.findall(r"M\[.*?\] = (.*?);", code)]
        want += [np.complex64(eval(e, {}, env)) for e in re.findall(r"F\[.*?\] = (.*?);", code)]
        reg = Y + q + dq + [np.complex64(c) for c in tape.consts]
        reg += [np.complex64(0)] * (tape.nregs - len(reg))
        words = tape.words()
        assert len(words) == tape.WIDTH * len(tape.steps)
        for s in range(0, len(words), tape.WIDTH):
            step = words[s:s + tape.WIDTH]
            written = {w & 1023 for w in step} - {tape.nregs - 1}
            assert not written & {r for w in step for r in ((w >> 10) & 1023, (w >> 20) & 1023)}
            new = []
            for w in step:
                a, b = reg[(w >> 10) & 1023], reg[(w >> 20) & 1023]
                new.append((w & 1023, a * b if w >> 31 else (a - b if (w >> 30) & 1 else a + b)))
            for d, v in new:
                reg[d] = v
        got = [-reg[w & 1023] if w >> 10 else reg[w & 1023] for w in tape.out_words()]
        assert got == want
