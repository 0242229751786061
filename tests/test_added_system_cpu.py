"""Plug-in systems other than the shipped ones, generated from a module as a user adds one,
on the CPU: the two tracking kernels of a plug-in (a path per thread, a path per warp) are
the same computation, so a path must come out of both alike, whatever kernel its call's size
selects. The kernels' own source runs here (tests/warp_emu): each path starts, takes a few
steps and ends on the step limit (FP64) or is still in hand at it (FP32 stage)."""
import importlib.util
import os
import re
import subprocess

import numpy as np
import pytest

import finite_root_generation_gb300 as frg
from finite_root_generation_gb300 import build as frg_build

pytest.importorskip("sympy")

from finite_root_generation_gb300.gen import gen_plugins  # noqa: E402

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(gen_plugins.__file__), "..", "csrc")


def system(name):
    """tests/added_systems/<name>.py, as a user's module."""
    spec = importlib.util.spec_from_file_location(name, os.path.join(HERE, "added_systems", name + ".py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


class Value:
    """A single-precision complex value."""

    def __init__(self, v):
        self.v = np.complex64(v.v if isinstance(v, Value) else v)

    def __mul__(self, o):
        return Value(self.v * Value(o).v)

    def __add__(self, o):
        return o.plus(self, 1) if isinstance(o, Multiple) else Value(self.v + o.v)

    def __sub__(self, o):
        return o.plus(self, -1) if isinstance(o, Multiple) else Value(self.v - o.v)

    def __neg__(self):
        return Value(-self.v)


class Multiple(Value):
    """c x, rounded where it is used; a sum that it enters may take it unrounded (fused)."""

    fused = False

    def __init__(self, c, x):
        super().__init__(np.complex64(complex(c * x.v.real, c * x.v.imag)))
        self.c, self.x = c, x

    def plus(self, o, sign):
        if not self.fused:
            return Value(o.v + np.float32(sign) * self.v)
        c, x = np.float64(sign * self.c), np.complex128(self.x.v)  # the product is exact in double precision
        return Value(complex(np.float32(c * x.real + o.v.real), np.float32(c * x.imag + o.v.imag)))

    def __add__(self, o):
        return self.plus(Value(o), 1)

    def __sub__(self, o):
        return self.plus(Value(-o), 1)

    def __neg__(self):
        return Multiple(-self.c, self.x)


class Real:
    def __init__(self, c):
        self.c = np.float32(c)

    def __mul__(self, x):
        return Multiple(self.c, x)


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("name", ["numeric4", "cubic2", "products8"])
def test_schedule_rounds_as_the_code_does(name, fused, monkeypatch):
    """Whether or not the compiler fuses the code's real multiples into the sums they enter, the
    warp's schedule has the same values bit for bit."""
    monkeypatch.setattr(Multiple, "fused", fused)
    mod = system(name)
    info = gen_plugins.analyse(mod)
    tape = gen_plugins.Tape(info)
    code = "\n".join(gen_plugins.emit_rows(mod, info, "cuda")).replace("cx<T>", "cx")
    rng = np.random.default_rng(3)
    for _ in range(10):
        Y, q, dq = ([Value(complex(*rng.normal(size=2))) for _ in range(n)]
                    for n in (info["nv"] + 1, info["np"], info["np"]))
        env = dict(Y=Y, q=q, dq=dq, T=Real, mul_rn=lambda c, x: Value(Multiple(c.c, Value(x))),
                   cx=lambda c: Value(complex(c.c)))
        for var, e in re.findall(r"const cx (\w+) = (.*?);", code):
            env[var] = eval(e, {}, env)
        want = [Value(eval(e, {}, env)).v for e in re.findall(r"[MF]\[.*?\] = (.*?);", code)]
        reg = [v.v for v in Y + q + dq] + [np.complex64(c) for c in tape.consts]
        reg += [np.complex64(0)] * (tape.nregs - len(reg))
        words = tape.words()
        for s in range(0, len(words), tape.WIDTH):
            step = words[s:s + tape.WIDTH]
            written = {w & 1023 for w in step} - {tape.nregs - 1}
            assert not written & {r for w in step for r in ((w >> 10) & 1023, (w >> 20) & 1023)}
            new = [(w & 1023, reg[(w >> 10) & 1023], reg[(w >> 20) & 1023], w >> 30) for w in step]
            for d, a, b, kind in new:
                reg[d] = a * b if kind >> 1 else (a - b if kind & 1 else a + b)
        assert [-reg[w & 1023] if w >> 10 else reg[w & 1023] for w in tape.out_words()] == want


def write_sources(mod, tmp_path, monkeypatch, smem):
    """The system's generated header and the tracking kernels' sources without the calls that
    need a GPU, shared memory being declared as `smem`."""
    monkeypatch.setattr(gen_plugins, "load_plugins", lambda: [mod])
    (tmp_path / "frg_plugins_gen.cuh").write_text(gen_plugins.generate()[0])
    for src, dst in (("frg_track.cu", "track.inc"), ("frg_track_warp.cuh", "frg_track_warp.cuh")):
        text = open(os.path.join(CSRC, src)).read()
        text = re.sub(r"[\w:]+(<[^<>;]*>)?<<<.*?>>>\(.*?\);", ";", text)
        text = re.sub(r"return cuda(Occupancy|Func)[^;]*;", "return cudaSuccess;", text)
        assert "<<<" not in text
        (tmp_path / dst).write_text(text.replace("extern __shared__ __align__(16) unsigned char warp_smem[];", smem))


def kernels_agree(mod, tmp_path, monkeypatch):
    write_sources(mod, tmp_path, monkeypatch, "unsigned char* const warp_smem = emu::smem();")
    cfg = frg.plugin_config("conic2", start_dist=frg.START_NORMAL, max_steps=4)
    (tmp_path / "config").write_bytes(bytes(cfg))
    exe = tmp_path / "kernels"
    emu = os.path.join(HERE, "warp_emu")
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-ffp-contract=off", f"-DEMU_SYSTEM=Sys_{mod.NAME}",
                    f"-I{tmp_path}", f"-I{emu}", f"-I{CSRC}", os.path.join(emu, "plugin_kernels.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe), str(tmp_path / "config")], capture_output=True, text=True, timeout=300)
    print(r.stdout, r.stderr)
    return r.returncode == 0


@pytest.mark.parametrize("name", ["numeric4", "cubic2", "sparse12", "products8"])
def test_kernels_of_an_added_system_agree(name, tmp_path, monkeypatch):
    assert kernels_agree(system(name), tmp_path, monkeypatch)


def test_system_without_a_schedule_has_no_warp_kernel(tmp_path, monkeypatch):
    """Too many values for the schedule's registers: the kernels compile, and the host is told
    that no block of the warp kernel fits."""
    monkeypatch.setattr(gen_plugins.Tape, "REGS", 50)
    write_sources(system("cubic2"), tmp_path, monkeypatch, "unsigned char* const warp_smem = emu::smem();")
    (tmp_path / "main.cpp").write_text("""#include "track.inc"
int main() {
  frg::TrackArgs a{};
  a.cfg.system = 1;
  for (int mode = 0; mode < 3; ++mode) {
    int blocks = 7;
    if (frg_warp_occupancy(1, mode, &blocks) != cudaSuccess || blocks != 0) return 1;
    if (frg_launch_warp(mode, a, 1, nullptr) != cudaErrorInvalidValue) return 2;
  }
}
""")
    exe = str(tmp_path / "main")
    subprocess.run(["g++", "-std=c++17", "-w", f"-I{tmp_path}", f"-I{os.path.join(HERE, 'warp_emu')}", f"-I{CSRC}",
                    str(tmp_path / "main.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe]).returncode == 0


def test_static_shared_memory_of_a_large_system(tmp_path, monkeypatch):
    """At most the 48 KB that a kernel may have without asking, whatever the system's size."""
    write_sources(system("sparse12"), tmp_path, monkeypatch, "extern __shared__ __align__(16) unsigned char warp_smem[];")
    (tmp_path / "warp.cu").write_text(
        '#include "track.inc"\n'
        "template __global__ void frg::warp_kernel<frg::MODE_PLAIN, double, frg::Sys_sparse12>(frg::TrackArgs);\n")
    r = subprocess.run([frg_build.nvcc(), *frg_build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", f"-I{tmp_path}",
                        f"-I{CSRC}", "-Xcicc", "-O1", "-Xptxas", "-O1,-v", "-c", str(tmp_path / "warp.cu"), "-o",
                        str(tmp_path / "warp.o")], capture_output=True, text=True, check=True)
    assert "warp_kernel" in r.stderr
    assert all(int(n) <= 48 * 1024 for n in re.findall(r"(\d+) bytes smem", r.stderr))
