"""Plug-in systems other than the shipped ones, generated from a module as a user adds one,
on the CPU: the two tracking kernels of a plug-in (a path per thread, a path per warp) are
the same computation, so a path must come out of both alike, whatever kernel its call's size
selects. The kernels' own source runs here (tests/warp_emu): each path starts, takes a few
steps and ends on the step limit (FP64) or is still in hand at it (FP32 stage)."""
import os
import re
import subprocess
import types

import pytest

import finite_root_generation_gb300 as frg

sp = pytest.importorskip("sympy")

from finite_root_generation_gb300.gen import gen_plugins  # noqa: E402

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(gen_plugins.__file__), "..", "csrc")


def numeric_quadrics():
    """Four quadrics in four unknowns with coefficients that are numbers, 65 of them different."""
    x = sp.symbols("x0:4")
    c = sp.symbols("c0:4")
    mono = [x[i] * x[j] for i in range(4) for j in range(i, 4)] + list(x)
    eqs = [sum(sp.Rational((m + 2) ** (k + 2) % 97, 32) * t for m, t in enumerate(mono)) + c[k] for k in range(4)]
    return types.SimpleNamespace(NAME="numeric4", UNKNOWNS=list(x), PARAMS=list(c), EQUATIONS=eqs, SOLVED=list(c))


def kernels_agree(mod, tmp_path, monkeypatch):
    monkeypatch.setattr(gen_plugins, "load_plugins", lambda: [mod])
    with open(tmp_path / "frg_plugins_gen.cuh", "w") as f:
        f.write(gen_plugins.generate()[0])
    track = open(os.path.join(CSRC, "frg_track.cu")).read()
    track = re.sub(r"[\w:]+(<[^<>;]*>)?<<<.*?>>>\(.*?\);", ";", track)
    assert "<<<" not in track
    (tmp_path / "track.inc").write_text(track)
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


@pytest.mark.parametrize("system", [numeric_quadrics], ids=lambda s: s.__name__)
def test_kernels_of_an_added_system_agree(system, tmp_path, monkeypatch):
    assert kernels_agree(system(), tmp_path, monkeypatch)
