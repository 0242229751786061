"""Plug-in systems added the documented way (a module in systems/, the generator, a build) on
the GPU: a path's result does not depend on its call's size, which selects the kernel that
tracks it. A call above the sizes that take a warp per path runs a thread per path, and a
warp for each of its last paths; its first paths must equal a smaller call's, bit for bit."""
import os
import shutil
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
PKG = "finite_root_generation_gb300"
SYSTEMS = ["numeric4", "cubic2", "sparse12"]

# The generator, with too few registers for the five unknowns of burmester5
GENERATE = """
import sys
from finite_root_generation_gb300.gen import gen_plugins as g
init = g.Tape.__init__
def few(self, info):
    self.REGS = 100 if info["nv"] == 5 else 1024
    init(self, info)
g.Tape.__init__ = few
g.main()
"""

RUN = """
import sys
import numpy as np
import finite_root_generation_gb300 as frg
info = next(s for s in frg.list_systems() if s.name == sys.argv[1])
rng = np.random.default_rng(5)
tasks = rng.normal(size=(2, info.np)) + 1j * rng.normal(size=(2, info.np))
for precision in (frg.PREC_FP64, frg.PREC_MIXED):
    cfg = frg.plugin_config(info.name, precision=precision, start_dist=frg.START_NORMAL, gamma_mode=frg.GAMMA_RANDOM)
    with frg.Tracker(cfg) as t:
        full = t.track(tasks, [6000, 4000], 7, want_yfinal=True, want_resid=True)
        part = t.track(tasks, [6000, 70], 7, want_yfinal=True, want_resid=True)
    n = len(part.codes)
    ok = full.codes == 0
    print(info.name, precision, np.bincount(full.codes, minlength=8), "residual", np.max(full.resid[ok], initial=0))
    assert ok.mean() > 0.2 and np.mean(full.resid[ok] <= 1e-10) > 0.99
    assert np.array_equal(part.codes, full.codes[:n])
    for k in ("roots", "yfinal", "resid"):
        assert np.array_equal(getattr(part, k), getattr(full, k)[:n], equal_nan=True), k
"""


@pytest.fixture(scope="module")
def added(tmp_path_factory):
    root = tmp_path_factory.mktemp("added")
    shutil.copytree(os.path.join(ROOT, PKG), root / PKG, ignore=shutil.ignore_patterns("*.so", "_build", "__pycache__"))
    shutil.copytree(os.path.join(ROOT, "include"), root / "include")
    (root / "oracle").mkdir()
    systems = root / PKG / "systems"
    for name in SYSTEMS:
        shutil.copy(os.path.join(HERE, "added_systems", name + ".py"), systems)
    init = systems / "__init__.py"
    init.write_text(init.read_text().replace('"burmester5"]', '"burmester5", ' + str(SYSTEMS)[1:]))
    for step in (["-c", GENERATE], [str(root / PKG / "build.py")]):
        subprocess.run([sys.executable, *step], cwd=root, env=dict(os.environ, PYTHONPATH=str(root)), check=True,
                       timeout=900)
    return root


@pytest.mark.parametrize("name", SYSTEMS)
def test_added_system_does_not_depend_on_the_call_size(added, name):
    env = dict(os.environ, PYTHONPATH=str(added))
    r = subprocess.run([sys.executable, "-c", RUN, name], cwd=added, env=env, capture_output=True, text=True, timeout=600)
    print(r.stdout, r.stderr)
    assert r.returncode == 0, r.stderr


DUMP = """
import sys
import numpy as np
import finite_root_generation_gb300 as frg
from finite_root_generation_gb300.systems import burmester5
task = burmester5.physical_task(np.random.default_rng(5))
out = {}
for precision in (frg.PREC_FP64, frg.PREC_MIXED):
    with frg.Tracker(frg.plugin_config("burmester5", precision=precision, start_dist=frg.START_NORMAL)) as t:
        for n in (300, 9800):
            r = t.track(task, [n], 3, want_yfinal=True, want_resid=True)
            out.update({f"{k}_{precision}_{n}": getattr(r, k) for k in ("codes", "roots", "yfinal", "resid")})
np.savez(sys.argv[1], **out)
"""


def test_system_without_warp_kernel_has_the_same_results(added, tmp_path):
    """A system whose schedule needs too many registers is tracked by a thread per path alone, as
    burmester5 is in the fixture's build; its results equal the usual build's."""
    out = []
    for k, root in enumerate((str(added), ROOT)):
        path = str(tmp_path / f"{k}.npz")
        subprocess.run([sys.executable, "-c", DUMP, path], cwd=root, env=dict(os.environ, PYTHONPATH=root), check=True,
                       timeout=600)
        out.append(dict(np.load(path)))
    assert "TAPE_STEPS = 0;" in (added / PKG / "csrc" / "frg_plugins_gen.cuh").read_text()
    for k, v in out[0].items():
        assert np.array_equal(v, out[1][k], equal_nan=True), k
