"""How a launch spreads its paths over the GPU: the team kernels put one to four paths in a
block; a plug-in's launch tracks a path per warp up to 16 paths per SM sub-partition and
a path per thread beyond, whose last paths go on a warp each. So the same path runs beside
different neighbours, and in different kernels, in different calls. A path depends on its random
stream alone: the first n paths of a call must equal the call of n paths bit for bit, at
the sizes where the spreading changes (one path, a block not full, one path per SM, every
block full, every sub-partition taken), and its first paths match the oracle (codes on
>= 97 % of them, roots within 1e-8 relative where both succeed on >= 99 %)."""
import numpy as np
import pytest

import finite_root_generation_gb300 as frg
from finite_root_generation_gb300 import build as frg_build
from finite_root_generation_gb300.tasks import REFERENCE_GAMMA, REFERENCE_TARGET

pytestmark = pytest.mark.gpu

SIZES = [1, 3, 5, 153, 305, 607]
FULL = 700


@pytest.mark.parametrize("precision", [frg.PREC_FP64, frg.PREC_MIXED], ids=["fp64", "mixed"])
def test_team_spread(precision, oracle):
    frg_build.build()
    cfg = frg.default_config() if precision == frg.PREC_FP64 else frg.chosen_config()
    with frg.Tracker(cfg) as t:
        full = t.track(REFERENCE_TARGET, [FULL], 41, want_yfinal=True, want_resid=True)
        for n in SIZES:
            part = t.track(REFERENCE_TARGET, [n], 41, want_yfinal=True, want_resid=True)
            assert np.array_equal(part.codes, full.codes[:n]), n
            assert np.array_equal(part.roots, full.roots[:n], equal_nan=True), n
            assert np.array_equal(part.yfinal, full.yfinal[:n], equal_nan=True), n
            assert np.array_equal(part.resid, full.resid[:n], equal_nan=True), n
    m = 128
    roots, codes, _, _ = oracle.homotopy_batch(REFERENCE_TARGET, REFERENCE_GAMMA, 41, np.arange(m))
    assert (full.codes[:m] == codes).mean() >= 0.97
    both = (codes == 0) & (full.codes[:m] == 0)
    rel = np.max(np.abs(full.roots[:m][both] - roots[both]), axis=1) / np.max(np.abs(roots[both]), axis=1)
    assert (rel < 1e-8).mean() >= 0.99


@pytest.mark.parametrize("precision", [frg.PREC_FP64, frg.PREC_MIXED], ids=["fp64", "mixed"])
def test_thread_spread(precision):
    frg_build.build()
    rng = np.random.default_rng(7)
    task = rng.normal(size=12) + 1j * rng.normal(size=12)
    cfg = frg.plugin_config("conic2", precision=precision, start_dist=frg.START_NORMAL,
                            gamma_mode=frg.GAMMA_RANDOM, inf_tol=1e-8)
    with frg.Tracker(cfg) as t:
        full = t.track(task, [20000], 43, want_resid=True)
        for n in (1, 33, 607, 609, 9728, 9729, 19455, 19457):
            part = t.track(task, [n], 43, want_resid=True)
            assert np.array_equal(part.codes, full.codes[:n]), n
            assert np.array_equal(part.roots, full.roots[:n], equal_nan=True), n
            assert np.array_equal(part.resid, full.resid[:n], equal_nan=True), n
