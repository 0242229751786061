"""burmester5 above the sizes that take a warp per path: a thread tracks a path, and a launch's
last paths go on a warp each. Two tasks of unequal counts, both precisions, endpoints
included: the first paths must equal those of a smaller call, a warp per path, bit for bit."""
import numpy as np
import pytest

import finite_root_generation_gb300 as frg
from finite_root_generation_gb300 import build as frg_build
from finite_root_generation_gb300.systems import burmester5

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(5000, 4900), (9000, 11000)])
@pytest.mark.parametrize("precision", [frg.PREC_FP64, frg.PREC_MIXED], ids=["fp64", "mixed"])
def test_thread_kernel_and_last_paths(precision, counts):
    frg_build.build()
    tasks = np.stack([burmester5.physical_task(np.random.default_rng(s)) for s in (5, 6)])
    cfg = frg.plugin_config("burmester5", precision=precision, start_dist=frg.START_NORMAL,
                            gamma_mode=frg.GAMMA_RANDOM, inf_tol=1e-8)
    with frg.Tracker(cfg) as t:
        full = t.track(tasks, counts, 29, want_yfinal=True, want_resid=True)
        part = t.track(tasks, [counts[0], 600], 29, want_yfinal=True, want_resid=True)
    n = counts[0] + 600
    assert n <= 9728 < sum(counts)
    assert np.array_equal(part.codes, full.codes[:n])
    for k in ("roots", "yfinal", "resid"):
        assert np.array_equal(getattr(part, k), getattr(full, k)[:n], equal_nan=True), k
