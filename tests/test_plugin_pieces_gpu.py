"""A plug-in call of more paths than a piece holds: its paths are those of smaller calls, and
its work buffers do not grow with it."""
import numpy as np
import pytest

import finite_root_generation_gb300 as frg
from finite_root_generation_gb300 import build as frg_build

pytestmark = pytest.mark.gpu
PIECE = 1 << 24


@pytest.mark.parametrize("precision", [frg.PREC_FP64, frg.PREC_MIXED], ids=["fp64", "mixed"])
def test_call_of_two_pieces(precision):
    torch = pytest.importorskip("torch")
    frg_build.build()
    rng = np.random.default_rng(5)
    tasks = rng.normal(size=(3, 12)) + 1j * rng.normal(size=(3, 12))
    counts = [PIECE - 500, 1500, PIECE // 2]
    n = sum(counts)
    cfg = dict(precision=precision, start_dist=frg.START_NORMAL, gamma_mode=frg.GAMMA_RANDOM)

    def buffers(m):
        return [torch.zeros(m * k, dtype=d, device="cuda") for k, d in ((4, torch.float64), (1, torch.int32),
                                                                       (8, torch.float64), (1, torch.float64))]

    full = buffers(n)
    with frg.Tracker(frg.plugin_config("conic2", **cfg)) as t:
        t.track_into(tasks, [20000, 0, 0], 11, *buffers(20000))  # modules and the kernels' stacks are in place
        torch.cuda.empty_cache()
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        stats = t.track_into(tasks, counts, 11, *full)
        held = free - torch.cuda.mem_get_info()[0]
    assert sum(stats["codes"]) == n
    assert stats["stage_ms"][1] > 0
    # start values, endpoints and the mixed call's records of one piece
    assert held < 1.1 * PIECE * (288 + (1400 if precision == frg.PREC_MIXED else 0)) + (64 << 20)
    # the first paths, those around the pieces' boundary (task 1 and the first of task 2), the last
    for first, ppt in ((0, [700, 0, 0]), (counts[0], [0, 1500, 900]), (n - 800, [0, 0, 800])):
        m = sum(ppt)
        part = buffers(m)
        with frg.Tracker(frg.plugin_config("conic2", path_offset=first, **cfg)) as t:
            t.track_into(tasks, ppt, 11, *part)
        for whole, some in zip(full, part):
            k = some.numel() // m
            a, b = whole[k * first:k * (first + m)].cpu().numpy(), some.cpu().numpy()
            assert np.array_equal(a, b, equal_nan=True)
