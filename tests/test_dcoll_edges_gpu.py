"""The device collection's batch paths at their edges, against the host collection (exact):
sizes around a warp and a block, a chain of roots each within tol of the one before (so that
nearly every root depends on another dependent one; 40 of them fit the resolver's list,
3,000 do not), repeats of one root, and a collection that fills up."""
import numpy as np
import pytest

import finite_root_generation_gb300 as frg
from finite_root_generation_gb300 import build as frg_build

pytestmark = pytest.mark.gpu

TOL = 1e-6


def _merge(roots, codes, capacity):
    torch = pytest.importorskip("torch")
    frg_build.build()
    dc = frg.DeviceCollection(capacity, TOL)
    d_codes = torch.from_numpy(codes.copy()).cuda()
    dc.merge(torch.from_numpy(np.ascontiguousarray(roots).view(np.float64)).cuda(), d_codes)
    return dc, d_codes.cpu().numpy()


def _rows(r):
    v = np.ascontiguousarray(r).view(np.float64).reshape(len(r), 42)
    return v[np.lexsort(v.T[::-1])]


@pytest.mark.parametrize("kind,n", [("random", 1), ("random", 31), ("random", 33), ("random", 257), ("chain", 40),
                                    ("chain", 3000), ("same", 1000)])
def test_batch_edges(kind, n):
    rng = np.random.default_rng(n)
    roots = rng.normal(size=(n, 21)) + 1j * rng.normal(size=(n, 21))
    codes = np.zeros(n, np.int32)
    if kind == "random":
        codes[::7] = 3
    elif kind == "chain":
        roots = roots[:1] + 0.9e-6 * np.arange(n)[:, None]
    else:
        roots = np.repeat(roots[:1], n, axis=0)
    host = frg.Collection(TOL)
    want = host.merge(roots, codes)
    dc, got = _merge(roots, codes, n)
    assert np.array_equal(got, want)
    got_roots, _ = dc.roots()
    assert np.array_equal(_rows(got_roots), _rows(host.roots()))
    dc.close()


def test_full_collection_reports_overflow():
    rng = np.random.default_rng(2)
    roots = rng.normal(size=(100, 21)) + 1j * rng.normal(size=(100, 21))
    dc, got = _merge(roots, np.zeros(100, np.int32), 70)
    assert np.all(got == 0)
    with pytest.raises(frg.FrgError):
        dc.size()
    dc.close()
