"""The L1-ball selects beyond and around their sorted candidate sets (4096 entries).
Deep stops: supports above 4096, so that the walk over ranks is certain to run,
on columns that are walked whole (up to 8192 entries behind the candidates) and
longer ones, for the reference's scan and the exact projection; steps against the
FP64 oracle's from the GPU's own loadings.  Given columns (exact projection): with one sample (m = 1) V = B^T Z is
B's row times a scalar, here with ties and few non-zeros, at lengths around the
sample's (2048 and 4096 entries) and 65536.  Starts that the oracle calls
ill-conditioned are left out; bounds as for the other wide supports."""
import importlib

import numpy as np
import pytest

import fast_oracle as fo

pytestmark = pytest.mark.gpu


def _settings(s, k, exact):
    am = importlib.import_module("24am_b200")
    return am.OptimizationSettings(formulation=2, constraintParameter=s, tolerance=0.0,
                                   maximumIterations=10, totalStartingPoints=k, batchSize=k,
                                   l1Mode=am.L1_EXACT if exact else am.L1_REFERENCE_SCAN)


def _check(V, val, r, what):
    keep = np.flatnonzero(~r.ill & np.isfinite(r.val))
    for j in keep:
        assert np.array_equal(V[:, j] != 0, r.V[:, j] != 0), (what, j)
        assert np.abs(V[:, j] - r.V[:, j]).max() <= 1e-4 * np.abs(r.V[:, j]).max(), (what, j)
        assert abs(val[j] - r.val[j]) <= 1e-5 * abs(r.val[j]), (what, j)
    return keep


@pytest.mark.parametrize("exact", [False, True], ids=["scan", "exact"])
@pytest.mark.parametrize("n,s", [(8000, 2500), (9000, 2500), (30000, 3000), (30000, 4096), (70000, 4096)])
def test_supports_beyond_the_candidates(solver, po, n, s, exact):
    m, k = 100, 32
    B = po.low_rank_data(m, n, 6, 400, seed=n + s, dtype=np.float32)
    V0 = po.uniform_starts(n, k, seed=62, dtype=np.float32)
    M = solver.matrix(B)
    b = M.batch(_settings(s, k, exact), k)
    b.load(V0)
    prev, val, widest = V0.astype(np.float64), np.zeros(k), 0
    for it in range(3):
        b.iterate(it, 1)
        V, v, _, _ = b.read()
        r = fo.iteration(B.astype(np.float64), prev, 2, s, 0.0, val, l1_exact=exact)
        if not exact:
            r.ill |= np.count_nonzero(V, axis=0) == 1  # the GPU's first-rank stops
        keep = _check(V, v, r, f"step {it + 1}")
        widest = max(widest, int(np.count_nonzero(r.V[:, keep], axis=0).max(initial=0)))
        prev, val = V.astype(np.float64), v.astype(np.float64)
    b.close()
    M.close()
    assert widest > 4096


@pytest.mark.parametrize("kind", ["grid", "ties", "few"])
@pytest.mark.parametrize("n", [33, 2047, 2052, 4100, 65541])
def test_given_columns(solver, n, kind):
    k = 4
    rng = np.random.default_rng(n + len(kind))
    if kind == "grid":  # distinct values differ by more than the products' rounding
        col = np.round(rng.standard_normal(n) * 4096) / 4096
    elif kind == "ties":
        col = rng.integers(-20, 21, n) / 4.0
    else:
        col = np.zeros(n)
        at = rng.choice(n, 20, replace=False)
        col[at] = rng.integers(1, 50, 20)
    V0 = rng.uniform(0.5, 1.0, (n, k)).astype(np.float32) * np.where(col < 0, -1, 1)[:, None]
    V0 = np.asfortranarray(V0.astype(np.float32))  # col . v > 0 without cancellation
    M = solver.matrix(col.astype(np.float32)[None, :])
    for s in (2, 12, 300, 1500):
        if s >= n:
            continue
        b = M.batch(_settings(s, k, True), k)
        b.load(V0)
        prev, val = V0.astype(np.float64), np.zeros(k)
        for it in range(2):
            b.iterate(it, 1)
            V, v, _, _ = b.read()
            r = fo.iteration(col[None, :], prev, 2, s, 0.0, val, l1_exact=True)
            _check(V, v, r, f"s = {s}, step {it + 1}")
            prev, val = V.astype(np.float64), v.astype(np.float64)
        b.close()
    M.close()
