"""Products of sparse-resident matrices around their tiles: start counts on
both sides of 32 and 128 (a lane takes four starts, a tile 128), rows and columns
just under, at and beyond 1024 entries (where sums run in segments), and steps
whose supports leave most rows of V empty.  Three steps from given starts against
the FP64 oracle's on the centred dense matrix: the best objective (FP32 sums of
some thousand terms: within 1e-5) and the variance of the returned loading."""
import importlib

import numpy as np
import pytest
import scipy.sparse as sp

import fast_oracle as fo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 31, 33, 127, 128, 130, 257])
@pytest.mark.parametrize("formulation", [0, 1])
def test_start_counts_around_the_tiles(solver, po, formulation, k):
    am = importlib.import_module("24am_b200")
    m, n = 1500, 1300
    rng = np.random.default_rng(k)
    A = np.where(rng.random((m, n)) < 0.01, rng.standard_normal((m, n)), 0.0)
    for c, filled in ((3, 1023), (700, 1024), (701, 1025), (1299, 1400)):
        rows = rng.choice(m, filled, replace=False)
        A[:, c] = 0.0
        A[rows, c] = rng.standard_normal(filled) + 0.5 * (c % 3)
    A[17, :] = np.where(rng.random(n) < 0.9, rng.standard_normal(n), 0.0)
    A = A.astype(np.float32)
    mu = A.mean(axis=0, dtype=np.float64).astype(np.float32)
    C = A.astype(np.float64) - mu.astype(np.float64)
    V0 = po.uniform_starts(n, k, seed=9, dtype=np.float32)
    M = am.Matrix.from_csc(solver, sp.csc_matrix(A), None, None, None, None, means=mu,
                           keep_sparse=True)
    x, f, stats = M.solve(am.OptimizationSettings(
        formulation=formulation, constraintParameter=6, tolerance=0.0, maximumIterations=3,
        totalStartingPoints=k, batchSize=k, startMode=am.START_INJECTED), start_points=V0)
    M.close()
    V, val = V0.astype(np.float64), np.zeros(k)
    for _ in range(3):
        r = fo.iteration(C, V, formulation, 6, 0.0, val)
        V, val = r.V, r.val
    best = int(np.argmax(val))
    assert abs(f - val[best]) <= 1e-5 * val[best]
    want = np.linalg.norm(C @ V[:, best]) ** 2
    assert abs(stats.explained_variance - want) <= 1e-4 * want
    assert abs(np.linalg.norm(C @ x.astype(np.float64)) ** 2 - want) <= 1e-4 * want
