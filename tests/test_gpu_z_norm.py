"""The norm of z = B v on sparse steps, where the samples are padded to 32 (and
taken four at a time): with loadings past FP32 the padding's products are 0 x inf,
which are no part of ||z||.  B is positive and so small that V = B^T Z lies
below FP32's normal range: the first step's select divides by a norm under
2^-128, whose reciprocal is infinite, so the second (sparse) step has infinite
loadings and every z_i, and the objective, is +inf, as on a dense step."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [33, 64, 99, 1024, 1026, 1056, 1499])
def test_infinite_loadings_give_an_infinite_norm(solver, m):
    am = importlib.import_module("24am_b200")
    n, k, s = 1500, 130, 8  # up to n / 32 = 46 non-zeros the step is sparse
    rng = np.random.default_rng(m)
    # V is about 85 m scale^2: 5e-41, some 35000 units of its last place
    scale = np.sqrt(5e-41 / (85 * m))
    M = solver.matrix((rng.uniform(1.0, 2.0, (m, n)) * scale).astype(np.float32))
    V0 = rng.uniform(0.5, 1.0, (n, k))
    V0 = np.asfortranarray((V0 / np.linalg.norm(V0, axis=0)).astype(np.float32))
    b = M.batch(am.OptimizationSettings(constraintParameter=s, tolerance=0.0), k)
    b.load(V0)
    b.iterate(0, 1)
    V, val, _, _ = b.read()
    on = V != 0
    assert np.all(np.isfinite(val)) and np.all(np.isposinf(V[on]))
    assert on.any(axis=0).all() and on.sum(axis=0).max() <= n // 32
    b.iterate(1, 1)
    assert np.all(np.isposinf(b.read()[1]))
    b.close()
    M.close()
