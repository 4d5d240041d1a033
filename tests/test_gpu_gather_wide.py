"""The sparse Z = B V on both sides of 1024 samples (one block per start up to
there, lists and tiles of 128 samples above), for start counts around a block's
eight, on one-CTA and pair tiles: each of three steps against the FP64 oracle's
step from the GPU's own loadings, per well-conditioned start (supports; loadings
within 1e-5 of the largest: FP32 sums of a few dozen products for z and of m
split-operand ones for V), and the grouped step bit for bit against the batch."""
import importlib

import numpy as np
import pytest

import fast_oracle as fo

pytestmark = pytest.mark.gpu

GAMMA = {4: 0.3}


@pytest.mark.parametrize("m", [100, 1024, 1025, 1152, 2049])
@pytest.mark.parametrize("k", [1, 9, 130])
@pytest.mark.parametrize("formulation", [0, 1, 4])
def test_sparse_steps_by_samples(solver, po, formulation, k, m):
    am = importlib.import_module("24am_b200")
    n, s = 2100, 12
    B = po.low_rank_data(m, n, 6, 24, seed=m + k, dtype=np.float32)
    B64 = B.astype(np.float64)
    V0 = po.uniform_starts(n, k, seed=5, dtype=np.float32)
    g = GAMMA.get(formulation, 0.0)
    st = am.OptimizationSettings(formulation=formulation, constraintParameter=s, penaltyParameter=g,
                                 tolerance=0.0, maximumIterations=3, totalStartingPoints=k,
                                 batchSize=k, startMode=am.START_INJECTED)
    M = solver.matrix(B)
    b = M.batch(st, k)
    b.load(V0)
    prev, val = V0.astype(np.float64), np.zeros(k)
    sparse = 0
    for it in range(3):
        sparse += np.count_nonzero(prev, axis=0).max() <= n // 32
        b.iterate(it, 1)
        V, v, _, _ = b.read()
        r = fo.iteration(B64, prev, formulation, s, g, val)
        keep = np.flatnonzero(~r.ill & np.isfinite(r.val) & (r.val > 0))
        for j in keep:
            assert np.array_equal(V[:, j] != 0, r.V[:, j] != 0), (it, j)
            scale = np.abs(r.V[:, j]).max()
            assert np.abs(V[:, j] - r.V[:, j]).max() <= 1e-5 * scale, (it, j)
        prev, val = V.astype(np.float64), v.astype(np.float64)
    assert sparse >= 1, "no step ran the gather"
    if k > 128:
        grp = am.Group(solver, capacity=1)
        pid = grp.add(M, st, start_points=V0)
        grp.run()
        for a, c in zip(grp.read(pid), b.read()):
            assert np.array_equal(a, c, equal_nan=True)
        grp.close()
    b.close()
    M.close()
