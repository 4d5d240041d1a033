"""As the stale-memory test, where Z = B V runs on lists and tiles (above 1024
samples), with sample counts that leave padding: a solve gives the same result, bit
for bit, before and after solves of huge and of non-finite values have been through
the pool's memory."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GAMMA = {4: 1.0, 7: 20.0}  # supports of some twenty: at most 31 make a sparse step


@pytest.mark.parametrize("m", [1026, 1055])
@pytest.mark.parametrize("k", [40, 140])
@pytest.mark.parametrize("formulation", [0, 1, 4, 7])
def test_tiled_steps_do_not_depend_on_the_pools_contents(solver, po, formulation, k, m):
    am = importlib.import_module("24am_b200")
    B = po.low_rank_data(m, 1003, 6, 24, seed=3, dtype=np.float32)

    def solve(data):
        M = solver.matrix(data)
        x, f, st = M.solve(am.OptimizationSettings(
            formulation=formulation, constraintParameter=9,
            penaltyParameter=GAMMA.get(formulation, 0.0), tolerance=0.0, maximumIterations=6,
            totalStartingPoints=k, batchSize=k, startMode=am.START_DEVICE_UNIFORM))
        M.close()
        return x, f, st.explained_variance

    first = solve(B)
    assert 0 < np.count_nonzero(first[0]) <= 1003 // 32
    bad = B.copy()
    bad[:, ::7] = np.inf
    bad[0, :] = np.nan
    for poison in ((B * 1e18).astype(np.float32), bad):
        solve(poison)
        for a, c in zip(first, solve(B)):
            assert np.array_equal(np.asarray(a), np.asarray(c), equal_nan=True)
