"""Buffers come from a pool and are not all cleared: a solve whose column length
is not a multiple of 32 (so that planes have padding) gives the same result, bit
for bit, before and after solves of huge and of non-finite values have been
through the pool's memory."""
import importlib

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

GAMMA = {4: 2.0, 5: 2000.0, 6: 1.0, 7: 40.0}


@pytest.mark.parametrize("kind", ["batch", "group", "sparse"])
@pytest.mark.parametrize("k", [40, 140])
@pytest.mark.parametrize("formulation", [0, 1, 2, 3, 4, 7])
def test_results_do_not_depend_on_the_pools_contents(solver, po, formulation, k, kind):
    am = importlib.import_module("24am_b200")
    m, n = 77, 1003
    B = po.low_rank_data(m, n, 6, 24, seed=3, dtype=np.float32)

    def settings(**kw):
        a = dict(formulation=formulation, constraintParameter=9,
                 penaltyParameter=GAMMA.get(formulation, 0.0), tolerance=0.0, maximumIterations=6,
                 totalStartingPoints=k, batchSize=k, startMode=am.START_DEVICE_UNIFORM)
        a.update(kw)
        return am.OptimizationSettings(**a)

    def solve(data):
        if kind == "sparse":
            M = am.Matrix.from_csc(solver, sp.csc_matrix(data), None, None, None, None,
                                   keep_sparse=True)
        else:
            M = solver.matrix(data)
        if kind == "group":
            with am.Group(solver, capacity=1) as g:
                pid = g.add(M, settings())
                g.run()
                x, st = g.result(pid)
        else:
            x, _, st = M.solve(settings())
        M.close()
        return x, st.fval, st.explained_variance

    first = solve(B)
    huge = (B * 1e18).astype(np.float32)
    bad = B.copy()
    bad[:, ::7] = np.inf
    bad[0, :] = np.nan
    for poison in (huge, bad):
        solve(poison)
        again = solve(B)
        for a, c in zip(first, again):
            assert np.array_equal(np.asarray(a), np.asarray(c), equal_nan=True)
