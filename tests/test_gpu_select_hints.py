"""Selects whose support takes a large share of the candidates that a block sorts
(2048 of the top-s select, 4096 of the L1 ball's): once the supports settle, a
step finds its candidates from the last step's hint and never reads the whole
column, so it takes a small part of the first step's time (a tenth and less;
the test asks for a third).  A bound that lies too low for the capacity sends
every step back to the column."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("formulation,s", [(0, 900), (0, 1700), (2, 1600), (2, 2048)])
def test_settled_supports_are_found_from_the_hint(solver, formulation, s):
    am = importlib.import_module("24am_b200")
    m, n, k = 200, 200000, 128
    rng = np.random.default_rng(1)
    B = rng.standard_normal((m, n), dtype=np.float32)
    loud = rng.random(n, dtype=np.float32) < 0.02  # some 4000 features carry four components
    W = rng.standard_normal((4, n), dtype=np.float32) * loud
    B += 2 * rng.standard_normal((m, 4), dtype=np.float32) @ W
    V0 = np.asfortranarray(rng.uniform(-1, 1, (n, k)).astype(np.float32))
    M = solver.matrix(B)
    b = M.batch(am.OptimizationSettings(formulation=formulation, constraintParameter=s,
                                        tolerance=0.0, l1Mode=am.L1_EXACT), k)
    first, settled = [], []
    for rep in range(3):
        b.load(V0)
        t = [dict(b.step_timed(it))["select"] for it in range(8)]
        first.append(t[0])
        settled.append(min(t[3:]))
    b.close()
    M.close()
    assert np.median(settled) < np.median(first) / 3, (first, settled)
