"""The top-s select on columns given entry by entry: with one sample (m = 1)
V = B^T Z is B's row times a scalar, so any column can be put before the
select.  Sizes around the sample's (2048 entries, 4096 from columns longer than
65536), s from 1 past the candidates' capacity (2048), and columns with ties,
a few non-zeros or one value.  Two steps: the
first finds its candidates from a sample, the second from the hint.

Expected: the entries with |b| at or above the s-th largest (ties kept, zeros
never), b / ||b||_2 over them.  Tolerance: a product is within 2^-21 of exact
(split operands 2^-22, one rounding), the norm too, and the scaling rounds
twice, so every loading is within 1e-6 of the largest."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _column(kind, n, rng):
    if kind == "grid":  # distinct values differ by more than the products' rounding
        return np.round(rng.standard_normal(n) * 4096) / 4096
    if kind == "ties":
        return rng.integers(-20, 21, n) / 4.0
    if kind == "few":
        b = np.zeros(n)
        at = rng.choice(n, min(n, 20), replace=False)
        b[at] = rng.integers(1, 50, at.size)
        return b
    return np.full(n, -1.5)  # "constant"


@pytest.mark.parametrize("k", [64, 130])
@pytest.mark.parametrize("kind", ["grid", "ties", "few", "constant"])
@pytest.mark.parametrize("n", [1, 5, 33, 2047, 2052, 4100, 65536, 65541])
def test_top_s_of_given_columns(solver, n, kind, k):
    am = importlib.import_module("24am_b200")
    rng = np.random.default_rng(n + len(kind))
    b = _column(kind, n, rng).astype(np.float32)
    if not np.any(b):
        b[0] = 1.0
    V0 = rng.uniform(0.5, 1.0, (n, k)).astype(np.float32) * np.where(b < 0, -1, 1)[:, None]
    V0 = np.asfortranarray(V0.astype(np.float32))  # b . v > 0 without cancellation
    M = solver.matrix(b[None, :])
    a = np.abs(b.astype(np.float64))
    for s in (1, 16, 700, 2048, 3000):
        if s > n:
            continue
        batch = M.batch(am.OptimizationSettings(constraintParameter=s, tolerance=0.0), k)
        batch.load(V0)
        level = np.sort(a)[::-1][s - 1]
        want = np.where((a >= level) & (a > 0), b.astype(np.float64), 0.0)
        want /= np.linalg.norm(want)
        for step in range(2):
            batch.iterate(step, 1)
            V = batch.read()[0].astype(np.float64)
            where = f"s = {s}, step {step + 1}"
            assert np.array_equal(V != 0, np.repeat((want != 0)[:, None], k, 1)), where
            assert np.abs(V - want[:, None]).max() <= 1e-6 * np.abs(want).max(), where
        batch.close()
    M.close()
