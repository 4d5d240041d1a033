"""The pass over Z of a sparse-resident step (norms, signs, scaling and the
centring's sums on the row-major Z) around its blocks: sample counts from one to
several rows per warp, start counts on both sides of 32 and 128, centred by columns
and rows, all formulations with one or two passes.  One step from given starts
against the FP64 oracle, every start's objective, within 4e-6 of what the products'
terms add up to without cancelling (FP32 sums of at most some 500 terms: 2^-24
sqrt(500) = 1.3e-6; the penalties sit at the median loading, and the objective is
continuous in them).  With L1 variance a start whose Z holds a value too near zero
to have a certain sign is left out."""
import ctypes as C
import importlib

import numpy as np
import pytest
import scipy.sparse as sp

import fast_oracle as fo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k", [(1, 3), (31, 33), (33, 1), (257, 128), (5000, 130)])
@pytest.mark.parametrize("formulation", [0, 1, 4, 5, 6, 7])
def test_pass_over_z(solver, po, formulation, m, k):
    am = importlib.import_module("24am_b200")
    n = 300
    rng = np.random.default_rng(m + k)
    A = np.where(rng.random((m, n)) < 0.1, rng.standard_normal((m, n)), 0.0).astype(np.float32)
    mu = (0.1 * rng.standard_normal(n)).astype(np.float32)
    r = (0.1 * rng.standard_normal(m)).astype(np.float32)
    B = A.astype(np.float64) - mu.astype(np.float64) - r.astype(np.float64)[:, None]
    V0 = po.uniform_starts(n, k, seed=5, dtype=np.float32)
    Z = B @ V0.astype(np.float64)
    Za = np.abs(B) @ np.abs(V0.astype(np.float64))
    l1var, penalized = formulation % 2 == 1, formulation >= 4
    sure = np.abs(Z).min(axis=0) > 1e-5 * np.abs(Z).max(axis=0) if l1var else np.ones(k, bool)
    gamma, terms = 0.0, (Za.sum(axis=0) if l1var else np.linalg.norm(Za, axis=0))
    if penalized:
        raw = np.abs(B.T @ (np.sign(Z) if l1var else Z / np.linalg.norm(Z, axis=0)))
        a = np.abs(B).T @ (np.ones_like(Z) if l1var else Za / np.linalg.norm(Z, axis=0))
        terms = 2 * (a * a).sum(axis=0) if formulation in (4, 5) else np.linalg.norm(a, axis=0)
        gamma = float(np.float32(np.median(raw) ** (2 if formulation in (4, 5) else 1)))
    M = am.Matrix.from_csc(solver, sp.csc_matrix(A), None, None, None, None, means=mu,
                           row_means=r, keep_sparse=True)
    cs = am.OptimizationSettings(
        formulation=formulation, constraintParameter=6, penaltyParameter=gamma, tolerance=0.0,
        maximumIterations=1, totalStartingPoints=k, batchSize=k, storeIterationsForAllPoints=True,
        startMode=am.START_INJECTED).to_c()
    st, got, x, V0 = am.am24_statistics(), np.full(k, -1.0), np.zeros(n, np.float32), np.asfortranarray(V0)
    st.values, st.per_start_capacity = got.ctypes.data_as(C.POINTER(C.c_double)), k
    am.check(am.lib().am24_solve_resident_f32(
        solver.h, M.mh, x.ctypes.data_as(C.c_void_p), C.byref(cs), C.byref(st),
        V0.ctypes.data_as(C.c_void_p), C.byref(C.c_float())))
    M.close()
    want = fo.iteration(B, V0.astype(np.float64), formulation, 6, gamma, np.zeros(k)).val
    assert sure.any()
    assert np.all(np.abs(got - want)[sure] <= 4e-6 * terms[sure]), (got, want)
