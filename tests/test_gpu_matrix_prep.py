"""Matrices taken in from device memory (any leading dimension and alignment) and
deflated by sparse components: what is read back is the input bit for bit, and
(float)(b - y_i x_c) in FP64 wherever that is defined, zeros of x and non-finite
data included."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("m,ld", [(1, 1), (31, 31), (32, 32), (33, 36), (130, 133), (1025, 1028)])
def test_device_matrix_is_taken_in_as_it_is(solver, m, ld, offset):
    import torch
    am = importlib.import_module("24am_b200")
    n = 67
    flat = torch.randn(n * ld + offset, device="cuda")
    torch.cuda.synchronize()
    M = am.Matrix(solver, None, on_device_ptr=flat.data_ptr() + 4 * offset, m=m, n=n, ldB=ld)
    want = flat[offset:].cpu().numpy().reshape(n, ld)[:, :m].T
    assert np.array_equal(M.read(), want)
    M.close()


@pytest.mark.parametrize("bad", [None, np.inf, np.nan])
@pytest.mark.parametrize("m,n", [(40, 70), (129, 515)])
def test_deflation_by_a_sparse_component(solver, po, m, n, bad):
    rng = np.random.default_rng(m)
    B = rng.standard_normal((m, n)).astype(np.float32)
    x = np.zeros(n, np.float32)
    at = rng.choice(n, 9, replace=False)
    x[at] = rng.standard_normal(9)
    if bad is not None:
        B[3, at[0]] = bad
    M = solver.matrix(B)
    st = importlib.import_module("24am_b200").OptimizationSettings(
        totalStartingPoints=130, batchSize=130, maximumIterations=1, constraintParameter=5)
    M.solve(st)  # so that the operand planes exist and are rebuilt
    M.deflate(x)
    got = M.read()
    M.close()
    with np.errstate(invalid="ignore"):
        y = (B[:, at].astype(np.float64) * x[at].astype(np.float64)).sum(axis=1)
        want = B.astype(np.float64) - y[:, None] * x.astype(np.float64)[None, :]
    finite = np.isfinite(want)
    assert np.array_equal(np.isfinite(got), finite)
    # y is summed in another order: an FP32 step at most
    assert np.allclose(got[finite], want[finite], rtol=1.2e-7, atol=1e-12)
    if bad is None:
        keep = np.setdiff1d(np.arange(n), at)
        assert np.array_equal(got[:, keep], B[:, keep])
