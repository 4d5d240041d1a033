"""Device arrays that kernels read in place: one that runs past its allocation is
refused before anything is launched, by the matrix's entry point and the
server's.  The refused span is wider than a process's address space, so it cannot
be mapped whatever lies behind the allocation.  One that does not start on a
float's boundary, which a copy takes, gives the bytes that it holds."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD, N = (1 << 31) - 1, 1 << 16  # 512 TiB


def _am():
    return importlib.import_module("24am_b200")


def test_a_matrix_past_its_allocation_is_refused(solver):
    import torch
    am = _am()
    src = torch.randn(64 << 20, device="cuda")
    torch.cuda.synchronize()
    with pytest.raises(am.Am24Error) as ex:
        am.Matrix(solver, None, on_device_ptr=src.data_ptr(), m=4, n=N, ldB=LD)
    assert "allocation" in str(ex.value)
    srv = am.Server(0, 1 << 30)
    with pytest.raises(am.Am24Error):
        srv.add_matrix(on_device_ptr=src.data_ptr(), m=4, n=N, ldB=LD)
    srv.close()
    # up to its last element it is taken
    ld, n = 1 << 19, 128
    M = am.Matrix(solver, None, on_device_ptr=src.data_ptr(), m=ld, n=n)
    M.close()
    M = am.Matrix(solver, None, on_device_ptr=src.data_ptr() + 4 * (ld - 3), m=3, n=n, ldB=ld)
    want = src.cpu().numpy().reshape(n, ld)[:, -3:].T
    assert np.array_equal(M.read(), want)
    M.close()


@pytest.mark.parametrize("offset", [1, 2, 6])
def test_odd_addresses_are_copied(solver, po, offset):
    import torch
    am = _am()
    m, n, k = 37, 130, 5
    B = po.low_rank_data(m, n, 4, 20, seed=3, dtype=np.float32)
    V = po.uniform_starts(n, k, seed=4, dtype=np.float32)

    def odd(a):
        raw = torch.zeros(a.nbytes + 16, dtype=torch.uint8)
        raw[offset:offset + a.nbytes] = torch.from_numpy(a.reshape(-1, order="F").view(np.uint8).copy())
        return raw.cuda()

    dB, dV = odd(B), odd(V)
    torch.cuda.synchronize()
    M = am.Matrix(solver, None, on_device_ptr=dB.data_ptr() + offset, m=m, n=n)
    assert np.array_equal(M.read(), B)
    b = M.batch(am.OptimizationSettings(constraintParameter=8), k)
    b.load(device_ptr=dV.data_ptr() + offset)
    assert np.array_equal(b.read()[0], V)
    b.close()
    M.close()
