"""What the server counts for a resident matrix is what it takes from the device:
measured on one sample and many features, where the layouts' per-feature words
are a visible share.  The matrix is two allocations, and the device hands out
memory in pieces of 2 MiB, so it may take 4 MiB more than it was counted for."""
import importlib
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_resident_matrix_is_counted_in_full():
    import torch
    am = importlib.import_module("24am_b200")
    B = np.ones((1, 1 << 21), np.float32)
    srv = am.Server(0, 1)
    with pytest.raises(am.Am24Error) as ex:
        srv.add_matrix(B)
    srv.close()
    counted = int(re.search(r"matrix needs (\d+) bytes", str(ex.value)).group(1))
    srv = am.Server(0, 4 << 30)
    srv.add_matrix(B[:, :1 << 16])  # the first upload's own buffers
    before = torch.cuda.mem_get_info()[0]
    srv.add_matrix(B)
    taken = before - torch.cuda.mem_get_info()[0]
    srv.close()
    assert counted <= taken <= counted + (4 << 20)
