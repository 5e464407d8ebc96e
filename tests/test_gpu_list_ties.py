"""The device's neighbour lists where ties, few distinct values and row lengths decide
the path: rows of at most 64 nodes, more than 64 equal values, all equal, ties inside
and just outside the list, lists of one entry, of 31 and past 32; against the host's."""
import ctypes

import numpy as np
import pytest

from cvrp_aco_ocl_b200 import compute_nn_lists
from cvrp_aco_ocl_b200._lib import check, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,values,depth", [
    (3, 9, 1), (40, 5, 20), (64, 10 ** 6, 31), (65, 10 ** 6, 31), (66, 3, 25), (129, 1, 25), (200, 40, 1),
    (300, 6, 25), (700, 300, 25), (701, 10 ** 7, 25), (702, 5000, 31), (1100, 900, 40), (1500, 2, 30)])
def test_lists_equal_host(gpu, n, values, depth):
    import torch
    m = np.random.default_rng(n + values).integers(0, values, (n, n)).astype(np.float32)
    ld = (n + 31) // 32 * 32
    dd = torch.zeros((n, ld), dtype=torch.float32, device="cuda")
    dd[:, :n] = torch.tensor(m, device="cuda")
    got, nn = ctypes.c_int(), torch.zeros(n * depth, dtype=torch.int32, device="cuda")
    check(lib().aco_compute_nn_lists_device(n, dd.data_ptr(), ld, depth, depth, nn.data_ptr(), ctypes.byref(got),
                                            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "nn")
    torch.cuda.synchronize()
    assert got.value == depth
    assert np.array_equal(nn.cpu().numpy().reshape(n, depth), compute_nn_lists(m, depth, depth))
