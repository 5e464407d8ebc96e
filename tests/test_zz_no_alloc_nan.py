"""aco_pheromone_update_noalloc on lengths whose bits are all ones (a buffer cleared to
0xff): the smallest index is the elite, as among any equal lengths, and what it
deposits is not a number."""
import ctypes

import numpy as np
import pytest

from cvrp_aco_ocl_b200._lib import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ants,ranks,finite", [(1, 2, None), (5, 8, None), (40, 6, None), (40, 6, 33), (2049, 3, None)])
def test_lengths_of_all_ones(gpu, ants, ranks, finite):
    import torch
    n = 37
    rng = np.random.default_rng(ants)
    T = 2 * n
    sol = np.zeros(T * (ants + 1) + 1, np.int32)
    for a in range(ants + 1):
        sol[a * T:a * T + n + 1] = np.r_[0, rng.permutation(np.arange(1, n)), 0]
        sol[a * T + T - 1] = n + 1
    lens = np.full(ants + 1, 0xffffffff, np.uint32).view(np.float32)
    elites = [ants] + [0] * (ranks - 1)
    if finite is not None:  # taken first, and again: +inf has the smaller bits
        lens[finite] = 500.0
        elites[1:] = [finite] * (ranks - 1)
    tau = rng.uniform(0.1, 1.0, (n, n)).astype(np.float32)
    dist = rng.uniform(1.0, 9.0, (n, n)).astype(np.float32)
    want = np.float32(1.0 - np.float32(0.1)) * tau
    for r, a in enumerate(elites):  # knocked-out lengths are only the selection's
        t = sol[a * T:a * T + n + 1]
        want[t[:-1], t[1:]] += np.float32(ranks - r) / lens[a]
    dev = [torch.from_numpy(a).cuda() for a in (tau, np.zeros_like(tau), dist, sol, lens)]
    el = torch.zeros(ranks, dtype=torch.int32, device="cuda")
    rc = lib().aco_pheromone_update_noalloc(
        n, n, ants, ranks, ctypes.c_float(0.1), ctypes.c_float(1.0), ctypes.c_float(2.0),
        *(ctypes.c_void_p(t.data_ptr()) for t in (*dev, el)), None)
    assert rc == 0
    torch.cuda.synchronize()
    assert list(el.cpu().numpy()) == elites
    got = dev[0].cpu().numpy()
    assert np.isnan(got).any() and np.array_equal(got, want, equal_nan=True)
