"""aco_pheromone_update_noalloc where its row blocks can go wrong: two nodes, a last
block of one row, rows a column short of and past a chunk, the largest n, more
ants than the kernel holds lengths for, equal lengths, fewer ants than ranks."""
import ctypes

import numpy as np
import pytest

from cvrp_aco_ocl_b200._lib import lib

from test_zz_no_alloc import _update_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ld,ants,ranks", [
    (2, 2, 1, 1), (3, 5, 2, 8), (127, 127, 40, 6), (128, 131, 2049, 8), (149, 149, 5000, 8), (297, 300, 64, 3),
    (1025, 1025, 20, 8), (4096, 4096, 9, 8)])
def test_row_blocks(gpu, n, ld, ants, ranks):
    import torch
    rng = np.random.default_rng(n + ants)
    T = 2 * n
    xy = rng.uniform(0, 100, (n, 2)).astype(np.float32)
    dist = np.sqrt(((xy[:, None] - xy[None]) ** 2).sum(-1, dtype=np.float32))
    sol = np.zeros(T * (ants + 1) + 1, np.int32)
    few = rng.permutation(ants)[:16]  # only these tours can be elite: the others are longer
    lens = np.full(ants + 1, 9e5, np.float32)
    lens[few] = rng.integers(500, 506, few.size).astype(np.float32)  # ties
    lens[ants] = 499.0
    for a in [*few, 0, ants]:
        perm = rng.permutation(np.arange(1, n)).astype(np.int32)
        tour = np.concatenate([np.r_[np.int32(0), r] for r in np.array_split(perm, max(1, (n - 1) // 9))] + [[0]])
        sol[a * T:a * T + tour.size] = tour
        sol[a * T + T - 1] = tour.size
    tau = rng.uniform(0.1, 1.0, n * n).astype(np.float32)
    want_tau, want_tot, elites = _update_np(tau, dist.ravel(), sol, lens, n, ants, ranks)

    def pitched(a):
        m = np.full((n, ld), 3.5, np.float32)
        m[:, :n] = a.reshape(n, n)
        return torch.from_numpy(m).cuda()
    tau_d, tot_d, dist_d = pitched(tau), pitched(np.zeros(n * n, np.float32)), pitched(dist)
    sol_d, lens_d = torch.from_numpy(sol).cuda(), torch.from_numpy(lens).cuda()
    el_d = torch.zeros(ranks, dtype=torch.int32, device="cuda")
    rc = lib().aco_pheromone_update_noalloc(
        n, ld, ants, ranks, ctypes.c_float(0.1), ctypes.c_float(1.0), ctypes.c_float(2.0),
        *(ctypes.c_void_p(t.data_ptr()) for t in (tau_d, tot_d, dist_d, sol_d, lens_d, el_d)), None)
    assert rc == 0
    torch.cuda.synchronize()
    assert list(el_d.cpu().numpy()) == elites
    got_tau, got_tot = tau_d.cpu().numpy(), tot_d.cpu().numpy()
    assert np.array_equal(got_tau[:, :n].ravel(), want_tau)
    assert np.array_equal(got_tot[:, :n].ravel(), want_tot)
    assert np.all(got_tau[:, n:] == 3.5) and np.all(got_tot[:, n:] == 3.5)
