"""Negative demands under a capacity at the end of its type: what is left is more than
the type holds, and every customer still fits.  Against the oracle, both modes."""
import numpy as np
import pytest

import oracle
from cvrp_aco_ocl_b200 import MODE_PARITY, MODE_THROUGHPUT, Solver
from cvrp_aco_ocl_b200 import instances as I

from test_gpu_parity import compare_state, params_for, problem_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,n,draw", [(MODE_PARITY, 60, 0), (MODE_PARITY, 300, 0), (MODE_THROUGHPUT, 200, 1),
                                         (MODE_THROUGHPUT, 200, -1), (MODE_THROUGHPUT, 1030, 1)])
def test_pickups_under_the_largest_capacity(gpu, mode, n, draw):
    inst = I.gen_mixed(5000 + n, n - 1)
    rng = np.random.default_rng(n)
    inst.demand[1:] = rng.integers(-9, 3, n - 1)
    cap, A, nloc, T0, rs, K = 2**31 - 1, 6, 64, 1796300000, 77, 8
    dist = oracle.compute_distances(inst.x, inst.y)
    thr = mode == MODE_THROUGHPUT
    nn = oracle.compute_nn_lists(dist, K, K)
    seeds, _ = oracle.make_seeds(T0, rs, A, nloc)
    O = oracle.Oracle(dist, inst.demand, cap, A, nloc, nn[:, :0], seeds, ls_flag=False,
                      nn_ants_list=nn if thr else None, n_threads=8)
    p = params_for(n, A, nloc, T0, rs, False, 0, mode=mode, nn_ants=K, draw_warps=draw)
    with Solver(problem_of(inst.x, inst.y, inst.demand, cap), p) as S:
        S.init(); O.init_aco(throughput=thr)
        compare_state(S, O)
        S.iterate(1); O.run_iteration(throughput=thr)
        compare_state(S, O)
