"""The swap stage with its warps on consecutive positions: tours shorter than the
warps' reach, a route length limit with service time, the four-warp shape of
many ants, candidates past one round of 64, against the oracle."""
import numpy as np
import pytest

import oracle
from cvrp_aco_ocl_b200 import MODE_THROUGHPUT, Solver
from cvrp_aco_ocl_b200 import instances as I

from test_gpu_parity import compare_state, params_for, problem_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_cust,per_route,A,limit", [
    (4, 2.0, 6, False), (9, 4.0, 8, True), (30, 1.2, 10, False), (60, 9.0, 700, False), (70, 12.0, 620, True),
    (330, 14.0, 12, False)])
def test_swap_positions_vs_oracle(gpu, n_cust, per_route, A, limit):
    inst = I.gen_mixed(500 + n_cust, n_cust, customers_per_route=per_route)
    dist = oracle.compute_distances(inst.x, inst.y)
    n, nloc, T0, rs = inst.n, 64, 1796300000, 808
    nn_ls = K = min(15, n - 2)
    maxd, serv = (float(np.max(dist[0]) * 2.4), 4.0) if limit else (np.inf, 0.0)
    prob = problem_of(inst.x, inst.y, inst.demand, inst.capacity, max_distance=maxd, service_time=serv)
    p = params_for(n, A, nloc, T0, rs, True, nn_ls, mode=MODE_THROUGHPUT, nn_ants=K)
    p.ls_flag = 3
    nn = oracle.compute_nn_lists(dist, K, K)
    seeds, _ = oracle.make_seeds(T0, rs, A, nloc)
    O = oracle.Oracle(dist, inst.demand, inst.capacity, A, nloc, nn, seeds, ls_flag=3, nn_ants_list=nn,
                      max_dist=maxd, serv_time=serv, n_threads=8, ls_pass_limit=4096)
    with Solver(prob, p) as S:
        S.init(); O.init_aco(throughput=True)
        compare_state(S, O)
        for _ in range(2):
            S.iterate(1); O.run_iteration(throughput=True)
            compare_state(S, O)
