"""The register 2-opt where its list membership by distance can go wrong: many equal
and zero distances (small integer grids), lists of one entry, of 32 and 33, of all
customers; routes of 31 to 34 nodes; a matrix with an infinite entry (which takes
the list-scanning paths); the per-ant kernel, the route list and the fused
construct.  Against the oracle."""
import numpy as np
import pytest

import oracle
from cvrp_aco_ocl_b200 import MODE_PARITY, MODE_THROUGHPUT, Solver
from cvrp_aco_ocl_b200 import instances as I

from test_gpu_parity import compare_state, params_for, problem_of

pytestmark = pytest.mark.gpu


def matrix_of(kind, inst):
    d = oracle.compute_distances(inst.x, inst.y)
    if kind == "coords":
        return d, False
    d = d.copy()
    d[3, 5] = d[5, 3] = np.inf
    return d, True


@pytest.mark.parametrize("kind,grid,n_cust,cap,A,mode,nn_ls,kw", [
    ("coords", 6, 90, 160, 32, MODE_PARITY, 88, {}),
    ("coords", 6, 90, 160, 32, MODE_PARITY, 7, {}),
    ("coords", 9, 120, 480, 24, MODE_PARITY, 33, {}),
    ("coords", 9, 120, 480, 24, MODE_THROUGHPUT, 12, {"route_ls": 1}),
    ("coords", 9, 120, 480, 24, MODE_THROUGHPUT, 12, {"route_ls": -1}),
    ("coords", 9, 120, 480, 24, MODE_THROUGHPUT, 12, {"fuse_ls": 1}),
    ("coords", 5, 60, 100, 40, MODE_THROUGHPUT, 1, {"route_ls": 1}),
    ("coords", 40, 100, 500, 40, MODE_THROUGHPUT, 32, {"route_ls": 1, "host_prep": 1}),
    ("coords", 40, 100, 500, 40, MODE_THROUGHPUT, 99, {"route_ls": 1}),
    ("inf", 30, 60, 300, 16, MODE_THROUGHPUT, 20, {"route_ls": 1}),
    ("inf", 30, 60, 300, 16, MODE_PARITY, 20, {})])
def test_2opt_matches_oracle(gpu, kind, grid, n_cust, cap, A, mode, nn_ls, kw):
    inst = I.gen_uniform_small(17 * n_cust + grid, n_cust, coord_max=grid, capacity=cap)
    dist, given = matrix_of(kind, inst)
    prob = problem_of(inst.x, inst.y, inst.demand, inst.capacity)
    if given:
        prob.distance = dist
    n, nloc, T0, rs, K = inst.n, 64, 1796300000, 41, 15
    depth = max(nn_ls, K)
    nn = oracle.compute_nn_lists(dist, depth, depth)
    seeds, _ = oracle.make_seeds(T0, rs, A, nloc)
    throughput = mode == MODE_THROUGHPUT
    extra = {"nn_ants": K} if throughput else {}
    p = params_for(n, A, nloc, T0, rs, True, nn_ls, mode=mode, **extra, **kw)
    O = oracle.Oracle(dist, inst.demand, inst.capacity, A, nloc, nn[:, :nn_ls], seeds, ls_flag=True,
                      nn_ants_list=nn[:, :K] if throughput else None, n_threads=8, ls_pass_limit=4096)
    with Solver(prob, p) as S:
        S.init(); O.init_aco(throughput=throughput)
        compare_state(S, O)
        for _ in range(3):
            S.iterate(1); O.run_iteration(throughput=throughput)
            compare_state(S, O)
