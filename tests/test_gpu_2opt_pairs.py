"""The 2-opt of routes of at most 16 nodes examines two positions at once: routes of
2, 3, 4, 15, 16 and 17 nodes (unit demands, so the capacity sets the length), many
equal distances (a small integer grid) and none, the depot's bit clear (one route)
and set; the per-ant kernel, the route list and the fused construct.  Against the
oracle."""
import numpy as np
import pytest

import oracle
from cvrp_aco_ocl_b200 import MODE_PARITY, MODE_THROUGHPUT, Solver

from test_gpu_parity import compare_state, params_for, problem_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,kw", [
    (MODE_PARITY, {}), (MODE_THROUGHPUT, {"route_ls": 1}), (MODE_THROUGHPUT, {"route_ls": -1}),
    (MODE_THROUGHPUT, {"fuse_ls": 1})])
@pytest.mark.parametrize("n_cust,cap,grid", [
    (40, 1, 8), (40, 2, 8), (41, 3, 8), (15, 15, 6), (14, 14, 1000), (70, 14, 7), (75, 15, 9), (90, 15, 1000), (80, 16, 9)])
def test_short_routes_match_oracle(gpu, n_cust, cap, grid, mode, kw):
    rng = np.random.default_rng(1000 * n_cust + cap)
    n = n_cust + 1
    x = rng.integers(0, grid + 1, n).astype(np.float32)
    y = rng.integers(0, grid + 1, n).astype(np.float32)
    dem = np.ones(n, np.int32)
    dem[0] = 0
    A, nloc, T0, rs, K, nn_ls = 24, 64, 1796300000, 43, 10, 9
    dist = oracle.compute_distances(x, y)
    nn = oracle.compute_nn_lists(dist, K, K)
    seeds, _ = oracle.make_seeds(T0, rs, A, nloc)
    throughput = mode == MODE_THROUGHPUT
    extra = {"nn_ants": K} if throughput else {}
    p = params_for(n, A, nloc, T0, rs, True, nn_ls, mode=mode, **extra, **kw)
    O = oracle.Oracle(dist, dem, cap, A, nloc, nn[:, :nn_ls], seeds, ls_flag=True,
                      nn_ants_list=nn[:, :K] if throughput else None, n_threads=8, ls_pass_limit=4096)
    with Solver(problem_of(x, y, dem, cap), p) as S:
        S.init(); O.init_aco(throughput=throughput)
        compare_state(S, O)
        for _ in range(3):
            S.iterate(1); O.run_iteration(throughput=throughput)
            compare_state(S, O)
