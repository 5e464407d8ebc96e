"""The 2-opt of routes of 33 to 64 nodes (two positions a lane) and the lengths beside
them: 33, 34, 48, 63, 64 and 65 nodes (unit demands, so the capacity sets the length),
many equal distances (a small integer grid) and none, one route (the depot's bit clear)
and several, lists inside and past one warp's width; the per-ant kernel, the route list
and the fused construct.  Against the oracle."""
import numpy as np
import pytest

import oracle
from cvrp_aco_ocl_b200 import MODE_PARITY, MODE_THROUGHPUT, Solver

from test_gpu_parity import compare_state, params_for, problem_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,kw", [
    (MODE_PARITY, {}), (MODE_THROUGHPUT, {"route_ls": 1}), (MODE_THROUGHPUT, {"route_ls": -1}),
    (MODE_THROUGHPUT, {"fuse_ls": 1})])
@pytest.mark.parametrize("n_cust,cap,grid,nn_ls", [
    (64, 32, 9, 9), (32, 32, 1000, 20), (99, 33, 9, 40), (47, 47, 8, 31), (141, 47, 1000, 33), (126, 62, 10, 12),
    (126, 63, 9, 100), (63, 63, 1000, 20), (128, 64, 1000, 20)])
def test_long_routes_match_oracle(gpu, n_cust, cap, grid, nn_ls, mode, kw):
    rng = np.random.default_rng(1000 * n_cust + cap)
    n = n_cust + 1
    x = rng.integers(0, grid + 1, n).astype(np.float32)
    y = rng.integers(0, grid + 1, n).astype(np.float32)
    dem = np.ones(n, np.int32)
    dem[0] = 0
    A, nloc, T0, rs, K = 16, 64, 1796300000, 47, 10
    nn_ls = min(nn_ls, n - 2)
    depth = max(K, nn_ls)
    dist = oracle.compute_distances(x, y)
    nn = oracle.compute_nn_lists(dist, depth, depth)
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


@pytest.mark.parametrize("near,far,A", [(40, 60, 24), (90, 16, 40), (0, 60, 24), (300, 70, 24)])
def test_full_route_list(gpu, near, far, A):
    """More routes than the list holds (a distance limit leaves the far customers a route
    each): the ants past its end are improved by the per-ant kernel.  The near customers
    give each ant a long route, listed from the other end (of more than 255 nodes: not
    listed)."""
    rng = np.random.default_rng(near + far)
    n = 1 + near + far
    ang = np.arange(far) * (2 * np.pi / max(far, 1))
    x = np.concatenate([[0.0], rng.uniform(-0.5, 0.5, near), 100 * np.cos(ang)]).astype(np.float32)
    y = np.concatenate([[0.0], rng.uniform(-0.5, 0.5, near), 100 * np.sin(ang)]).astype(np.float32)
    dem = np.ones(n, np.int32)
    dem[0] = 0
    maxd = 203.0
    nloc, T0, rs, K, nn_ls = 64, 1796300000, 53, 10, 12
    dist = oracle.compute_distances(x, y)
    nn = oracle.compute_nn_lists(dist, nn_ls, nn_ls)
    seeds, _ = oracle.make_seeds(T0, rs, A, nloc)
    p = params_for(n, A, nloc, T0, rs, True, nn_ls, mode=MODE_THROUGHPUT, nn_ants=K, route_ls=1)
    O = oracle.Oracle(dist, dem, 10 * n, A, nloc, nn[:, :nn_ls], seeds, ls_flag=True, nn_ants_list=nn[:, :K],
                      max_dist=maxd, n_threads=8, ls_pass_limit=4096)
    with Solver(problem_of(x, y, dem, 10 * n, max_distance=maxd), p) as S:
        S.init(); O.init_aco(throughput=True)
        compare_state(S, O)
        for _ in range(3):
            S.iterate(1); O.run_iteration(throughput=True)
            compare_state(S, O)
