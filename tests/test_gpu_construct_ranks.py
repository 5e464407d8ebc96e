"""The throughput construct by demand rank: sizes around groups of 32 and the
1024-node register limit, all demands equal, zero demands, demands past 16 bits
(the unpacked table), equal distances (ties of total_info in the scan and in the
sorted depot row), with and without helper draw warps and the two-CTA shape, one
limited member in a batch.  Against the oracle."""
import numpy as np
import pytest

import oracle
from cvrp_aco_ocl_b200 import MODE_THROUGHPUT, Batch, Solver
from cvrp_aco_ocl_b200 import instances as I

from test_gpu_parity import compare_state, params_for, problem_of

pytestmark = pytest.mark.gpu


def instance(n, demands, grid, seed):
    rng = np.random.default_rng(seed)
    inst = I.gen_uniform_small(seed, n - 1, coord_max=grid) if grid else I.gen_mixed(seed, n - 1)
    if demands == "equal":
        inst.demand[1:] = 7
        inst.capacity = 50
    elif demands == "zeros":
        inst.demand[1:] = rng.integers(0, 3, n - 1)
        inst.capacity = 9
    elif demands == "wide":
        inst.demand[1:] = rng.integers(1, 200000, n - 1)
        inst.capacity = 700000
    return inst


@pytest.mark.parametrize("n,demands,grid,A,K,draw,ctas,limit", [
    (12, "drawn", 0, 6, 3, 0, 0, False), (32, "equal", 0, 8, 5, 1, 0, False), (33, "drawn", 0, 8, 5, -1, 0, True),
    (64, "zeros", 12, 9, 8, -1, 2, False), (65, "wide", 0, 9, 8, 1, 0, False), (97, "wide", 7, 9, 6, -1, 2, True),
    (200, "equal", 10, 12, 10, 1, 0, False), (257, "drawn", 20, 16, 25, -1, 1, False),
    (1023, "drawn", 0, 5, 25, 1, 0, False), (1024, "equal", 60, 5, 20, -1, 2, False),
    (1025, "zeros", 60, 5, 20, -1, 0, False), (1025, "drawn", 0, 5, 20, 1, 0, True)])
def test_construct_vs_oracle(gpu, n, demands, grid, A, K, draw, ctas, limit):
    inst = instance(n, demands, grid, 3000 + n)
    dist = oracle.compute_distances(inst.x, inst.y)
    nloc, T0, rs = 64, 1796300000, 515
    maxd, serv = (float(np.max(dist[0]) * 2.6), 3.0) if limit else (np.inf, 0.0)
    prob = problem_of(inst.x, inst.y, inst.demand, inst.capacity, max_distance=maxd, service_time=serv)
    p = params_for(n, A, nloc, T0, rs, False, 0, mode=MODE_THROUGHPUT, nn_ants=K, draw_warps=draw, construct_ctas=ctas)
    nn = oracle.compute_nn_lists(dist, K, K)
    seeds, _ = oracle.make_seeds(T0, rs, A, nloc)
    O = oracle.Oracle(dist, inst.demand, inst.capacity, A, nloc, nn[:, :0], seeds, ls_flag=False, nn_ants_list=nn,
                      max_dist=maxd, serv_time=serv, n_threads=8)
    with Solver(prob, p) as S:
        S.init(); O.init_aco(throughput=True)
        compare_state(S, O)
        for _ in range(2):
            S.iterate(1); O.run_iteration(throughput=True)
            compare_state(S, O)
        S.pheromone_init(0.25)  # the table and the depot's order follow every change of total_info
        tau, tot = S.pheromone()
        S.set_state(tau=tau * 2, total=tot[::-1].copy())
        S.construct()
        assert S.status() == 0 and S.validate()[1] <= 1


def test_limited_member_beside_unlimited(gpu):
    probs = []
    for k, (n, lim) in enumerate([(60, False), (45, True), (80, False)]):
        inst = instance(n, "drawn", 0, 70 + k)
        d0 = np.hypot(inst.x - inst.x[0], inst.y - inst.y[0])
        probs.append(problem_of(inst.x, inst.y, inst.demand, inst.capacity,
                                max_distance=float(d0.max() * 2.6) if lim else np.inf, service_time=1.0 if lim else 0.0))
    p = params_for(80, 16, 64, 1796300000, 9, True, 10, mode=MODE_THROUGHPUT, nn_ants=10)
    with Batch(probs, p) as B:
        B.init(); B.iterate(3)
        for b, prob in enumerate(probs):
            q = params_for(prob.num_node, 16, 64, 1796300000, 9 + b, True, 10, mode=MODE_THROUGHPUT, nn_ants=10)
            with Solver(prob, q) as S:
                S.init(); S.iterate(3)
                assert np.array_equal(B.solutions(b)[0], S.solutions()[0])
                assert np.array_equal(B.solutions(b)[1], S.solutions()[1])
