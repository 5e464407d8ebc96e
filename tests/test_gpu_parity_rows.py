"""The parity construct's register kernel at the edges of its row split: a row one
node short of, at and past the threads of an ant, 16 and 17 nodes a thread (the
latter goes to the shared-memory kernel), one to sixteen nodes an RNG lane, with
and without a route length limit, against the oracle."""
import numpy as np
import pytest

import oracle
from cvrp_aco_ocl_b200 import MODE_PARITY, Solver
from cvrp_aco_ocl_b200 import instances as I

from test_gpu_parity import compare_state, params_for, problem_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,A,nloc,wpa,apc,limit", [
    (5, 3, 32, 1, 0, False), (31, 5, 32, 1, 0, True), (32, 5, 32, 1, 2, False), (33, 5, 32, 1, 0, True),
    (64, 6, 64, 2, 3, False), (65, 6, 64, 2, 0, True), (128, 9, 128, 4, 0, False), (129, 9, 128, 0, 0, True),
    (256, 10, 256, 8, 2, True), (257, 10, 256, 8, 0, False), (512, 6, 32, 1, 0, False), (513, 4, 32, 1, 0, False),
    (300, 7, 64, 2, 0, True), (385, 7, 256, 4, 0, False), (200, 600, 256, 0, 0, False), (90, 12, 256, 0, 16, False)])
def test_row_split_vs_oracle(gpu, n, A, nloc, wpa, apc, limit):
    inst = I.gen_mixed(1000 + n, n - 1)
    dist = oracle.compute_distances(inst.x, inst.y)
    T0, rs = 1796300000 + n, 99
    maxd, serv = (float(np.max(dist[0]) * 2.5), 2.0) if limit else (np.inf, 0.0)
    prob = problem_of(inst.x, inst.y, inst.demand, inst.capacity, max_distance=maxd, service_time=serv)
    p = params_for(n, A, nloc, T0, rs, False, 0, mode=MODE_PARITY, warps_per_ant=wpa, ants_per_block=apc)
    seeds, _ = oracle.make_seeds(T0, rs, A, nloc)
    O = oracle.Oracle(dist, inst.demand, inst.capacity, A, nloc, np.zeros((n, 0), np.int32), seeds, ls_flag=False,
                      max_dist=maxd, serv_time=serv, n_threads=8)
    with Solver(prob, p) as S:
        S.init(); O.init_aco()
        compare_state(S, O)
        S.iterate(2); O.run_iteration(); O.run_iteration()
        compare_state(S, O)
