"""The depot's row with fewer customers at a finite distance than the candidate list
has places: the depot is then on its own list.  Against the oracle."""
import numpy as np
import pytest

import oracle
from cvrp_aco_ocl_b200 import MODE_THROUGHPUT, Solver
from cvrp_aco_ocl_b200 import instances as I

from test_gpu_parity import compare_state, params_for, problem_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,K,near", [(9, 7, 1), (12, 10, 3), (40, 30, 5), (60, 32, 2)])
def test_depot_on_its_own_list(gpu, n, K, near):
    rng = np.random.default_rng(n)
    inst = I.gen_mixed(4000 + n, n - 1)
    dist = oracle.compute_distances(inst.x, inst.y)
    far = rng.permutation(np.arange(1, n))[near:]
    dist[0, far] = np.inf  # one way only: a route that starts at a near customer has a finite length
    nn = oracle.compute_nn_lists(dist, K, K)
    assert 0 in nn[0, :K]
    cap = int(inst.demand.sum())  # one route
    A, nloc, T0, rs = 7, 64, 1796300000, 31
    prob = problem_of(inst.x, inst.y, inst.demand, cap)
    prob.distance = dist
    p = params_for(n, A, nloc, T0, rs, False, 0, mode=MODE_THROUGHPUT, nn_ants=K)
    seeds, _ = oracle.make_seeds(T0, rs, A, nloc)
    O = oracle.Oracle(dist, inst.demand, cap, A, nloc, nn[:, :0], seeds, ls_flag=False, nn_ants_list=nn, n_threads=8)
    with Solver(prob, p) as S:
        S.init(); O.init_aco(throughput=True)
        compare_state(S, O)
        for _ in range(2):
            S.iterate(1); O.run_iteration(throughput=True)
            compare_state(S, O)
    assert np.isfinite(O.lens).all()
