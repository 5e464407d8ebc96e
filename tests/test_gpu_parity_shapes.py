"""Parity launch shapes and the 32 nodes a thread of the construct: shapes that leave
more are refused whoever chose them, shapes of exactly 32 give the oracle's
tours, and the autotuner returns a shape that holds the instance."""
import numpy as np
import pytest

import oracle
from cvrp_aco_ocl_b200 import MODE_PARITY, AcoError, Problem, Solver
from cvrp_aco_ocl_b200 import instances as I
from cvrp_aco_ocl_b200.tune import autotune

from test_gpu_parity import compare_state, params_for, problem_of

pytestmark = pytest.mark.gpu


def shaped(n, A, nloc, wpa, apc):
    inst = I.gen_mixed(2000 + n, n - 1)
    p = params_for(n, A, nloc, 1796300000 + n, 7, False, 0, mode=MODE_PARITY, warps_per_ant=wpa, ants_per_block=apc)
    return inst, p


@pytest.mark.parametrize("n,nloc,wpa,apc", [
    (1025, 256, 0, 16), (1100, 256, 0, 16), (2049, 256, 0, 8), (4097, 256, 0, 4), (1025, 256, 1, 0),
    (2049, 256, 2, 1), (1025, 32, 0, 0), (2049, 64, 0, 0), (8193, 256, 0, 0)])
def test_too_many_nodes_a_thread_are_refused(gpu, n, nloc, wpa, apc):
    inst, p = shaped(n, 4, nloc, wpa, apc)
    with pytest.raises(AcoError) as e:
        Solver(Problem.from_instance(inst), p)
    assert e.value.code == -1


@pytest.mark.parametrize("n,nloc,wpa,apc", [(1024, 32, 0, 0), (1024, 256, 1, 16), (1024, 256, 0, 16), (1025, 256, 0, 8)])
def test_32_nodes_a_thread_vs_oracle(gpu, n, nloc, wpa, apc):
    inst, p = shaped(n, 3, nloc, wpa, apc)
    dist = oracle.compute_distances(inst.x, inst.y)
    seeds, _ = oracle.make_seeds(p.seed_time, p.rnd_seed, 3, nloc)
    O = oracle.Oracle(dist, inst.demand, inst.capacity, 3, nloc, np.zeros((n, 0), np.int32), seeds, ls_flag=False,
                      n_threads=8)
    with Solver(problem_of(inst.x, inst.y, inst.demand, inst.capacity), p) as S:
        apc_run, wpa_run = S.config()[:2]
        assert n <= 1024 * wpa_run
        S.init(); O.init_aco()
        S.iterate(1); O.run_iteration()
        compare_state(S, O)


def test_autotuned_shape_holds_the_instance(gpu):
    inst, p = shaped(1100, 4, 256, 0, 0)
    out, _ = autotune(Problem.from_instance(inst), p, iters=1)
    assert 1100 <= 1024 * out.warps_per_ant
    with Solver(Problem.from_instance(inst), out):
        pass
