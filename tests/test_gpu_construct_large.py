"""The largest instances of the throughput construct (without a 2-opt, whose own
arrays end earlier): the shared memory of one ant holds 19072 nodes, 18720 beside
a helper warp's draws, with and without a route length limit; one more is refused."""
import numpy as np
import pytest

from cvrp_aco_ocl_b200 import MODE_THROUGHPUT, AcoError, Solver
from cvrp_aco_ocl_b200 import instances as I

from test_gpu_parity import params_for, problem_of

pytestmark = pytest.mark.gpu


def solver(n, limit, draw):
    inst = I.gen_mixed(n, n - 1)
    d0 = np.hypot(inst.x - inst.x[0], inst.y - inst.y[0])
    prob = problem_of(inst.x, inst.y, inst.demand, inst.capacity,
                      max_distance=float(d0.max() * 2.6) if limit else np.inf, service_time=1.0 if limit else 0.0)
    return Solver(prob, params_for(n, 2, 32, 1796300000, 9, False, 0, mode=MODE_THROUGHPUT, nn_ants=8,
                                   draw_warps=draw))


@pytest.mark.parametrize("n,limit,draw", [(16353, True, 0), (18720, False, 0), (19072, False, -1), (19072, True, -1)])
def test_largest_instances(gpu, n, limit, draw):
    with solver(n, limit, draw) as S:
        S.init()
        S.iterate(1)
        assert S.validate()[1] == 0


def test_one_node_more_is_refused(gpu):
    with pytest.raises(AcoError) as e:
        solver(19073, False, -1)
    assert e.value.code == -1
