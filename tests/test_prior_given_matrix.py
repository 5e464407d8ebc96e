"""A given distance matrix of another shape than the instance's is refused before
anything is uploaded (the device list kernel would read n rows of n)."""
import numpy as np
import pytest

from cvrp_aco_ocl_b200 import Problem
from cvrp_aco_ocl_b200 import instances as I
from cvrp_aco_ocl_b200 import prior as PR


@pytest.mark.parametrize("shape", [(40, 40), (60, 61), (61, 60), (62, 62), (61 * 61,)])
def test_wrong_shape_is_refused(shape):
    prob = Problem.from_instance(I.gen_mixed(3, 60))
    prob.distance = np.ones(shape, np.float32)
    with pytest.raises(ValueError):
        PR.GraphBatch.from_problem(prob, 20)
