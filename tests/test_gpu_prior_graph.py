"""The learned prior's graph built on the device: the same bits as build_graph's for
every distance type, integer coordinates with ties, a given matrix, the smallest
graph, and the same prior from either."""
import numpy as np
import pytest

from cvrp_aco_ocl_b200 import Problem
from cvrp_aco_ocl_b200 import instances as I
from cvrp_aco_ocl_b200 import prior as PR

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make,k,kind", [
    (lambda: I.gen_mixed(3, 60), 20, "coords"), (lambda: I.gen_uniform_small(4, 100, coord_max=8), 16, "coords"),
    (lambda: I.gen_large(5, 700), 25, "coords"), (lambda: I.gen_mixed(6, 21), 20, "coords"),
    (lambda: I.gen_uniform_small(7, 80, coord_max=60), 10, "ceil"), (lambda: I.gen_mixed(8, 90), 12, "att"),
    (lambda: I.gen_uniform_small(9, 70, coord_max=80), 12, "geo"), (lambda: I.gen_mixed(10, 64), 31, "given")])
def test_device_graph_equals_host(gpu, make, k, kind):
    prob = Problem.from_instance(make())
    prob.dis_type = {"ceil": I.CEIL_2D, "att": I.ATT, "geo": I.GEO}.get(kind, I.EUC_2D)
    if kind == "given":
        prob.distance = np.random.default_rng(1).integers(1, 40, (prob.num_node,) * 2).astype(np.float32)
    g = PR.build_graph(prob, k)
    b, nbr = PR.GraphBatch.from_problem(prob, k)
    assert np.array_equal(nbr, g.nbr) and b.n_edges == g.n * k
    assert np.array_equal(b.node_feat.cpu().numpy(), g.node_feat)
    assert np.array_equal(b.edge_feat.cpu().numpy(), g.edge_feat)
    S = PR.EdgeScorer.load()
    assert np.array_equal(S.prior(prob, k=k), S.prior(prob, k=k, graph=g))
    with pytest.raises(ValueError):
        S.prior(prob, k=prob.num_node - 1)
