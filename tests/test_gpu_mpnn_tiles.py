"""The edge-scoring network's kernels at the edges of their tiles: row counts one
below, at and above a 128-row tile, one and 32 neighbours a node, one layer (the
first and the last at once), more tiles than resident CTAs, a gradient buffer
that is not 16-byte aligned."""
import ctypes

import numpy as np
import pytest

from oracle import mpnn_oracle as M
from cvrp_aco_ocl_b200 import prior as PR
from cvrp_aco_ocl_b200._lib import check, lib

from test_gpu_mpnn import GRAD_RTOL, SCORE_RTOL, concat

pytestmark = pytest.mark.gpu


def graphs(seed, sizes, k):
    """k distinct random neighbours of every node: the node's id plus distinct offsets."""
    rng = np.random.default_rng(seed)
    out = []
    for n in sizes:
        off = np.argsort(rng.uniform(size=(n, n - 1)), axis=1)[:, :k] + 1
        nbr = ((np.arange(n)[:, None] + off) % n).astype(np.int32).ravel()
        out.append(PR.Graph(n, k, rng.uniform(0, 1, size=(n, M.F_NODE)).astype(np.float32),
                            rng.uniform(0, 1.5, size=n * k).astype(np.float32), nbr, None))
    return out


@pytest.mark.parametrize("k,sizes,layers,shift", [
    (1, [128], 1, 0), (3, [43], 1, 0), (1, [127], 3, 1), (32, [64], 2, 0), (13, [65, 128], 3, 0), (20, [3001], 3, 0)])
def test_network_at_tile_edges(gpu, k, sizes, layers, shift):
    import torch
    gs = graphs(31 * k + layers, sizes, k)
    rng = np.random.default_rng(9)
    labels = [(rng.uniform(size=g.n * k) < 0.15).astype(np.float32) for g in gs]
    flat = (M.init_params(3, layers) + rng.normal(0, 0.02, M.init_params(3, layers).shape)).astype(np.float32)
    S = PR.EdgeScorer(layers=layers, params=flat)
    b = PR.GraphBatch(gs, labels)
    infer = S.scores(b).cpu().numpy()
    ws = S._workspace(b.n_nodes, k)
    buf = torch.full((S.count + 1,), 7.0, dtype=torch.float32, device="cuda")
    grad, logits = buf[shift:shift + S.count], torch.empty(b.n_edges, dtype=torch.float32, device="cuda")
    check(lib().aco_mpnn_grad(b.n_nodes, k, layers, S.params.data_ptr(), b.node_feat.data_ptr(), b.edge_feat.data_ptr(),
                              b.nbr.data_ptr(), b.labels.data_ptr(), 3.0, ctypes.c_void_p(ws.data_ptr()), ws.numel(),
                              grad.data_ptr(), S.loss.data_ptr(), logits.data_ptr(), S._stream()), "aco_mpnn_grad")
    S._status()
    assert float(buf[0 if shift else S.count]) == 7.0  # the word beside the gradient stays
    nf, ef, nbr = concat(gs)
    s, saved = M.forward(flat.astype(np.float64), nf, ef, nbr, k, layers, bf16=True)
    for got in (infer, logits.cpu().numpy()):
        assert np.max(np.abs(got - s)) <= SCORE_RTOL * (1.0 + np.max(np.abs(s)))
    loss, ds = M.loss_and_dlogit(s, np.concatenate(labels), 3.0)
    want = M.backward(flat.astype(np.float64), nf, ef, nbr, k, saved, ds, layers, bf16=True)
    assert abs(float(S.loss.item()) - loss) <= 1e-4 * (1 + abs(loss))
    got, o = grad.cpu().numpy().astype(np.float64), 0
    for name, sh in M.param_shapes(layers):
        m = int(np.prod(sh))
        err = np.linalg.norm(got[o:o + m] - want[o:o + m]) / max(np.linalg.norm(want[o:o + m]), 1e-12)
        assert err <= GRAD_RTOL, (name, err)
        o += m
