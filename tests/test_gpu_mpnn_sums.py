"""The order of the network's gradient sums, to the bit, and two training steps.

One layer with weights under which every number of the backward is known: the
edge embedding is 0, q = 1 on every edge, z = 1, the logit an exact 0 (the output
weights come in pairs v, -v), so dL/dq of an edge is the BF16 rounding of
(0.5 - label) / E times the output weight.  dB, the biases and the embeddings must
then be the fp32 sums in the stated orders: an edge tile's rows in order, a node's
edges in order, 128 nodes in order, 256 strands of the embeddings.  A bias is
compared where at most two CTAs add to it (a sum of two has no order)."""
import numpy as np
import pytest

from oracle import mpnn_oracle as M
from cvrp_aco_ocl_b200 import prior as PR

from test_gpu_mpnn import SCORE_RTOL, concat, random_graphs

pytestmark = pytest.mark.gpu
f32 = np.float32


def in_order(a):
    """The fp32 sum of a's rows, first to last."""
    return np.add.accumulate(a.astype(f32), axis=0, dtype=f32)[-1]


def strands(a):
    """Rows t, t + 256, ... in order, a butterfly over 32 strands, the eight results in order."""
    p = np.zeros((256,) + a.shape[1:], f32)
    for i in range(0, a.shape[0], 256):
        p[:min(256, a.shape[0] - i)] += a[i:i + 256]
    p = p.reshape(8, 32, *a.shape[1:])
    for off in (16, 8, 4, 2, 1):
        p = p + p[:, np.arange(32) ^ off]
    return in_order(p[:, 0])


@pytest.mark.parametrize("n,k", [(1, 32), (1, 1), (6, 20), (12, 20), (9, 13), (128, 20), (129, 5), (256, 1), (300, 20), (40001, 1)])
def test_gradient_sums_in_order(gpu, n, k):
    H = M.H
    rng = np.random.default_rng(1000 * n + k)
    d = {name: np.zeros(sh) for name, sh in M.param_shapes(1)}
    d["W0"][2 * H:3 * H] = np.eye(H)  # dL/dh of the embedding is then dB
    d["a0"][:] = 1.0
    d["W_h"][:] = np.eye(H)
    v = rng.uniform(0.5, 1.5, H // 2).astype(f32)
    d["w_o"][0::2], d["w_o"][1::2] = v, -v
    nf, ef = rng.uniform(0, 1, (n, M.F_NODE)).astype(f32), rng.uniform(0, 1.5, n * k).astype(f32)
    y = rng.uniform(-3, 3, n * k).astype(f32)
    S = PR.EdgeScorer(layers=1, params=M.pack(d, 1).astype(f32))
    g = PR.Graph(n, k, nf, ef, rng.integers(0, n, n * k).astype(np.int32), None)
    s = S.compute_grad(PR.GraphBatch([g], [y]), 1.0).cpu().numpy()
    assert not s.any()
    got = M.unpack(S.grad.cpu().numpy(), 1)

    half, inv_e = f32(0.5), f32(1.0) / f32(n * k)
    ds = (y * -half + (f32(1.0) - y) * half) * inv_e
    dq = M.bf16_round(ds[:, None] * d["w_o"].astype(f32)).astype(f32)
    dB = np.stack([in_order(dq[i * k:(i + 1) * k]) for i in range(n)])
    dh = M.bf16_round(dB).astype(f32)
    assert np.array_equal(got["b_e"], strands(dq))
    assert np.array_equal(got["W_e"][:, 0], strands(dq * ef[:, None]))
    assert np.array_equal(got["b_n"], strands(dh))
    for c in range(M.F_NODE):
        assert np.array_equal(got["W_n"][:, c], strands(dh * nf[:, c:c + 1]))
    rows = 128 // k * k
    tiles = [in_order(dq[e:e + rows]) for e in range(0, n * k, rows)]
    groups = [in_order(dB[i:i + 128]) for i in range(0, n, 128)]
    for bias, parts, terms in ((got["a0"], tiles, dq), (got["b0"][2 * H:3 * H], groups, dB)):
        if len(parts) <= 2:
            assert np.array_equal(bias, in_order(np.stack(parts)))
        else:  # any order of m fp32 terms is within m 2^-24 of their absolute sum
            t = terms.astype(np.float64)
            assert np.all(np.abs(bias - t.sum(0)) <= len(t) * 2.0**-24 * np.abs(t).sum(0))


def test_second_step_matches_oracle(gpu):
    """Gradient, Adam, logits again.  The parameters after the step are off by the
    optimiser's 0.1 lr / sqrt(v) times the gradient's error (2e-2 of about 1e-3, so 3e-6 of
    weights of about 0.1): less than a BF16 unit, but it moves operands that lie at a rounding
    boundary to the next one, as FP32 accumulation does in the first pass.  So the second
    logits may be off by the forward's bound twice."""
    import torch
    k, sizes, lr, step = 20, [45, 33, 60], 1e-3, 200
    gs = random_graphs(77, sizes, k)
    rng = np.random.default_rng(8)
    labels = [(rng.uniform(size=g.n * k) < 0.15).astype(f32) for g in gs]
    flat = (M.init_params(3) + rng.normal(0, 0.02, M.param_count())).astype(f32)
    m, v = 1e-3 * rng.standard_normal(flat.size), 1e-6 * rng.uniform(0.5, 2.0, flat.size)
    S = PR.EdgeScorer(params=flat)
    S.m.copy_(torch.from_numpy(m.astype(f32)))
    S.v.copy_(torch.from_numpy(v.astype(f32)))
    S.step = step
    b = PR.GraphBatch(gs, labels)
    S.compute_grad(b, 3.0)
    S.adam(lr)
    got = S.compute_grad(b, 3.0).cpu().numpy()

    nf, ef, nbr = concat(gs)
    p, y = flat.astype(np.float64), np.concatenate(labels)
    s, saved = M.forward(p, nf, ef, nbr, k, bf16=True)
    g = M.backward(p, nf, ef, nbr, k, saved, M.loss_and_dlogit(s, y, 3.0)[1], bf16=True)
    m, v, t = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g, step + 1
    p = p - lr * (m / (1 - 0.9 ** t)) / (np.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
    want, _ = M.forward(p, nf, ef, nbr, k, bf16=True)
    assert np.max(np.abs(want - s)) > 10 * SCORE_RTOL  # the step did move them
    assert np.max(np.abs(got - want)) <= 2 * SCORE_RTOL * (1.0 + np.max(np.abs(want)))
