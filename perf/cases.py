"""What a user of this framework has it do, as cases that can be timed and compared.

A case names a kind of work and its sizes; ``prepare`` makes what a program has
in hand before the call (instances from a seeded generator, a solver or batch
handle, network weights and graphs), ``run`` is one pass through the public
entry points.  Kinds:

* ``driver``: the reference's driver surface (``GACO.run``): parity mode, a
  best-so-far readback after every iteration; the smallest calls.
* ``solve``: one instance on a solver handle: initial iteration, some
  iterations, the ants' lengths and the best tour.  Both modes, with or without
  a route length limit, the inter-route swap stage on or off.
* ``batch``: many uneven instances in the same launches.
* ``cold``: a batch from host arrays to its best tours, handle included.
* ``train``: one training step of the edge-scoring network on whole graphs.
* ``prior``: the learned prior of an instance, graph build to dense matrix.
* ``update``: the pheromone update on the caller's own device buffers.
"""
import ctypes
import math

import numpy as np
import torch

from cvrp_aco_ocl_b200 import instances as gen
from cvrp_aco_ocl_b200 import prior as learned
from cvrp_aco_ocl_b200._lib import MODE_PARITY, MODE_THROUGHPUT, check, lib
from cvrp_aco_ocl_b200.aco import GACO, Batch, Problem, Solver, default_params, init_problem

SEED_TIME = 1796300000
RANKS = 6


def listed():
    return [
        # the reference's own use: 50 customers, one ant a node, full lists, read back after every iteration
        {"name": "driver_50", "kind": "driver", "customers": 50, "iters": 20},
        # the library's defaults on a mid-size instance: parity mode, one ant a node, full 2-opt lists
        {"name": "parity_200", "kind": "solve", "mode": "parity", "customers": 200, "ants": 201, "nn_ants": 25,
         "nn_ls": 199, "iters": 5, "limit": False, "swap": False},
        # parity mode on an odd, larger instance with a route length limit and service time, shorter lists
        {"name": "parity_483_limit", "kind": "solve", "mode": "parity", "customers": 483, "ants": 120, "nn_ants": 25,
         "nn_ls": 60, "iters": 3, "limit": True, "swap": False},
        # one clustered instance in throughput mode, latency bound: few ants per multiprocessor
        {"name": "single_200", "kind": "solve", "mode": "throughput", "customers": 200, "ants": 200, "nn_ants": 25,
         "nn_ls": 25, "iters": 10, "limit": False, "swap": False},
        # one large instance, 30-entry lists
        {"name": "single_1000", "kind": "solve", "mode": "throughput", "customers": 1000, "ants": 256, "nn_ants": 30,
         "nn_ls": 30, "iters": 5, "limit": False, "swap": False},
        # 2-opt followed by the inter-route swap of the CPU local search
        {"name": "single_301_swap", "kind": "solve", "mode": "throughput", "customers": 301, "ants": 128,
         "nn_ants": 20, "nn_ls": 20, "iters": 4, "limit": False, "swap": True},
        # serving: 512 independent instances of 100-1000 customers in the same launches
        {"name": "batch_512", "kind": "batch", "count": 512, "n_min": 100, "n_max": 1000, "ants": 128, "nn": 25,
         "iters": 3, "limit": False},
        # a small batch of small instances with a route length limit and service time
        {"name": "batch_40_limit", "kind": "batch", "count": 40, "n_min": 30, "n_max": 260, "ants": 64, "nn": 20,
         "iters": 5, "limit": True},
        # host arrays in, best tours out: creation, initial iteration, two iterations
        {"name": "cold_64", "kind": "cold", "count": 64, "n_min": 100, "n_max": 700, "ants": 64, "nn": 25, "iters": 2,
         "limit": False},
        # one optimiser step of the network: 32 graphs of 100-500 nodes, the training recipe's mini-batch
        {"name": "train_32", "kind": "train", "graphs": 32, "n_min": 100, "n_max": 500, "k": 20},
        # the prior of one large instance for the colony, as time to a usable matrix
        {"name": "prior_1000", "kind": "prior", "customers": 1000, "k": 20},
        # the pheromone update of a host that owns all device memory
        {"name": "update_1000", "kind": "update", "customers": 1000, "ants": 256, "pad": 0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["driver", "solve", "solve", "solve", "batch", "batch", "cold", "train", "prior", "update"])
    if kind == "driver":
        return {"kind": kind, "customers": rng.randint(20, 120), "iters": rng.randint(5, 30)}
    if kind == "solve":
        mode = rng.choice(["parity", "throughput", "throughput"])
        customers = _log_int(rng, 40, 800 if mode == "parity" else 1200)
        nn = rng.randint(10, 30)
        return {"kind": kind, "mode": mode, "customers": customers, "ants": _log_int(rng, 32, 400), "nn_ants": nn,
                "nn_ls": nn if mode == "throughput" else rng.randint(nn, customers - 1), "iters": rng.randint(2, 6),
                "limit": rng.random() < 0.3, "swap": rng.random() < 0.2}
    if kind in ("batch", "cold"):
        n_min = _log_int(rng, 25, 200)
        n_max = _log_int(rng, n_min + 40, 1000)
        return {"kind": kind, "count": _log_int(rng, 8, 256 if kind == "batch" else 96), "n_min": n_min,
                "n_max": n_max, "ants": rng.choice([32, 64, 100, 128]), "nn": rng.randint(10, min(30, n_min - 1)),
                "iters": rng.randint(2, 5), "limit": rng.random() < 0.3}
    if kind == "train":
        n_min = rng.randint(60, 200)
        return {"kind": kind, "graphs": _log_int(rng, 2, 32), "n_min": n_min, "n_max": rng.randint(n_min + 20, 500),
                "k": rng.choice([10, 16, 20, 25])}
    if kind == "prior":
        return {"kind": kind, "customers": _log_int(rng, 100, 1200), "k": rng.choice([10, 16, 20, 25])}
    return {"kind": kind, "customers": _log_int(rng, 50, 2500), "ants": _log_int(rng, 32, 400),
            "pad": rng.choice([0, 0, 3, 27])}


# ---- inputs ----------------------------------------------------------------
def _limit(p):
    """A route length limit of about two thirds of what capacity alone allows, with
    service time, under which every customer can still be served."""
    d = np.hypot(p.x - p.x[0], p.y - p.y[0])
    p.service_time = 5.0
    p.max_distance = float(2.0 * d.max() * 1.05 + p.service_time + 0.6 * float(d.mean()))
    return p


def _one(case, seed):
    """The instance of a single-instance case: both generators, by seed."""
    c = case["customers"]
    return Problem.from_instance(gen.gen_mixed(seed, c) if c <= 400 else gen.gen_large(seed, c))


def _sizes(case, count):
    """Customers of every instance: uniform over the case's range, the same for all seeds."""
    lo, hi = case["n_min"], case["n_max"]
    return np.random.default_rng(lo * 4099 + hi).integers(lo, hi + 1, size=count)


def _many(case, seed):
    """Instances of the mixed and the large generators alternately, as the batched workload has them."""
    rng = np.random.default_rng(seed)
    ps = []
    for b, c in enumerate(_sizes(case, case["count"])):
        make = gen.gen_mixed if b % 2 == 0 else gen.gen_large
        ps.append(Problem.from_instance(make(int(rng.integers(1 << 30)), int(c))))
    return [_limit(p) for p in ps] if case["limit"] else ps


def _batch_params(case, seed, problems):
    p = default_params(max(q.num_node for q in problems))
    p.mode, p.n_ants, p.nn_ants, p.nn_ls, p.ras_ranks = MODE_THROUGHPUT, case["ants"], case["nn"], case["nn"], RANKS
    p.seed_time, p.rnd_seed = SEED_TIME, seed % 100000
    return p


def _sweep_tour(p):
    """A feasible tour: customers by angle around the depot, cut at capacity."""
    order = np.argsort(np.arctan2(p.y[1:] - p.y[0], p.x[1:] - p.x[0]), kind="stable") + 1
    tour, load = [0], 0
    for c in order:
        if load + int(p.demand[c]) > p.vehicle_capacity:
            tour.append(0)
            load = 0
        tour.append(int(c))
        load += int(p.demand[c])
    return np.array(tour + [0])


def _train_inputs(case, seed):
    rng = np.random.default_rng(seed)
    problems = [Problem.from_instance(gen.gen_mixed(int(rng.integers(1 << 30)), int(c)))
                for c in _sizes(case, case["graphs"])]
    graphs = [learned.build_graph(p, case["k"], keep_dist=False) for p in problems]
    labels = [learned.route_labels(g, _sweep_tour(p)) for g, p in zip(graphs, problems)]
    return graphs, labels


def _train_state(seed, count):
    """Optimiser moments of a run under way (gradients of this loss are about 1e-3)."""
    rng = np.random.default_rng(seed + 77)
    m = (1e-3 * rng.standard_normal(count)).astype(np.float32)
    v = (1e-6 * rng.uniform(0.5, 2.0, count)).astype(np.float32)
    return m, v


LR, STEP, POS_WEIGHT = 1e-3, 200, 9.0


def _update_inputs(case, seed):
    """tau, distances, ant tours and lengths in the reference layout (host arrays)."""
    rng = np.random.default_rng(seed)
    n, A = case["customers"] + 1, case["ants"]
    ld, T = n + case["pad"], 2 * n
    xy = rng.uniform(0.0, 1000.0, size=(n, 2)).astype(np.float32)
    d = np.zeros((n, ld), np.float32)
    d[:, :n] = np.sqrt(((xy[:, None, :] - xy[None, :, :]) ** 2).sum(-1, dtype=np.float32))
    tau = rng.uniform(1e-6, 1e-4, size=(n, ld)).astype(np.float32)
    sol = np.zeros(T * (A + 1) + 1, np.int32)
    lens = np.zeros(A + 1, np.float32)
    for a in range(A + 1):
        perm = rng.permutation(n - 1) + 1
        tour = np.concatenate([np.concatenate([[0], r]) for r in np.array_split(perm, max(1, n // 12))] + [[0]])
        sol[a * T:a * T + tour.size] = tour
        sol[a * T + T - 1] = tour.size
        lens[a] = d[tour[:-1], tour[1:]].sum(dtype=np.float64)
    best = int(np.argmin(lens[:A]))
    sol[A * T:(A + 1) * T] = sol[best * T:(best + 1) * T]
    lens[A] = lens[best]
    sol[-1] = best
    return n, ld, A, tau, d, sol, lens


def prepare(case, seed):
    kind = case["kind"]
    if kind == "driver":
        p = Problem.from_instance(gen.gen_uniform_small(seed, case["customers"]))
        init_problem(p)
        p.max_iteration, p.rnd_seed = case["iters"], seed % 100000
        return {"kind": kind, "aco": GACO(p, seed_time=SEED_TIME)}
    if kind == "solve":
        p = _one(case, seed)
        if case["limit"]:
            _limit(p)
        q = default_params(p.num_node)
        q.mode = MODE_PARITY if case["mode"] == "parity" else MODE_THROUGHPUT
        q.n_ants, q.nn_ants, q.nn_ls, q.ras_ranks = case["ants"], case["nn_ants"], case["nn_ls"], RANKS
        q.ls_flag = 3 if case["swap"] else 1
        q.seed_time, q.rnd_seed = SEED_TIME, seed % 100000
        return {"kind": kind, "solver": Solver(p, q), "iters": case["iters"]}
    if kind == "batch":
        ps = _many(case, seed)
        return {"kind": kind, "batch": Batch(ps, _batch_params(case, seed, ps)), "iters": case["iters"],
                "nodes": [p.num_node for p in ps]}
    if kind == "cold":
        ps = _many(case, seed)
        return {"kind": kind, "problems": ps, "params": _batch_params(case, seed, ps), "iters": case["iters"],
                "nodes": [p.num_node for p in ps]}
    if kind == "train":
        graphs, labels = _train_inputs(case, seed)
        scorer = learned.EdgeScorer.load()
        m, v = _train_state(seed, scorer.count)
        scorer.m.copy_(torch.from_numpy(m))
        scorer.v.copy_(torch.from_numpy(v))
        scorer.step = STEP
        return {"kind": kind, "scorer": scorer, "batch": learned.GraphBatch(graphs, labels)}
    if kind == "prior":
        return {"kind": kind, "scorer": learned.EdgeScorer.load(), "problem": _one(case, seed), "k": case["k"]}
    n, ld, A, tau, d, sol, lens = _update_inputs(case, seed)
    dev = [torch.from_numpy(a).cuda() for a in (tau, np.zeros_like(tau), d, sol, lens)]
    return {"kind": kind, "n": n, "ld": ld, "ants": A, "bufs": dev,
            "elites": torch.zeros(RANKS, dtype=torch.int32, device="cuda")}


def _padded(tours, nodes):
    """Tours end to end, each in 2n places, the room a tour of n nodes can need."""
    out = np.zeros(2 * sum(nodes), np.int32)
    at = 0
    for t, n in zip(tours, nodes):
        out[at:at + t.size] = t
        at += 2 * n
    return out


def run(state):
    kind = state["kind"]
    if kind == "driver":
        aco = state["aco"]
        aco.run()
        return {"tour": _padded([aco.instance.best_tour], [aco.instance.num_node]),
                "length": aco.instance.best_length}
    if kind in ("solve", "batch"):
        s = state["solver"] if kind == "solve" else state["batch"]
        s.init()
        s.iterate(state["iters"])
        lens = s.read_lengths(s.enqueue_lengths())
        if kind == "solve":
            tour, length = s.best()
            return {"tour": _padded([tour], [s.n]), "length": length, "lens": lens}
        tours, lengths = s.best_all()
        return {"tours": _padded(tours, state["nodes"]), "lengths": lengths, "lens": lens}
    if kind == "cold":
        with Batch(state["problems"], state["params"]) as b:
            b.init()
            b.iterate(state["iters"])
            tours, lengths = b.best_all()
        return {"tours": _padded(tours, state["nodes"]), "lengths": lengths}
    if kind == "train":
        scorer = state["scorer"]
        logits = scorer.compute_grad(state["batch"], POS_WEIGHT, sync=False)
        scorer.adam(LR)
        return {"logits": logits, "loss": scorer.loss, "grad": scorer.grad, "params": scorer.params}
    if kind == "prior":
        return state["scorer"].prior(state["problem"], k=state["k"])
    tau, total, d, sol, lens = state["bufs"]
    check(lib().aco_pheromone_update_noalloc(state["n"], state["ld"], state["ants"], RANKS, 0.1, 1.0, 2.0,
                                             tau.data_ptr(), total.data_ptr(), d.data_ptr(), sol.data_ptr(),
                                             lens.data_ptr(), state["elites"].data_ptr(),
                                             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)),
          "aco_pheromone_update_noalloc")
    return {"tau": tau, "total": total, "elites": state["elites"]}


# ---- the cost of a pass ------------------------------------------------------
def _iteration_work(n, ants, nn, parity):
    """One iteration on one instance: the matrices of the pheromone pass once, every
    ant's tour written by the construct and rewritten by the 2-opt, every step's
    row of weights (the whole row in parity mode, the candidates otherwise)."""
    steps = ants * 1.08 * n
    row = n if parity else nn
    return (16.0 * n * n + steps * (8.0 * (row if parity else 1.5 * row) + 16.0)), steps * row * 12.0 + 3.0 * n * n


def work(case):
    kind = case["kind"]
    if kind in ("driver", "solve"):
        n = case["customers"] + 1
        parity = kind == "driver" or case["mode"] == "parity"
        b, f = _iteration_work(n, n if kind == "driver" else case["ants"], 0 if parity else case["nn_ants"], parity)
        # row data stays on chip between steps of the ants: the matrices and tours are the traffic
        b = 16.0 * n * n + (n if kind == "driver" else case["ants"]) * 2.0 * n * 8.0
        return {"bytes": b * (case["iters"] + 1), "flops": f * (case["iters"] + 1)}
    if kind in ("batch", "cold"):
        lo, hi = case["n_min"], case["n_max"]
        n = (lo + hi) / 2 + 1
        n2 = (hi ** 3 - lo ** 3) / (3.0 * (hi - lo))
        ants = case["ants"] or n
        per = 16.0 * n2 + ants * 2.0 * n * 8.0
        passes = case["iters"] + 1 + (1 if kind == "cold" else 0)
        return {"bytes": case["count"] * per * passes,
                "flops": case["count"] * passes * (ants * 1.08 * n * case["nn"] * 12.0 + 3.0 * n2)}
    if kind in ("train", "prior"):
        n = case["customers"] + 1 if kind == "prior" else case["graphs"] * (case["n_min"] + case["n_max"]) / 2
        e, L, H = n * case["k"], learned.LAYERS, learned.HIDDEN
        fwd = 2.0 * e * H * H * (L + 1) + 2.0 * n * 4 * H * H * L
        if kind == "prior":
            return {"bytes": 4.0 * n * n + e * 12.0, "flops": fwd}
        # activations kept for the backward (e, q of every layer) written and read once
        return {"bytes": 4.0 * H * e * (4 * L + 2) + 4.0 * H * n * 12 * L, "flops": 3 * fwd}
    n = case["customers"] + 1
    return {"bytes": 16.0 * n * n, "flops": 6.0 * n * n}


# ---- 64-bit values -------------------------------------------------------------
def _unpack(flat, layers):
    """The packed parameters (embeddings, layers (W, b, A, a), head) by name."""
    H, F = learned.HIDDEN, learned.NODE_FEATURES
    shapes = [("W_n", (H, F)), ("b_n", (H,)), ("W_e", (H, 1)), ("b_e", (H,))]
    for l in range(layers):
        shapes += [(f"W{l}", (4 * H, H)), (f"b{l}", (4 * H,)), (f"A{l}", (H, H)), (f"a{l}", (H,))]
    shapes += [("W_h", (H, H)), ("b_h", (H,)), ("w_o", (H,)), ("b_o", (1,))]
    out, at = {}, 0
    for name, shape in shapes:
        size = math.prod(shape)
        out[name] = flat[at:at + size].view(shape)
        at += size
    return out


def _network(flat, layers, k, node_feat, edge_feat, nbr):
    """Edge logits in 64 bits."""
    H = learned.HIDDEN
    p = _unpack(flat, layers)
    n = node_feat.shape[0]
    h = node_feat @ p["W_n"].T + p["b_n"]
    e = edge_feat[:, None] * p["W_e"][:, 0] + p["b_e"]
    for l in range(layers):
        u, v, b, c = (h @ p[f"W{l}"].T + p[f"b{l}"]).split(H, dim=1)
        q = e @ p[f"A{l}"].T + p[f"a{l}"] + b.repeat_interleave(k, dim=0) + c[nbr]
        e = e + torch.relu(q)
        h = h + torch.relu(u + (torch.sigmoid(e) * v[nbr]).view(n, k, H).sum(1) / k)
    return torch.relu(e @ p["W_h"].T + p["b_h"]) @ p["w_o"] + p["b_o"]


def _weights():
    d = np.load(learned.DEFAULT_WEIGHTS)
    return d["params"], int(d["layers"])


def _exact_train(case, seed):
    graphs, labels = _train_inputs(case, seed)
    flat, layers = _weights()
    off = np.cumsum([0] + [g.n for g in graphs])
    to = lambda a: torch.from_numpy(np.asarray(a, np.float64)).cuda()  # noqa: E731
    nbr = torch.from_numpy(np.concatenate([g.nbr.astype(np.int64) + o for g, o in zip(graphs, off)])).cuda()
    w = to(flat).requires_grad_(True)
    y = to(np.concatenate(labels))
    s = _network(w, layers, case["k"], to(np.concatenate([g.node_feat for g in graphs])),
                 to(np.concatenate([g.edge_feat for g in graphs])), nbr)
    F = torch.nn.functional
    loss = (POS_WEIGHT * y * F.softplus(-s) + (1.0 - y) * F.softplus(s)).mean()
    loss.backward()
    g = w.grad
    m, v = (to(a) for a in _train_state(seed, flat.size))
    m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
    t = STEP + 1
    new = w.detach() - LR * (m / (1 - 0.9 ** t)) / (torch.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
    return {"logits": s.detach(), "loss": loss.detach().reshape(1), "grad": g, "params": new}


def _exact_prior(case, seed):
    p, k = _one(case, seed), case["k"]
    n = p.num_node
    x, y = np.asarray(p.x, np.float32), np.asarray(p.y, np.float32)
    dx, dy = x[:, None] - x[None, :], y[:, None] - y[None, :]
    d = np.sqrt(dx * dx + dy * dy)
    rank = d.copy()
    rank[:, 0] = np.inf
    rank[np.arange(n), np.arange(n)] = np.inf
    nn = np.argsort(rank, axis=1, kind="stable")[:, :k]
    side = max(float(x.max() - x.min()), float(y.max() - y.min())) or 1.0
    nf = np.zeros((n, learned.NODE_FEATURES))
    nf[:, 0], nf[:, 1] = (x - x.min()) / side, (y - y.min()) / side
    nf[:, 2] = p.demand / float(p.vehicle_capacity)
    nf[0, 3] = 1.0
    nf[:, 4] = d[:, 0] / side
    rows = np.repeat(np.arange(n), k)
    flat, layers = _weights()
    to = lambda a: torch.from_numpy(np.asarray(a, np.float64)).cuda()  # noqa: E731
    s = _network(to(flat), layers, k, to(nf), to(d[rows, nn.ravel()] / side),
                 torch.from_numpy(nn.ravel().astype(np.int64)).cuda()).cpu().numpy()
    out = np.full((n, n), 1e-3)
    out[rows, nn.ravel()] = np.maximum((1.0 / (1.0 + np.exp(-s))) ** learned.DEFAULT_GAMMA, 1e-3)
    return out


def _exact_update(case, seed):
    n, ld, A, tau, d, sol, lens = _update_inputs(case, seed)
    T = 2 * n
    t = tau.astype(np.float64)
    t[:, :n] *= 1.0 - 0.1
    elites = [A] + [int(a) for a in np.argsort(lens[:A], kind="stable")[:RANKS - 1]]
    for r, a in enumerate(elites):
        tour = sol[a * T:a * T + sol[a * T + T - 1]]
        np.add.at(t, (tour[:-1], tour[1:]), (RANKS - r) / float(lens[a]))
    total = np.zeros_like(t)
    total[:, :n] = t[:, :n] * (1.0 / (d[:, :n].astype(np.float64) + 0.1)) ** 2
    return {"tau": t, "total": total, "elites": None}


def exact(case, seed):
    """The computed numbers of a pass in 64 bits.  Tours come from a random search, so the
    colony's cases have none: their tours and lengths stand as they are."""
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] == "prior":
        return _exact_prior(case, seed)
    if case["kind"] == "update":
        return _exact_update(case, seed)
    return None
