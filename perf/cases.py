"""What this framework's users run, as cases to be timed.

A case is one call sequence through the public entry points (engine.BPGraph,
engine.BPBatch, unrolled.UnrolledBP), named by its "path":

  loopy     a resident graph solved again from its priors (beliefs in, first
            messages, loopy BP, beliefs out), node or edge schedule
  serve     a graph that arrives in pinned host memory: upload and build, a
            fixed number of iterations, beliefs back to the host
  tree      a resident tree solved again from its priors
  tree_new  a tree that arrives in device memory: build, level lists, both
            passes, beliefs out
  batch     many independent networks in one call, each with its own stop
  unrolled  one training step of unrolled BP on grids: forward, loss, both
            gradients

Inputs follow the benchmark workloads: endpoints uniform or out-degrees by a
power law, row-normalised U(0,1) tables, Dirichlet(1) priors, a share of the
nodes observed, grid potentials N(0, sigma).  They are made on the GPU.
"""
import math

import numpy as np
import torch

import belief_network_wrapper as W

from belief_propagation_b200 import native
from belief_propagation_b200.engine import BPBatch, BPGraph
from belief_propagation_b200.unrolled import UnrolledBP, nll_loss

MIXES = {"2,3,4": (2, 3, 4), "2,3,4,8": (2, 3, 4, 8)}


def listed():
    return [
        # a diagnostic network of a few dozen variables with uneven state
        # counts, solved per query: latency only
        {"name": "loopy_small_mixed", "path": "loopy", "graph": "uniform", "nodes": 61, "edges": 185,
         "states": 0, "mix": "2,3,4", "evidence": 0.1, "tol": 1e-3, "iterations": 100, "schedule": "node",
         "reorder": False},
        # the 10,000-node graph the reference's C code can run too, with its
        # own stopping rule
        {"name": "loopy_10k", "path": "loopy", "graph": "uniform", "nodes": 10_000, "edges": 40_000, "states": 2,
         "mix": "", "evidence": 0.1, "tol": 1e-3, "iterations": 100, "schedule": "node", "reorder": False},
        # the edge schedule, the reference drivers' other variant
        {"name": "loopy_edge_50k", "path": "loopy", "graph": "uniform", "nodes": 50_001, "edges": 200_003,
         "states": 3, "mix": "", "evidence": 0.1, "tol": 1e-3, "iterations": 50, "schedule": "edge",
         "reorder": False},
        # the size the network generator script writes (300,000 nodes, two
        # arcs a node, each arc an edge in both directions), four states
        {"name": "loopy_300k_s4", "path": "loopy", "graph": "uniform", "nodes": 300_000, "edges": 1_200_000,
         "states": 4, "mix": "", "evidence": 0.1, "tol": 1e-4, "iterations": 100, "schedule": "node",
         "reorder": False},
        # the large power-law graph of the headline benchmark
        {"name": "loopy_16m", "path": "loopy", "graph": "power_law", "nodes": 1 << 24, "edges": 1 << 26,
         "states": 2, "mix": "", "evidence": 0.1, "tol": 1e-3, "iterations": 100, "schedule": "node",
         "reorder": True},
        # a service that gets a new graph with every request
        {"name": "serve_1m", "path": "serve", "graph": "power_law", "nodes": 1_000_000, "edges": 4_000_000,
         "states": 2, "mix": "", "evidence": 0.1, "tol": 1e-4, "iterations": 20, "schedule": "node",
         "reorder": False},
        # exact inference on a large tree with uneven state counts
        {"name": "tree_2m", "path": "tree", "nodes": 2_000_000, "states": 0, "mix": "2,3,4,8", "evidence": 0.05},
        # a tree seen once: its build and level lists are part of the call
        {"name": "tree_new_200k", "path": "tree_new", "nodes": 200_003, "states": 0, "mix": "2,3,4,8",
         "evidence": 0.05},
        # many networks of uneven size and state count in one call
        {"name": "batch_1024", "path": "batch", "networks": 1024, "least": 32, "most": 4096, "mix": "2,3,4,8",
         "evidence": 0.1, "tol": 1e-4, "iterations": 200},
        # training a grid model: one image-sized grid
        {"name": "unrolled_512_s4", "path": "unrolled", "grids": 1, "least": 512, "most": 512, "states": 4,
         "tables": 1, "iterations": 30, "keep_every": 5, "sigma": 0.5},
        # ... a minibatch of grids of several sizes, eight states
        {"name": "unrolled_batch_s8", "path": "unrolled", "grids": 64, "least": 32, "most": 256, "states": 8,
         "tables": 1, "iterations": 20, "keep_every": 5, "sigma": 0.5},
        # ... a grid with its own tables for rows and columns, a short unroll
        {"name": "unrolled_2tables_s5", "path": "unrolled", "grids": 1, "least": 201, "most": 201, "states": 5,
         "tables": 2, "iterations": 10, "keep_every": 5, "sigma": 0.5},
    ]


def _spread(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["loopy", "loopy", "loopy", "loopy", "serve", "tree", "tree_new", "batch", "unrolled", "unrolled"])
    if path in ("loopy", "serve"):
        large = path == "loopy" and rng.random() < 0.25
        schedule = "edge" if path == "loopy" and not large and rng.random() < 0.25 else "node"
        if large:
            nodes, states, graph = _spread(rng, 1_000_000, 8_000_000), rng.randint(2, 3), "power_law"
        elif path == "serve":
            nodes, states, graph = _spread(rng, 100_000, 1_000_000), rng.randint(2, 4), "power_law"
        else:
            nodes, states, graph = _spread(rng, 12, 300_000), rng.randint(2, 5), "uniform"
        mixed = path == "loopy" and not large and schedule == "node" and rng.random() < 0.3
        return {"path": path, "graph": graph, "nodes": nodes, "edges": max(1, int(nodes * rng.uniform(2.0, 4.0))),
                "states": 0 if mixed else states, "mix": rng.choice(sorted(MIXES)) if mixed else "",
                "evidence": 0.1, "tol": rng.choice([1e-3, 1e-4]), "iterations": 20 if path == "serve" else rng.randint(20, 100),
                "schedule": schedule, "reorder": large}
    if path in ("tree", "tree_new"):
        uniform = rng.random() < 0.4
        return {"path": path, "nodes": _spread(rng, 100, 2_000_000 if path == "tree" else 200_000),
                "states": rng.randint(2, 5) if uniform else 0, "mix": "" if uniform else rng.choice(sorted(MIXES)),
                "evidence": 0.05}
    if path == "batch":
        return {"path": path, "networks": _spread(rng, 16, 1024), "least": 32, "most": _spread(rng, 64, 4096),
                "mix": rng.choice(sorted(MIXES)), "evidence": 0.1, "tol": 1e-4, "iterations": rng.randint(50, 200)}
    grids = _spread(rng, 1, 48)
    least = rng.randint(16, 64)
    return {"path": path, "grids": grids, "least": least, "most": least if grids == 1 else rng.randint(least, 200),
            "states": rng.choice([2, 3, 4, 5, 6, 8]), "tables": rng.choice([1, 1, 2]),
            "iterations": rng.randint(4, 16), "keep_every": 5, "sigma": 0.5}


# ---- inputs, on the GPU ----------------------------------------------------

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _rand(gen, *shape):
    return torch.rand(shape, generator=gen, device="cuda")


def _below(gen, n, limit):
    """n whole numbers, each uniform below `limit` (a number or a tensor)."""
    r = (torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) * limit).long()
    return torch.minimum(r, (limit if torch.is_tensor(limit) else torch.tensor(limit, device="cuda")) - 1)


def _states(gen, case, nodes):
    if not case["mix"]:
        return None, case["states"]
    choices = torch.tensor(MIXES[case["mix"]], device="cuda")
    return choices[_below(gen, nodes, len(choices))], max(MIXES[case["mix"]])


def _beliefs(gen, num_states, nodes, s, evidence):
    """Dirichlet(1) priors, some nodes observed in one of their states."""
    b = -torch.log(_rand(gen, nodes, s).clamp_min(1e-30))
    if num_states is not None:
        b = b * (torch.arange(s, device="cuda")[None] < num_states[:, None])
    b = b / b.sum(1, keepdim=True)
    seen = _rand(gen, nodes) < evidence
    state = _below(gen, nodes, torch.full((nodes,), s, device="cuda") if num_states is None else num_states)
    return torch.where(seen[:, None], torch.nn.functional.one_hot(state, s).float(), b).contiguous()


def _tables(gen, src, dst, num_states, s):
    """Row-normalised U(0,1) tables, zero beyond the two nodes' state counts."""
    t = _rand(gen, len(src), s, s)
    if num_states is not None:
        at = torch.arange(s, device="cuda")
        t = t * (at[None, :, None] < num_states[src][:, None, None]) * (at[None, None, :] < num_states[dst][:, None, None])
    return (t / t.sum(2, keepdim=True).clamp_min(1e-30)).contiguous()


def _edges(gen, case):
    """Directed edges without self-loops, grouped by source."""
    nodes, edges = case["nodes"], case["edges"]
    if case["graph"] == "power_law":  # out-degrees k with probability ~ k^-2.5, at least 1
        x_min = edges / nodes / 3.0 + 0.5
        u = torch.rand(nodes, generator=gen, device="cuda", dtype=torch.float64).clamp_min(1e-12)
        deg = (x_min * u.pow(-1.0 / 1.5)).floor().clamp(1, nodes - 1).long()
        src = torch.repeat_interleave(torch.arange(nodes, device="cuda"), deg)
        if len(src) > edges:
            src = src[torch.randperm(len(src), generator=gen, device="cuda")[:edges]]
        elif len(src) < edges:
            src = torch.cat([src, _below(gen, edges - len(src), nodes)])
    else:
        src = _below(gen, edges, nodes)
    src = src.sort().values
    dst = _below(gen, edges, nodes - 1)
    return src, dst + (dst >= src)


def _graph_inputs(case, seed):
    gen = _generator(seed)
    num_states, s = _states(gen, case, case["nodes"])
    src, dst = _edges(gen, case)
    joint = _tables(gen, src, dst, num_states, s)
    return src, dst, joint, _beliefs(gen, num_states, case["nodes"], s, case["evidence"]), num_states, s


def _tree_inputs(case, seed):
    """A random recursive tree, each child's edge in both directions with the
    table and its transpose."""
    gen = _generator(seed)
    nodes = case["nodes"]
    num_states, s = _states(gen, case, nodes)
    child = torch.arange(1, nodes, device="cuda")
    parent = _below(gen, nodes - 1, child)
    t = _tables(gen, parent, child, num_states, s)
    src = torch.stack([parent, child], 1).reshape(-1)
    dst = torch.stack([child, parent], 1).reshape(-1)
    joint = torch.stack([t, t.transpose(1, 2)], 1).reshape(-1, s, s)
    return src, dst, joint, _beliefs(gen, num_states, nodes, s, case["evidence"]), num_states, s


def _build(nodes, src, dst, joint, num_states, s, reorder=False):
    """A BPGraph of arrays in device or pinned host memory."""
    return BPGraph(nodes, src, dst, joint, num_states=num_states, uniform_states=0 if num_states is not None else s,
                   reorder=reorder)


def _networks(case, seed):
    """The batch's networks: node counts spread over their logarithm, two to
    six edges a node, one state count a network (sizes by the case, contents
    by the seed)."""
    count = case["networks"]
    rng = np.random.default_rng(count)
    nodes = np.round(np.exp(rng.uniform(np.log(case["least"]), np.log(case["most"]), count))).astype(np.int64)
    edges = np.round(rng.uniform(2.0, 6.0, count) * nodes).astype(np.int64)
    states = rng.choice(MIXES[case["mix"]], count)
    nets = [None] * count
    gen = _generator(seed)
    for s in sorted(set(states.tolist())):
        which = np.flatnonzero(states == s)
        v, e = nodes[which], edges[which]
        v_off, e_off = np.concatenate([[0], v.cumsum()]), np.concatenate([[0], e.cumsum()])
        of = torch.repeat_interleave(torch.arange(len(which), device="cuda"), torch.from_numpy(e).cuda())
        size, first = torch.from_numpy(v).cuda()[of], torch.from_numpy(v_off[:-1]).cuda()[of]
        src = (_below(gen, len(of), size) + first).sort().values - first
        dst = _below(gen, len(of), size - 1)
        dst = dst + (dst >= src)
        joint = _tables(gen, src, dst, None, s).cpu().numpy()
        beliefs = _beliefs(gen, None, int(v_off[-1]), s, case["evidence"]).cpu().numpy()
        src, dst = (x.to(torch.int32).cpu().numpy().view(np.uint32) for x in (src, dst))
        for k, n in enumerate(which):
            a, b, c, d = v_off[k], v_off[k + 1], e_off[k], e_off[k + 1]
            nets[n] = W.bp.synth.Network(np.full(b - a, s, np.uint32), beliefs[a:b], np.zeros(b - a, np.uint8),
                                         src[c:d], dst[c:d], joint[c:d], name="net%d" % n)
    return nets


def _grids(case, seed):
    """Edges of the grids' disjoint union: right and down neighbours, each pair
    in both directions; with two tables, rows use one and columns the other
    (sides by the case, potentials by the seed)."""
    rng = np.random.default_rng(case["grids"])
    sides = rng.integers(case["least"], case["most"] + 1, case["grids"])
    src, dst, table, off = [], [], [], 0
    for side in (int(x) for x in sides):
        at = (np.arange(side * side, dtype=np.int32) + off).reshape(side, side)
        a = np.concatenate([at[:, :-1].ravel(), at[:-1].ravel()])
        b = np.concatenate([at[:, 1:].ravel(), at[1:].ravel()])
        k = np.repeat(np.array([0, 1 if case["tables"] > 1 else 0], np.uint8), len(a) // 2)
        src.append(np.stack([a, b], 1).ravel())
        dst.append(np.stack([b, a], 1).ravel())
        table.append(np.stack([k, k | 0x80], 1).ravel())
        off += side * side
    src, dst, table = (np.concatenate(x) for x in (src, dst, table))
    gen = _generator(seed)
    unary = torch.randn(off, case["states"], generator=gen, device="cuda")
    pair = case["sigma"] * torch.randn(case["tables"], case["states"], case["states"], generator=gen, device="cuda")
    labels = torch.randint(0, case["states"], (off,), generator=gen, device="cuda")
    return off, src, dst, table, unary, pair, labels


def prepare(case, seed):
    path = case["path"]
    if path in ("loopy", "serve", "tree", "tree_new"):
        make = _tree_inputs if path.startswith("tree") else _graph_inputs
        src, dst, joint, prior, num_states, s = make(case, seed)
        src, dst = src.to(torch.int32), dst.to(torch.int32)
        num_states = None if num_states is None else num_states.to(torch.int32)
        out = torch.zeros_like(prior)
        torch.cuda.current_stream().synchronize()
        if path in ("loopy", "tree"):
            g = _build(case["nodes"], src, dst, joint, num_states, s, case.get("reorder", False))
            if path == "tree":
                g.tree()  # the level lists stay with the graph
            return {"case": case, "graph": g, "prior": prior, "out": out}
        arrays = (src, dst, joint, num_states, prior, out)
        if path == "serve":
            arrays = tuple(None if x is None else x.cpu().pin_memory() for x in arrays)
        return {"case": case, "arrays": arrays, "s": s}
    if path == "batch":
        batch = BPBatch(_networks(case, seed))
        return {"case": case, "batch": batch, "prior": torch.from_numpy(batch.pack_beliefs()).cuda(),
                "out": torch.zeros(int(batch.belief_off[-1]), device="cuda")}
    nodes, src, dst, table, unary, pair, labels = _grids(case, seed)
    engine = UnrolledBP(nodes, src, dst, table, states=case["states"], iterations=case["iterations"],
                        checkpoint_every=case["keep_every"], num_tables=case["tables"])
    return {"case": case, "engine": engine, "unary": unary.requires_grad_(), "pair": pair.requires_grad_(),
            "labels": labels}


def _solve(g, case, prior, out):
    g.set_beliefs(prior)
    g.latest_slot = 1
    g.init_messages()
    r = g.loopy(case["tol"], case["iterations"], schedule=case["schedule"])
    g.beliefs(out=out)
    return {"beliefs": out, "iterations": r["iterations"], "delta": r["delta"]}


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "loopy":
        return _solve(state["graph"], case, state["prior"], state["out"])
    if path == "tree":
        g = state["graph"]
        g.set_beliefs(state["prior"])
        g.tree()
        return {"beliefs": g.beliefs(out=state["out"])}
    if path in ("serve", "tree_new"):
        src, dst, joint, num_states, prior, out = state["arrays"]
        with _build(case["nodes"], src, dst, joint, num_states, state["s"]) as g:
            if path == "serve":
                return _solve(g, case, prior, out)
            g.set_beliefs(prior)
            levels = g.tree()["num_levels"]
            return {"beliefs": g.beliefs(out=out), "levels": levels}
    if path == "batch":
        b = state["batch"]
        b.set_beliefs(state["prior"])
        b.loopy(tol=case["tol"], max_iterations=case["iterations"])
        native.check(b.lib.bp_batch_get_beliefs(b.h, state["out"].data_ptr(), native.BP_MEM_DEVICE))
        r = b.results()
        return {"beliefs": state["out"], "iterations": r["iterations"].astype(np.int64), "delta": r["delta"]}
    unary, pair = state["unary"], state["pair"]
    unary.grad = pair.grad = None
    log_beliefs = state["engine"](unary, pair)
    loss = nll_loss(log_beliefs, state["labels"])
    loss.backward()
    return {"loss": loss.detach(), "log_beliefs": log_beliefs.detach(), "unary_grad": unary.grad, "pair_grad": pair.grad}


# ---- what a pass cannot do without -----------------------------------------

def work(case):
    """Loopy BP: an iteration reads each edge's table, source and old message,
    writes its new message, and reads and writes each node's belief (the next
    one needs all of it); it depends on the whole one before, so a pass is that
    many of them.  Trees: each edge's table and message once, each node's
    belief in and out.  A build adds its inputs once.  Unrolled: each node's
    state in and out an iteration, forward and backward."""
    path = case["path"]
    if path == "unrolled":
        side = (case["least"] + case["most"]) / 2
        nodes = case["grids"] * side * side
        s, t = case["states"], case["iterations"]
        edges = 4 * nodes
        return {"bytes": nodes * s * 4.0 * (4 * (t + 1) + 4 * (t + 1)),
                "flops": (t + 1) * (2 * edges * s * s + 10 * nodes * s) * 3.0}
    mean = {"": lambda p: float(case.get("states", 0)) ** p,
            "2,3,4": lambda p: (2 ** p + 3 ** p + 4 ** p) / 3,
            "2,3,4,8": lambda p: (2 ** p + 3 ** p + 4 ** p + 8 ** p) / 4}[case["mix"]]
    s = mean(1)
    if path in ("tree", "tree_new"):
        nodes, edges = case["nodes"], 2 * (case["nodes"] - 1)
        table = 4 * s * s
        once = edges * (table + 8 + 4 * s) + nodes * 8 * s
        return {"bytes": once + (edges * (table + 8) if path == "tree_new" else 0), "flops": edges * 2.0 * s * s}
    if path == "batch":
        lo, hi = math.log(case["least"]), math.log(max(case["most"], case["least"] + 1))
        nodes = case["networks"] * (math.exp(hi) - math.exp(lo)) / (hi - lo)
        edges, table = 4 * nodes, 4 * mean(2)
    else:
        nodes, edges = case["nodes"], case["edges"]
        table = 4 * (s * s if case["mix"] else mean(2))
    turn = edges * (table + 4 + 8 * s) + nodes * (4 + 8 * s)
    build = edges * (table + 8) + nodes * 8 * s if path == "serve" else 0
    return {"bytes": case["iterations"] * turn + build, "flops": case["iterations"] * edges * 2.0 * mean(2)}


# ---- the same in 64 bits ----------------------------------------------------

def _exact_loopy(case, seed):
    """Synchronous flooding: every message from the source's belief times its
    incoming messages, then every belief times its new incoming messages."""
    src, dst, joint, b, num_states, s = _graph_inputs(case, seed)
    joint, b = joint.double(), b.double()
    live = torch.ones_like(b) if num_states is None else (torch.arange(s, device="cuda")[None] < num_states[:, None]).double()

    def send(q):
        m = torch.einsum("eij,ej->ei", joint, q[src])
        total = m.sum(1, keepdim=True)
        return m / torch.where(total > 0, total, torch.ones_like(total))

    def product(m):
        return torch.ones_like(b).index_reduce_(0, dst, m, "prod") * live

    has = torch.zeros(len(b), dtype=torch.bool, device="cuda").index_fill_(0, dst, True)[:, None]
    m = send(b)
    for _ in range(case["iterations"]):
        # the product skips slots beyond a node's states: those stay zero in b
        new = send(b * torch.where(has, product(m), torch.ones_like(b)))
        delta = (m - new).abs().sum()
        m = new
        b = b * torch.where(has, product(m), torch.ones_like(b))
        total = b.sum(1, keepdim=True)
        b = b / torch.where(total > 0, total, torch.ones_like(total))
    return {"beliefs": b, "iterations": None, "delta": delta}


def _exact_unrolled(case, seed):
    nodes, src, dst, table, unary, pair, labels = _grids(case, seed)
    unary, pair = unary.double().requires_grad_(), pair.double().requires_grad_()
    src, dst = (torch.from_numpy(x.astype(np.int64)).cuda() for x in (src, dst))
    table = torch.from_numpy(table).cuda()
    groups = [(k, t, torch.nonzero(table == (k | (0x80 if t else 0))).squeeze(1)) for k in range(case["tables"]) for t in (0, 1)]
    groups = [(k, t, src[at], dst[at]) for k, t, at in groups]

    def incoming(x):
        """The sum of each node's incoming log-messages: a message depends on
        its source and its table alone."""
        e = (x - x.max(1, keepdim=True).values).exp()
        total = torch.zeros_like(x)
        for k, t, a, b in groups:
            j = pair[k].exp()
            m = e @ (j if t else j.t())
            m = m.log() - m.sum(1, keepdim=True).log()
            total = total.index_add(0, b, m[a])
        return total

    lb = torch.log_softmax(unary, 1)
    lq = lb + incoming(lb)
    for _ in range(case["iterations"]):
        lp = incoming(lq)
        lb = torch.log_softmax(lb + lp, 1)
        lq = lb + lp
    loss = torch.nn.functional.nll_loss(lb, labels)
    loss.backward()
    return {"loss": loss.detach(), "log_beliefs": lb.detach(), "unary_grad": unary.grad, "pair_grad": pair.grad}


def exact(case, seed):
    """The update multiplies each belief into itself every iteration, so a long
    loopy run amplifies rounding until 32 and 64 bits part: it has no value to
    compare with beyond 20 iterations.  Trees go by the library's level lists."""
    if case["path"] == "unrolled":
        return _exact_unrolled(case, seed)
    if case["path"] in ("loopy", "serve") and case["schedule"] == "node" and case["iterations"] <= 20:
        return _exact_loopy(case, seed)
    return None
