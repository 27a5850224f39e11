"""The workloads this engine is timed on: whole queries, a query batch, single
products, the reference's worklist loop, the row-block closure and one
gradient of the cost model, each through the package's public entry points.

A case's "kind" says which call it makes; `listed()` gives the fixed cases,
`draw()` more of the same ranges.  Graphs, matrices and samples are made from
the seed; grammars belong to the case, since a program keeps its query while
the data changes.  One context per process, as in a program that serves
several prepared queries on one GPU.
"""
import functools
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("cfpq-on-gpgpu_b200")

MOD = 1000000007
FEATURES, HIDDEN, OUTPUTS = 16, 64, 3


@functools.lru_cache(maxsize=None)
def _context():
    return pkg.capi.Context(0)


# ---- the cases ------------------------------------------------------------

def listed():
    return [
        # the shortest whole query: launches, synchronisation and host work count
        {"name": "query_brackets_300", "kind": "query", "family": "brackets", "n": 300, "degree": 4.0,
         "edges": "host"},
        # balanced brackets on the uniform graph with 4096 edges, edges in pinned memory
        {"name": "query_brackets_1024", "kind": "query", "family": "brackets", "n": 1024, "degree": 4.0,
         "edges": "pinned"},
        # the ontology-like same-generation query (a sparse result), edges in pinned memory
        {"name": "query_ontology_8192", "kind": "query", "family": "ontology", "n": 8192, "degree": 3.0,
         "edges": "pinned"},
        # an ordinary query whose answer is dense, at a size that is no multiple of a tile
        {"name": "query_random_cnf_3001", "kind": "query", "family": "random_cnf", "n": 3001, "degree": 4.0,
         "grammar": 4, "edges": "host"},
        # a large local graph with a long and then dense closure, edges already on the GPU
        {"name": "query_chain_16384", "kind": "query", "family": "chain", "n": 16384, "degree": 2.0, "grammar": 1000004,
         "edges": "device"},
        # independent queries of mixed size and grammar closed together
        {"name": "batch_40", "kind": "batch", "count": 40, "n": 4096, "grammar": 4},
        # one dense product on the tensor cores
        {"name": "product_tc_8192", "kind": "product", "n": 8192, "variant": "tc", "halvings": 1},
        # one product with the default variant, ragged size, a thinner operand
        {"name": "product_auto_5003", "kind": "product", "n": 5003, "variant": "auto", "halvings": 3},
        # the reference's own loop: one small product at a time, the flag read after each
        {"name": "worklist_brackets_777", "kind": "worklist", "family": "brackets", "n": 777, "degree": 4.0},
        # a closure whose answer relation the program reads back as row bits
        {"name": "pairs_ontology_3001", "kind": "pairs", "family": "ontology", "n": 3001, "degree": 3.0},
        # the row-block closure, as one rank runs it (row products, deltas, block export)
        {"name": "rows_ontology_2500", "kind": "rows", "family": "ontology", "n": 2500, "degree": 3.0},
        # forward and backward of the learned selector on its logged samples
        {"name": "gradient_39685", "kind": "gradient", "samples": 39685},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# size range of a query by family (largest: the sizes of the listed cases)
SIZES = {"brackets": (256, 4096), "ontology": (1024, 8192), "random_cnf": (256, 4096), "chain": (1024, 12288)}
GRAMMARS = (1, 2, 3, 4, 5, 6, 8)  # random CNF seeds whose closure is not empty


def _draw_graph(rng, family):
    case = {"family": family, "n": _log_uniform(rng, *SIZES[family]), "degree": round(rng.uniform(2.0, 5.0), 2)}
    if family == "random_cnf":
        case["grammar"] = rng.choice(GRAMMARS)
    if family == "chain":
        case.update(degree=2.0, grammar=1000004)
    return case


def draw(rng):
    kind = rng.choice(("query", "query", "query", "batch", "product", "product", "worklist", "pairs", "rows",
                       "gradient"))
    if kind == "query":
        return {"kind": kind, **_draw_graph(rng, rng.choice(sorted(SIZES))),
                "edges": rng.choice(("host", "pinned", "device"))}
    if kind == "batch":
        return {"kind": kind, "count": _log_uniform(rng, 4, 40), "n": _log_uniform(rng, 1024, 4096),
                "grammar": rng.choice(GRAMMARS)}
    if kind == "product":
        return {"kind": kind, "n": _log_uniform(rng, 500, 8192), "variant": rng.choice(("auto", "lop3", "m4r", "tc")),
                "halvings": rng.randint(1, 8)}
    if kind == "worklist":
        return {"kind": kind, "family": "brackets", "n": _log_uniform(rng, 256, 1024),
                "degree": round(rng.uniform(2.0, 5.0), 2)}
    if kind == "pairs":
        return {"kind": kind, "family": "ontology", "n": _log_uniform(rng, 1024, 6000),
                "degree": round(rng.uniform(2.0, 4.0), 2)}
    if kind == "rows":
        return {"kind": kind, "family": "ontology", "n": _log_uniform(rng, 1000, 2500),
                "degree": round(rng.uniform(2.0, 4.0), 2)}
    return {"kind": kind, "samples": _log_uniform(rng, 1000, 39685)}


# ---- inputs ---------------------------------------------------------------

def _graph(family, n, degree, seed):
    w = pkg.workloads
    if family == "brackets":
        return w.uniform_graph(n, int(round(degree * n)), ["a", "b"], seed)
    if family == "ontology":
        return w.ontology_graph(n, seed, mean_degree=degree)
    if family == "random_cnf":
        return w.uniform_graph(n, int(round(degree * n)), [f"l{i}" for i in range(4)], seed)
    return w.chain_graph(n, degree, 0.9, 64, [f"l{i}" for i in range(6)], seed)


def _grammar(family, grammar_seed):
    w = pkg.workloads
    text = {"brackets": lambda: w.BRACKETS_GRAMMAR, "ontology": lambda: w.SAME_GENERATION_GRAMMAR,
            "random_cnf": lambda: w.random_cnf(8, 20, [f"l{i}" for i in range(4)], grammar_seed),
            "chain": lambda: w.random_cnf(10, 24, [f"l{i}" for i in range(6)], grammar_seed)}[family]()
    return pkg.query.CnfGrammar.from_text(text)


def _seed(seed, *more):
    """A generator seed from the run's seed and what it is for."""
    return int(np.random.SeedSequence((int(seed), *more)).generate_state(1)[0])


def _problem(case, seed):
    return (_grammar(case["family"], case.get("grammar", 0)),
            _graph(case["family"], case["n"], case["degree"], _seed(seed, 1)))


def _batch_shapes(case):
    """(family, n, degree) of a batch's queries: the three families in turn,
    sizes log-uniform up to case["n"] (the same for every seed: a batch's work
    belongs to the case)."""
    sizes = np.random.default_rng(case["count"])
    out = []
    for i in range(case["count"]):
        n = int(round(math.exp(sizes.uniform(math.log(256), math.log(case["n"])))))
        out.append((("brackets", "ontology", "random_cnf")[i % 3], n, float(sizes.uniform(2.0, 5.0))))
    return out


def _batch_problems(case, seed):
    return [(_grammar(family, case["grammar"]), _graph(family, n, degree, _seed(seed, 2, i)))
            for i, (family, n, degree) in enumerate(_batch_shapes(case))]


def _random_rows(n, halvings, rng):
    """Row bits of an n x n relation between the vertices that take part in
    it: three quarters of the rows and of the columns, and between those every
    bit set with probability 2^-halvings (closed relations look like this: the
    rest of the vertices reach nothing, or are not reached)."""
    words = (n + 63) // 64
    a = rng.integers(0, 2**64, (n, words), dtype=np.uint64)
    for _ in range(halvings - 1):
        a &= rng.integers(0, 2**64, (n, words), dtype=np.uint64)
    columns = np.zeros(words * 64, dtype=np.uint8)
    columns[:n] = rng.random(n) < 0.75
    a &= np.packbits(columns, bitorder="little").view(np.uint64)
    a[rng.random(n) < 0.25] = 0
    return a


def _samples(case, seed):
    """Weights, features in [0, 1], targets (log microseconds) and the mask of
    the timed variants, as the closure's product log gives them."""
    rng = np.random.default_rng(seed)
    k = case["samples"]
    dims = ((FEATURES, HIDDEN), (HIDDEN, HIDDEN), (HIDDEN, OUTPUTS))
    w = np.concatenate([np.concatenate([rng.normal(0, math.sqrt(2 / i), i * o), rng.normal(0, 0.1, o)])
                        for i, o in dims]).astype(np.float32)
    x = rng.random((k, FEATURES), dtype=np.float32)
    x[:, 14:] = 0
    y = rng.normal(3, 1, (k, OUTPUTS)).astype(np.float32)
    m = np.ones((k, OUTPUTS), dtype=np.float32)
    m[:, 2] = rng.random(k) < 0.5  # tensor cores are timed for the larger terms only
    return w, x, y, m


class _Held:
    """Device objects of one state, freed with it."""

    def __init__(self, *objects):
        self.objects = objects

    def __del__(self):
        try:
            for o in self.objects:
                (o.close if hasattr(o, "close") else o.destroy)()
        except Exception:  # the library may be gone at interpreter exit
            pass


def prepare(case, seed):
    ctx, kind = _context(), case["kind"]
    state = {"kind": kind, "ctx": ctx}
    if kind == "batch":
        state["queries"] = [pkg.query.PreparedQuery(ctx, *p) for p in _batch_problems(case, seed)]
        state["held"] = _Held(*state["queries"])
    elif kind == "product":
        rng = np.random.default_rng(seed)
        mats = [ctx.matrix(case["n"]) for _ in range(3)]
        for m in mats[1:]:
            m.upload_rows(_random_rows(case["n"], case["halvings"], rng))
        block = torch.empty(mats[0].block_bytes(0, case["n"]), dtype=torch.uint8, device="cuda")
        state.update(mats=mats, variant=case["variant"], block=block, held=_Held(*mats))
    elif kind == "gradient":
        state["args"] = _samples(case, seed)
    elif kind == "rows":
        q = pkg.query.PreparedQuery(ctx, *_problem(case, seed), order=None)
        engine = pkg.rowblock.DeviceRowEngine(ctx, q.mats)
        block = torch.empty(engine.block_bytes(0, engine.n), dtype=torch.uint8, device="cuda")
        state.update(query=q, engine=engine, block=block, held=_Held(engine, q))
    else:
        grammar, graph = _problem(case, seed)
        q = pkg.query.PreparedQuery(ctx, grammar, graph)
        state.update(query=q, held=_Held(q))
        if kind == "query":
            arrays = [torch.from_numpy(a.astype(np.uint32).view(np.int32)) for a in (graph.src, graph.label, graph.dst)]
            if case["edges"] == "device":
                arrays = [a.cuda() for a in arrays]
                edges = [a.data_ptr() for a in arrays]
            elif case["edges"] == "pinned":
                arrays = [a.pin_memory() for a in arrays]
                edges = [a.numpy().view(np.uint32) for a in arrays]
            else:
                edges = [a.numpy().view(np.uint32) for a in arrays]
            state.update(arrays=arrays, edges=edges, nedges=graph.nedges)
    torch.cuda.synchronize()
    return state


# ---- one pass -------------------------------------------------------------

def _lines(pairs):
    """The answer lines (hash, count), one row per nonterminal."""
    return np.asarray(pairs, dtype=np.int64).reshape(-1, 2)


def run(state):
    ctx, kind = state["ctx"], state["kind"]
    if kind == "query":
        q = state["query"]
        _, lines = ctx.intersection(q.grammar.rules, q.mats, *state["edges"], q.off, q.lm, q.grammar.epsilon,
                                    nedges=state["nedges"])
        return _lines(lines)
    if kind == "batch":
        qs = state["queries"]
        for q in qs:
            q.load()
        ctx.closure_batch([(q.grammar.rules, q.mats) for q in qs])
        return _lines(ctx.hash_count_many([m for q in qs for m in q.mats]))
    if kind == "product":
        c, a, b = state["mats"]
        c.clear()
        changed = ctx.add_mul(c, a, b, state["variant"])
        c.export_block(0, c.n, state["block"].data_ptr())
        return {"changed": changed, "block": state["block"]}
    if kind == "worklist":
        q = state["query"]
        res = q.run(driver="worklist")
        return _lines([res.lines[name] for name in q.grammar.nonterminals])
    if kind == "pairs":
        q = state["query"]
        res = q.run()
        return {"lines": _lines([res.lines[name] for name in q.grammar.nonterminals]),
                "relation": q.mats[0].download_rows().view(np.int64)}
    if kind == "rows":
        q, engine = state["query"], state["engine"]
        q.load()
        ctx.clear_many(engine.prev + engine.delta)
        pkg.rowblock.closure(engine, q.grammar.rules)
        engine.export(0, 0, engine.n, state["block"])
        return {"lines": _lines(ctx.hash_count_many(q.mats)), "block": state["block"]}
    loss, grad = ctx.selector_loss_grad(*state["args"])
    return {"loss": loss, "grad": grad}


def work(case):
    kind = case["kind"]
    if kind == "gradient":
        weights = FEATURES * HIDDEN + HIDDEN * HIDDEN + HIDDEN * OUTPUTS
        return {"bytes": 4 * case["samples"] * (FEATURES + 2 * OUTPUTS) + 8 * weights,
                "flops": 6 * case["samples"] * weights}
    if kind == "product":
        n, tiles = case["n"], (case["n"] + 63) // 64
        return {"bytes": 2 * n * n // 8 + tiles * tiles * 516, "flops": 2 * n**3}
    problems = _batch_shapes(case) if kind == "batch" else [(case["family"], case["n"], case["degree"])]
    total = {"bytes": 0, "flops": 0}
    for family, n, degree in problems:
        nonterminals, rules = {"brackets": (4, 3), "ontology": (7, 6), "random_cnf": (8, 20), "chain": (10, 24)}[family]
        edges = n * degree * (2 if family == "ontology" else 1)
        if family == "ontology":  # a sparse answer: about 30 tiles of 64 x 64 bits per tile row
            total["bytes"] += 12 * edges + 30 * (n / 64) * 512
            total["flops"] += 2 * rules * 30 * (n / 64) * 64**3
        elif family == "brackets":  # one dense relation and its helper, thin operands
            total["bytes"] += 12 * edges + 2 * n * n / 8
            total["flops"] += 2 * rules * n * n * degree
        else:
            total["bytes"] += 12 * edges + nonterminals * n * n / 8
            total["flops"] += 2 * rules * n**3
    if kind == "pairs":
        total["bytes"] += case["n"] ** 2 / 8
    return total


# ---- the same results by plain torch -----------------------------------------

def _fixpoint(grammar, graph):
    """The least fixpoint as 0/1 matrices: sums of at most n ones are compared
    with zero only, so half precision products are exact."""
    n, dev = graph.n, "cuda"
    off, mats = pkg.query.label_map(grammar, graph)
    m = [torch.zeros(n, n, dtype=torch.float16, device=dev) for _ in grammar.nonterminals]
    src, lab, dst = (torch.from_numpy(a.astype(np.int64)).to(dev) for a in (graph.src, graph.label, graph.dst))
    for label in range(len(graph.labels)):
        for x in mats[off[label]:off[label + 1]]:
            m[x][src[lab == label], dst[lab == label]] = 1
    for x in grammar.epsilon:
        m[x].fill_diagonal_(1)
    changed = True
    while changed:
        changed = False
        for head, body1, body2 in grammar.rules:
            new = torch.where(m[body1] @ m[body2] > 0, 1, m[head])
            if not torch.equal(new, m[head]):
                m[head], changed = new, True
    return m


def _exact_lines(mats):
    """Sum of 11^(n-1-c) * 13^(n-1-r) modulo p over the set bits (r, c), and their count."""
    out = []
    for m in mats:
        n = m.shape[0]
        p11, p13 = (torch.tensor([pow(base, n - 1 - i, MOD) for i in range(n)], dtype=torch.float64) for base in (11, 13))
        rows = torch.cat([part.double() @ p11.to(m.device) for part in m.split(2048)]).cpu().to(torch.int64) % MOD
        h = int((rows * p13.to(torch.int64) % MOD).sum()) % MOD
        out.append((h, int(m.sum(dtype=torch.float64))))
    return _lines(out)


def _packed(bits):
    """Last dimension of 0/1 values packed into bytes, bit i of a byte its value i."""
    return (bits.view(*bits.shape[:-1], -1, 8).to(torch.uint8) << torch.arange(8, device=bits.device,
                                                                              dtype=torch.uint8)).sum(-1, dtype=torch.uint8)


def _exact_block(m):
    """A whole matrix as an exported row block: 64 x 64-bit tiles, occupancy words, tile populations."""
    n = m.shape[0]
    t = (n + 63) // 64
    full = torch.zeros(t * 64, t * 64, dtype=torch.uint8, device=m.device)
    full[:n, :n] = m > 0
    tiles = full.view(t, 64, t, 64).permute(0, 2, 1, 3).contiguous()
    count = tiles.sum((2, 3), dtype=torch.int32)
    occ = torch.zeros(t, (t + 31) // 32 * 32, dtype=torch.uint8, device=m.device)
    occ[:, :t] = count > 0
    return torch.cat([_packed(tiles).reshape(-1), _packed(occ).reshape(-1), count.view(torch.uint8).reshape(-1)])


def _unpacked(rows, n):
    return torch.from_numpy(np.unpackbits(rows.view(np.uint8), axis=1, bitorder="little")[:, :n]).to("cuda",
                                                                                                     torch.float16)


def exact(case, seed):
    kind = case["kind"]
    if kind == "gradient":
        w, x, y, m = (torch.from_numpy(a).double() for a in _samples(case, seed))
        w.requires_grad_()
        h, at = x, 0
        for i, o in ((FEATURES, HIDDEN), (HIDDEN, HIDDEN), (HIDDEN, OUTPUTS)):
            h = h @ w[at:at + i * o].view(i, o) + w[at + i * o:at + i * o + o]
            at += i * o + o
            h = h.relu() if o == HIDDEN else h
        loss = (m * (h - y) ** 2).sum() / (2 * m.sum())
        loss.backward()
        return {"loss": float(loss), "grad": w.grad.numpy()}
    if kind == "product":
        rng = np.random.default_rng(seed)
        a, b = (_unpacked(_random_rows(case["n"], case["halvings"], rng), case["n"]) for _ in range(2))
        c = a @ b > 0
        return {"changed": bool(c.any()), "block": _exact_block(c)}
    if kind == "batch":
        return np.concatenate([_exact_lines(_fixpoint(*p)) for p in _batch_problems(case, seed)])
    m = _fixpoint(*_problem(case, seed))
    lines = _exact_lines(m)
    if kind == "pairs":
        n = case["n"]
        bits = torch.zeros(n, (n + 63) // 64 * 64, dtype=torch.uint8, device="cuda")
        bits[:, :n] = m[0] > 0
        return {"lines": lines, "relation": _packed(bits).cpu().numpy().view(np.int64)}
    if kind == "rows":
        return {"lines": lines, "block": _exact_block(m[0])}
    return lines
