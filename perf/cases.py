"""The work this engine is measured on: twelve cases through its public entry
points, and draw() for more cases of the same ranges.

A case names a graph (what a program keeps resident: a handle is made once and
shared by every state of the process), the sampling job, and the entry point
that runs it.  A state's own inputs -- seed vertices, the Philox key, output
buffers -- come from the seed.  Graphs and sizes are those of the benchmark
and the tests: R-MAT 16 symmetrised, the 875,713-vertex power-law graph, R-MAT
22 (serving), R-MAT 24 (streaming) and R-MAT 25 heavy-tailed (the headline
step).
"""
import collections
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "c-saw_b200"))

import csaw  # noqa: E402
from csaw import graphgen  # noqa: E402

SCHEDULES = {"plain": csaw.SCHED_PLAIN, "batched": csaw.SCHED_BATCHED}


def listed():
    return [
        # smallest call: the small symmetrised R-MAT, default (plain) schedule
        dict(name="small_plain", kind="neighbor", graph="rmat", scale=16, bias="unbiased", schedule="plain",
             n=1000, frontier=1, fanout="2,2", depth_out=True, dedup=False),
        # the smallest request of the serving mix: 64 seeds, 2 hops
        dict(name="request_64", kind="neighbor", graph="rmat", scale=22, bias="weight", schedule="batched",
             n=64, frontier=1, fanout="25,10", depth_out=True, dedup=False),
        # the latency-target request: 1024 seeds, 2 hops
        dict(name="request_1024", kind="neighbor", graph="rmat", scale=22, bias="weight", schedule="batched",
             n=1024, frontier=1, fanout="25,10", depth_out=True, dedup=False),
        # the largest request of the serving mix: 8192 seeds, 3 hops
        dict(name="request_8192", kind="neighbor", graph="rmat", scale=22, bias="weight", schedule="batched",
             n=8192, frontier=1, fanout="15,10,5", depth_out=True, dedup=False),
        # a GNN mini-batch: unbiased fan-out, a ragged number of seeds
        dict(name="minibatch", kind="neighbor", graph="powerlaw", scale=0, bias="unbiased", schedule="batched",
             n=3001, frontier=1, fanout="15,10", depth_out=True, dedup=False),
        # subgraph extraction on the mid-size power-law graph
        dict(name="powerlaw_neighbor", kind="neighbor", graph="powerlaw", scale=0, bias="degree", schedule="batched",
             n=4000, frontier=4, fanout="20,20,20", depth_out=True, dedup=False),
        # few long walks: a latency chain
        dict(name="powerlaw_walk", kind="walk", graph="powerlaw", scale=0, bias="degree", schedule="batched",
             n=4000, length=64, depth_out=True),
        # an unbiased walk corpus (DeepWalk)
        dict(name="walk_corpus", kind="walk", graph="rmat", scale=22, bias="unbiased", schedule="batched",
             n=262144, length=40, depth_out=True),
        # multi-dimensional random walk, the reference's dispatch for FrontierSize > 1
        dict(name="mdrw", kind="mdrw", graph="powerlaw", scale=0, bias="degree", schedule="batched",
             n=4000, frontier=4, length=3, depth_out=True),
        # the headline step: neighbor samples and walks as one batch, int64 row offsets
        dict(name="headline", kind="batch", graph="heavy", scale=25, bias="weight", schedule="batched",
             n=65536, frontier=8, fanout="10,10,10", walks=1048576, length=40, depth_out=False),
        # the request loop: a burst of mixed requests, host buffers in and out
        dict(name="serve_burst", kind="serve", graph="rmat", scale=22, bias="weight", schedule="batched",
             requests=32, slots=8, depth_out=True),
        # a graph above the device budget: its adjacency stays in host memory
        dict(name="streaming", kind="stream", graph="rmat", scale=24, bias="weight", schedule="batched",
             n=32768, frontier=1, fanout="10,10", walks=131072, length=20, partition_bits=16, budget=1 << 30,
             depth_out=True),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["neighbor", "neighbor", "neighbor", "walk", "walk", "mdrw", "batch", "serve", "stream"])
    graph, scale = rng.choice([("rmat", 16), ("rmat", 18), ("rmat", 20), ("rmat", 22), ("powerlaw", 0),
                               ("heavy", 20), ("heavy", 22)])
    bias = rng.choice(["unbiased", "degree", "weight", "weight"])
    schedule = "batched"
    if kind in ("neighbor", "walk") and (graph == "powerlaw" or scale <= 16) and rng.random() < 0.4:
        schedule = "plain"   # the default; it rescans a row for every draw, so it runs on graphs without large hubs
    c = dict(kind=kind, graph=graph, scale=scale, bias=bias, schedule=schedule, depth_out=rng.random() < 0.7)
    if kind in ("neighbor", "batch"):
        c["frontier"] = rng.choice([1, 1, 1, 2, 4, 8])
        hops = rng.choice([1, 2, 2, 3, 3])
        fan, width = [], c["frontier"]
        for _ in range(hops):
            k = rng.randint(1, min(32, max(2, 6000 // width)))
            fan.append(k)
            width *= k
        c["fanout"] = ",".join(map(str, fan))
        c["n"] = _log(rng, 1, max(2, min(16384, 12_000_000 // width)))
        if kind == "neighbor":
            c["dedup"] = rng.random() < 0.15
    if kind in ("walk", "batch"):
        c["length"] = _log(rng, 3, 100)
        c["n" if kind == "walk" else "walks"] = _log(rng, 1, max(2, min(300_000, 12_000_000 // c["length"])))
    if kind == "mdrw":
        c["bias"] = rng.choice(["unbiased", "degree"])
        c["frontier"], c["length"], c["n"] = _log(rng, 2, 200), _log(rng, 1, 64), _log(rng, 16, 16000)
    if kind == "serve":
        c["bias"], c["requests"], c["slots"] = "weight", _log(rng, 1, 96), rng.choice([4, 8, 16])
    if kind == "stream":
        c["graph"], c["scale"] = "rmat", rng.choice([18, 20, 22])
        c.update(frontier=1, fanout=rng.choice(["10,10", "5,5", "25", "7,3,2"]), n=_log(rng, 64, 32768),
                 length=_log(rng, 2, 40), walks=_log(rng, 64, 131072), partition_bits=c["scale"] - 8,
                 budget=(1 << c["scale"]) * 32)
    return c


# ------------------------------------------------------------------ graphs
# A program makes a handle once and keeps it; the eight used last are kept.
_HANDLES = collections.OrderedDict()
_KEPT = 8


def _csr(graph, scale):
    if graph == "powerlaw":
        return graphgen.powerlaw_directed()
    if graph == "heavy":
        return graphgen.rmat_device(scale, 16, 0.6, 0.2, 0.15, seed=25, symmetrize=False, weight="pareto:1.5")
    small = scale <= 18
    return graphgen.rmat_device(scale, 8 if small else 16, seed=scale, symmetrize=small, weight="uniform")


def _handle(kind, *key):
    key = (kind,) + key
    if key in _HANDLES:
        _HANDLES.move_to_end(key)
        return _HANDLES[key]
    while len(_HANDLES) >= _KEPT:
        for h in reversed(_HANDLES.popitem(last=False)[1]):
            h.close()
    csr = _csr(*key[1:3])
    torch.cuda.empty_cache()
    if kind == "stream":
        g = csaw.StreamGraph(csr, partition_bits=key[3], slot_budget_bytes=key[4])
        if key[5] != "unbiased":
            g.cache(key[5])
        made = (g,)
    else:
        g = csaw.Graph(csr, rowptr64=True if key[1] == "heavy" else None)
        made = (g,)
        if kind == "serve":
            made = (g, csaw.Server(g, n_slots=key[3], device_budget=1 << 30))
    _HANDLES[key] = made
    return made


# ------------------------------------------------------------------- states
def _fanout(case):
    return [int(k) for k in case["fanout"].split(",")]


def _neighbor(case, seed, schedule):
    fan = _fanout(case)
    return csaw.make_params("neighbor", case["bias"], case["n"], case["frontier"], fan[0], len(fan), fan, seed=seed,
                            schedule=schedule, dedup=case.get("dedup", False))


def _walk(case, n, seed, schedule):
    return csaw.make_params("walk", case["bias"], n, 1, 1, case["length"], seed=seed, schedule=schedule)


def _requests(case, seed):
    """The serving mix: 2-hop [25,10], 3-hop [15,10,5] and walks of 10-80
    steps, seeds per request lognormal around 512 clipped to 64-8192.  The
    mix belongs to the case, its draws to the seed."""
    rng = torch.Generator()
    rng.manual_seed(case["requests"])
    out = []
    for k in range(case["requests"]):
        n = int(min(8192, max(64, 512 * torch.exp(torch.randn((), generator=rng)).item())))
        what, length = (int(x) for x in torch.randint(0, 71, (2,), generator=rng))
        if what % 3 == 2:
            p = csaw.make_params("walk", "weight", n, 1, 1, 10 + length, seed=seed + k, schedule=csaw.SCHED_BATCHED)
        else:
            fan = [25, 10] if what % 3 == 0 else [15, 10, 5]
            p = csaw.make_params("neighbor", "weight", n, 1, fan[0], len(fan), fan, seed=seed + k,
                                 schedule=csaw.SCHED_BATCHED)
        out.append(p)
    return out


def prepare(case, seed):
    kind, graph, scale = case["kind"], case["graph"], case["scale"]
    sched, wd = SCHEDULES[case["schedule"]], case["depth_out"]
    rows = 3 + wd

    def outputs(p):
        return torch.empty((rows, max(1, csaw.edge_bound(p))), dtype=torch.int32, device="cuda")

    if kind == "serve":
        g, server = _handle("serve", graph, scale, case["slots"])
        plist = _requests(case, seed)
        seeds = [_make_seeds(graph, scale, p.n_samples, seed + 77 * k) for k, p in enumerate(plist)]
        bufs = [torch.empty((rows, max(1, csaw.edge_bound(p))), dtype=torch.int32, pin_memory=True) for p in plist]
        return dict(kind=kind, server=server, jobs=list(zip(plist, seeds, bufs)), depth=wd)
    if kind == "stream":
        (g,) = _handle("stream", graph, scale, case["partition_bits"], case["budget"], case["bias"])
        p, w = _neighbor(case, seed, sched), _walk(case, case["walks"], seed + 1, sched)
        jobs = []
        for q, k in ((w, 3), (p, 5)):
            s = torch.from_numpy(_make_seeds(graph, scale, q.n_samples * q.frontier_size, seed + k, g.csr)).cuda()
            jobs.append((q, s, outputs(q)))
        return dict(kind=kind, g=g, jobs=jobs, depth=wd)
    (g,) = _handle("graph", graph, scale)
    if kind == "batch":
        jobs = []
        for q in (_neighbor(case, seed, sched), _walk(case, case["walks"], seed + 1, sched)):
            s = g.make_seeds(q.n_samples * q.frontier_size, q.seed + 5)
            jobs.append(csaw.BatchJob(q, s, out=outputs(q), with_depth=wd))
        return dict(kind=kind, g=g, jobs=jobs)
    if kind == "neighbor":
        p = _neighbor(case, seed, sched)
    elif kind == "walk":
        p = _walk(case, case["n"], seed, sched)
    else:
        p = csaw.make_params("mdrw", case["bias"], case["n"], case["frontier"], 1, case["length"], seed=seed,
                             schedule=sched)
    return dict(kind=kind, g=g, p=p, seeds=g.make_seeds(p.n_samples * p.frontier_size, seed + 5), out=outputs(p),
                depth=wd)


def _make_seeds(graph, scale, n, seed, csr=None):
    """Host seed vertices, uniform over the vertices that have an edge."""
    if csr is None:
        csr = next(h[0].csr for k, h in _HANDLES.items() if k[1:3] == (graph, scale))
    if not hasattr(csr, "connected"):
        csr.connected = torch.nonzero(torch.from_numpy(csr.degrees()) > 0).flatten().to(torch.int32)
    rng = torch.Generator()
    rng.manual_seed(seed)
    return csr.connected[torch.randint(0, csr.connected.numel(), (n,), generator=rng)].numpy()


class EdgeList(dict):
    """The columns of a sampled edge list.  The engine leaves the order of an
    edge list open (its contract is the multiset), so a column is read in one
    order -- by sample, depth, source, destination -- and filled up with -1 to
    the job's edge bound (the length of the caller's buffers)."""

    def __init__(self, columns, bound):
        src, dst, sample, depth = columns
        super().__init__(src=src, dst=dst, sample=sample)
        if depth is not None:
            self["depth"] = depth
        self._bound, self._order = bound, None

    def __getitem__(self, name):
        get = super().__getitem__
        if self._order is None:
            c = {k: torch.as_tensor(get(k)).cuda().long() for k in self}
            o = torch.sort((c["src"] << 32) | c["dst"]).indices
            key = (c["sample"] << 32) | c["depth"] if "depth" in c else c["sample"]
            self._order = o[torch.sort(key[o], stable=True).indices]
        out = torch.full((self._bound,), -1, dtype=torch.int32, device="cuda")
        out[:self._order.numel()] = torch.as_tensor(get(name)).cuda()[self._order]
        return out


class Burst(dict):
    """The edge lists of a burst of requests, end to end, when they are read."""

    def __init__(self, lists):
        super().__init__({k: lists for k in lists[0]})

    def __getitem__(self, name):
        return torch.cat([e[name] for e in super().__getitem__(name)])


def run(state):
    kind = state["kind"]
    if kind == "batch":
        jobs = state["jobs"]
        return [EdgeList(e, j.capacity) for e, j in zip(state["g"].sample_batch(jobs), jobs)]
    if kind == "serve":
        server, jobs = state["server"], state["jobs"]
        tickets = [server.submit(p, s, out=b, with_depth=state["depth"]) for p, s, b in jobs]
        return Burst([EdgeList(server.wait(t)[2], b.shape[1]) for t, (_, _, b) in zip(tickets, jobs)])
    if kind == "stream":
        return [EdgeList(state["g"].sample(p, s, out=o, with_depth=state["depth"]), o.shape[1])
                for p, s, o in state["jobs"]]
    out = state["out"]
    return EdgeList(state["g"].sample(state["p"], state["seeds"], out=out, with_depth=state["depth"]), out.shape[1])


def exact(case, seed):
    """Every output is whole numbers: there is no rounding to measure."""
    return None


# Mean edges per expanded vertex over its fan-out k, measured on each graph:
# shares of k at the seeds and at later hops (a later hop meets higher
# degrees), at most `most`; and the share of a walk's steps before it ends.
FILL = {"rmat": (0.45, 0.86, 32.0, 0.88), "heavy": (0.45, 0.92, 32.0, 0.61), "powerlaw": (1.0, 1.0, 4.0, 1.0)}


def work(case):
    """One pass: each output edge written once, its column and (biased) one
    prefix or weight entry read once, and the row range of each expanded
    vertex."""
    first, later, most, alive = FILL[case["graph"]]
    if case["graph"] == "rmat" and case["scale"] <= 18:   # symmetrised
        first = later = 0.94

    def neighbor(width, fan):
        edges = items = 0.0
        for hop, k in enumerate(fan):
            items += width
            width *= min(most, k * (later if hop else first))
            edges += width
        return edges, items

    def walk(n, length):
        return n * length * alive, n * length * alive

    jobs = []
    if "fanout" in case:
        jobs.append(neighbor(case["n"] * case["frontier"], _fanout(case)))
    if case["kind"] in ("walk", "mdrw", "batch", "stream"):
        jobs.append(walk(case.get("walks", case["n"]), case["length"]))
    if case["kind"] == "serve":
        for p in _requests(case, 0):
            if p.mode == csaw.MODE_WALK:
                jobs.append(walk(p.n_samples, p.depth))
            else:
                jobs.append(neighbor(p.n_samples, [p.fanout[i] for i in range(p.depth)]))
    edges, items = (sum(x) for x in zip(*jobs))
    row = 2 * (8 if case["graph"] == "heavy" else 4)
    per_edge = 4 * (3 + case["depth_out"]) + 4 + (4 if case["bias"] != "unbiased" else 0)
    return {"bytes": edges * per_edge + items * row, "flops": 0}
