"""The group pass (32 / N items per warp over a cached prefix) and its prefix
search at the sizes where they can go wrong: rows around the 32-edge tile,
the 1024-edge group and the 512-edge refill bound, at every offset of a row
in its tile, one to sixteen slots (32 to two items a warp), rows without
mass and rows whose mass sits on one neighbor (every slot collides).  The
edges are compared with the oracle's, exactly."""
import numpy as np
import pytest

import oracle
from conftest import sort_edges

pytestmark = pytest.mark.gpu

DEGREES = [3, 9, 30, 31, 32, 33, 48, 63, 64, 65, 96, 255, 511, 512, 513, 991, 1023, 1024, 1025, 1056, 2047, 2049, 33_000]


@pytest.fixture(scope="module")
def csaw():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("gpu test without a CUDA device")
    import csaw as c
    c.lib()
    return c


@pytest.fixture(scope="module")
def rows_graph():
    """Three rows of every degree (uniform, heavy-tailed and one-neighbor
    weights), each shifted in its tile by the rows before it, and a row of
    zero weights."""
    from csaw import graphgen
    V = 40_000
    rng = np.random.default_rng(3)
    deg = np.zeros(V, dtype=np.int64)
    weights, cols = [], []
    v = 0
    for d in DEGREES:
        for kind in range(4 if d == 64 else 3):
            w = [rng.random(d) + 1e-3, 1 + rng.pareto(1.1, d), np.full(d, 1e-6), np.zeros(d)][kind].astype(np.float32)
            if kind == 2:
                w[rng.integers(d)] = 1e6
            deg[v] = d
            cols.append(np.sort(rng.choice(V, d, replace=False)))
            weights.append(w)
            v += 1
    hubs = v
    deg[hubs:] = rng.integers(0, 6, V - hubs)
    rest = int(deg[hubs:].sum())
    cols.append(rng.integers(0, hubs, rest))   # later hops come back to the rows
    weights.append((rng.random(rest) + 1e-3).astype(np.float32))
    rowptr = np.concatenate([[0], np.cumsum(deg)])
    return graphgen.CSR(rowptr, np.concatenate(cols), np.concatenate(weights), name="rows"), hubs


@pytest.mark.parametrize("rowptr64", [False, True])
@pytest.mark.parametrize("bias", [1, 2])
@pytest.mark.parametrize("n_slots", [1, 2, 3, 5, 7, 10, 11, 16])
def test_group_pass_equals_oracle(csaw, rows_graph, rowptr64, bias, n_slots):
    import torch
    from csaw import _lib
    g, hubs = rows_graph
    G = csaw.Graph(g, rowptr64=rowptr64)
    G.set_option(_lib.OPT_GRID_PCT, 200)   # a launch shape of the per-level passes
    G.set_option(_lib.OPT_THREAD_SELECT, 0)
    n, seed = hubs * 9 + 1, 0x61 + n_slots
    seeds = (np.arange(n) % hubs).astype(np.int32)
    fan = [n_slots, 2]
    p = csaw.make_params(0, bias, n, 1, fan[0], 2, fan, seed, schedule=csaw.SCHED_BATCHED)
    G.profile(True)
    out = [x.cpu().numpy() for x in G.sample(p, torch.from_numpy(seeds).cuda())]
    assert G.kernel_stats("pair")["items"] > 0
    G.close()
    ref = oracle.run(g.rowptr, g.col, g.weight, seeds, 0, bias, n, 1, 2, fan, seed=seed, n_threads=8)
    a, b = sort_edges(*out), sort_edges(*ref)
    assert a.shape == b.shape and np.array_equal(a, b)


@pytest.mark.parametrize("rowptr64", [False, True])
@pytest.mark.parametrize("bias", [1, 2])
def test_rows_read_in_place_equal_oracle(csaw, rows_graph, rowptr64, bias):
    """The same rows from a streaming graph: the first job finds no partition on
    the device and reads the page-locked host prefix sector by sector, the
    second reads the partitions' device copies."""
    import torch
    g, hubs = rows_graph
    G = csaw.StreamGraph(g, partition_bits=6, slot_budget_bytes=16 * int(g.rowptr[hubs]), rowptr64=rowptr64)
    G.cache(bias)
    n = hubs * 5 + 3
    seeds = (np.arange(n) % hubs).astype(np.int32)
    for mode, fan, depth in ((0, [7, 2], 2), (1, None, 12), (0, [7, 2], 2), (1, None, 12)):
        p = csaw.make_params(mode, bias, n, 1, (fan or [1])[0], depth, fan, 77)
        out = [x.cpu().numpy() for x in G.sample(p, torch.from_numpy(seeds).cuda())]
        ref = oracle.run(g.rowptr, g.col, g.weight, seeds, mode, bias, n, 1, depth, fan, seed=77, n_threads=8)
        a, b = sort_edges(*out), sort_edges(*ref)
        assert a.shape == b.shape and np.array_equal(a, b), (mode, depth)
    assert G.info()["items_read_in_place"] > 0
    G.close()
