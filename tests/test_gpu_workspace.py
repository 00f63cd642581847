"""A graph's workspace: counted whole by stats(), and given back by close()."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

N, FAN = 100_000, [10, 10]
ITEMS = N * FAN[0]          # entries of the widest level's lists
LIST = 48 * ITEMS           # bytes of one list of items with their output slots


@pytest.fixture(scope="module")
def csaw():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("gpu test without a CUDA device")
    import csaw as c
    c.lib()
    return c


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def run(csaw, g, seeds, out, persistent):
    """One job on a graph of its own; its counted workspace and what the device
    gave for it (on the null stream, where buffers come from cudaMalloc)."""
    from csaw import _lib
    G = csaw.Graph(g)
    G.set_option(_lib.OPT_TREE, 0)
    G.set_option(_lib.OPT_PERSISTENT, persistent)
    p = csaw.make_params(0, 2, N, 1, FAN[0], len(FAN), FAN, 3, schedule=csaw.SCHED_BATCHED)
    G.sample(csaw.make_params(0, 2, 1, 1, 1, 1, [1], 3, schedule=csaw.SCHED_BATCHED), seeds[:1], out=out)   # caches
    before, counted = free_bytes(), G.stats()["workspace_bytes"]
    G.sample(p, seeds, out=out)
    taken, counted = before - free_bytes(), G.stats()["workspace_bytes"] - counted
    G.close()
    return taken, counted


@pytest.mark.parametrize("persistent", [0, 1])
def test_workspace_is_counted_and_given_back(csaw, rmat12_pareto, persistent):
    import torch
    g = rmat12_pareto
    seeds = torch.from_numpy(oracle.make_seeds(g.rowptr, N, 8)).cuda()
    out = torch.empty((4, N * 110), dtype=torch.int32, device="cuda")
    run(csaw, g, seeds, out, persistent)
    before = free_bytes()
    for _ in range(4):
        taken, counted = run(csaw, g, seeds, out, persistent)
        assert taken - counted < LIST   # some 20 buffers, each rounded up by at most 2 MiB
    assert before - free_bytes() < LIST
