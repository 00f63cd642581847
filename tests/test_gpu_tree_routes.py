"""Both routes of neighbor jobs that either may take: whole sample trees in one
launch and the per-level launches, named by CSAW_OPT_TREE and seen in the
launches by kind.  What the one-launch route took over by default is run here
by the per-level launches too: plain unbiased levels, hubs that go on from
their failed first phase with and without incremental rebuilds.  Edges equal
the oracle's exactly."""
import numpy as np
import pytest

import oracle
from conftest import sort_edges
from test_gpu_incr_rebuild import make_concentrated_hubs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def csaw():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("gpu test without a CUDA device")
    import csaw as c
    c.lib()
    return c


@pytest.fixture(scope="module")
def concentrated():
    return make_concentrated_hubs()


def run(G, p, seeds):
    import torch
    G.profile(True)
    out = [x.cpu().numpy() for x in G.sample(p, torch.from_numpy(seeds).cuda())]
    kinds = {k: G.kernel_stats(k) for k in ("tree", "expand", "heavy", "pair")}
    G.profile(False)
    return sort_edges(*out), kinds


def expected(g, seeds, bias, n, F, fan, seed):
    return sort_edges(*oracle.run(g.rowptr, g.col, g.weight, seeds, 0, bias, n, F, len(fan), fan, seed=seed, n_threads=8))


@pytest.mark.parametrize("rowptr64", [False, True])
@pytest.mark.parametrize("bias,schedule", [(0, 0), (0, 1), (1, 1), (2, 2), (3, 1)])
def test_both_routes_equal_oracle(csaw, skewed_hubs, rowptr64, bias, schedule):
    from csaw import _lib
    g = skewed_hubs
    G = csaw.Graph(g, rowptr64=rowptr64)
    hubs = np.argsort(np.diff(g.rowptr))[-12:].astype(np.int32)
    for k, (n, F, fan) in enumerate([(1, 12, [16, 3]), (97, 1, [32, 7]), (31, 5, [2, 17, 2])]):
        seeds = np.concatenate([hubs, oracle.make_seeds(g.rowptr, n * F, 5 + k)])[: n * F].astype(np.int32)
        p = csaw.make_params(0, bias, n, F, fan[0], len(fan), fan, 0xB0 + k, schedule=schedule)
        ref = expected(g, seeds, bias, n, F, fan, 0xB0 + k)
        for tree in (2, 0):
            G.set_option(_lib.OPT_TREE, tree)
            got, kinds = run(G, p, seeds)
            assert kinds["tree"]["launches"] == (tree != 0), (n, F, fan, tree)
            assert (kinds["expand"]["launches"] > 0) == (tree == 0), (n, F, fan, tree)
            assert got.shape == ref.shape and np.array_equal(got, ref), (n, F, fan, tree)
    G.close()


@pytest.mark.parametrize("rowptr64", [False, True])
@pytest.mark.parametrize("bias,fan", [(2, [10, 4]), (2, [16, 2]), (2, [6, 6]), (1, [12, 3]), (3, [12, 3])])
def test_hub_resume_by_both_routes(csaw, concentrated, rowptr64, bias, fan):
    """Hubs whose first phase fails: resumed by the CTA pass from the group
    pass's state (per-level launches) and redone by the chunk's CTA (one
    launch), with and without the tile summaries."""
    from csaw import _lib
    g, hubs = concentrated
    n, F, seed = 600, 2, 0x3C0 + fan[0]
    seeds = np.concatenate([np.tile(hubs.astype(np.int32), n // hubs.size + 1)[:n],
                            oracle.make_seeds(g.rowptr, n * F - n, 0x3C)]).astype(np.int32)
    ref = expected(g, seeds, bias, n, F, fan, seed)
    G = csaw.Graph(g, rowptr64=rowptr64)
    p = csaw.make_params(0, bias, n, F, fan[0], len(fan), fan, seed, schedule=csaw.SCHED_BATCHED)
    heavy = set()
    for tree in (0, 2):
        G.set_option(_lib.OPT_TREE, tree)
        for incr in (1, 0):
            G.set_option(_lib.OPT_INCR_REBUILD, incr)
            got, kinds = run(G, p, seeds)
            assert kinds["tree"]["launches"] == (tree != 0)
            assert (kinds["pair"]["items"] > 0) == (tree == 0)
            heavy.add(kinds["heavy"]["items"])
            assert got.shape == ref.shape and np.array_equal(got, ref), (tree, incr)
    assert len(heavy) == 1 and heavy.pop() > 0   # the same hubs by either route
    G.close()


def test_tree_option_range(csaw, powerlaw_small):
    from csaw import _lib
    G = csaw.Graph(powerlaw_small)
    for bad in (-1, 3):
        with pytest.raises(csaw.CsawError, match="tree"):
            G.set_option(_lib.OPT_TREE, bad)
    G.close()


def test_unbiased_walks_take_columns(csaw):
    """The rule that reads columns and row offsets (records above the L2 size,
    offsets below half of it, many walks) is seen in the counted bytes of a
    step: two 8-byte offsets where a record counts 12."""
    import torch
    from csaw import graphgen
    V, E = 1 << 16, 9_000_000
    rng = np.random.default_rng(6)
    deg = rng.multinomial(E, np.full(V, 1.0 / V))
    rowptr = np.concatenate([[0], np.cumsum(deg)])
    g = graphgen.CSR(rowptr, rng.integers(0, V, int(rowptr[-1])), None, name="wide")
    G = csaw.Graph(g, rowptr64=True)
    for n, per_step in ((120_001, 4 + 16 + 16), (20_000, 4 + 12 + 16)):
        seeds = oracle.make_seeds(g.rowptr, n, 9)
        p = csaw.make_params(1, 0, n, 1, 1, 5, None, 9, schedule=csaw.SCHED_BATCHED)
        G.profile(True)
        out = [x.cpu().numpy() for x in G.sample(p, torch.from_numpy(seeds).cuda())]
        st = G.kernel_stats("walk_thread")
        G.profile(False)
        assert st["bytes"] == per_step * len(out[0])
        got = sort_edges(*out)
        ref = sort_edges(*oracle.run(g.rowptr, g.col, g.weight, seeds, 1, 0, n, 1, 5, None, seed=9, n_threads=8))
        assert got.shape == ref.shape and np.array_equal(got, ref)
    G.close()
