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


def regular(V, d, seed):
    """V vertices of d distinct neighbors each, uniform weights."""
    from csaw import graphgen
    rng = np.random.default_rng(seed)
    step = rng.permutation(np.arange(1, V))[:d]
    col = (np.arange(V)[:, None] + np.sort(step)[None, :]) % V
    col.sort(axis=1)
    return graphgen.CSR(np.arange(V + 1, dtype=np.int64) * d, col.reshape(-1).astype(np.int32),
                        (rng.random(V * d) + 1e-3).astype(np.float32), name="regular")


@pytest.mark.parametrize("bias,schedule", [(0, 0), (0, 1), (1, 1), (2, 1)])
def test_wide_trees_of_few_roots_use_the_whole_gpu(csaw, bias, schedule):
    """The default rule: a tree whose levels would keep one SM's warps waiting
    goes by the per-level launches; the same fan-outs on short rows (taken
    whole), the same items from more roots, and narrow levels go in one."""
    long_rows, short_rows = regular(3000, 200, 1), regular(3000, 3, 2)
    for g, n, F, fan, tree in ((long_rows, 4, 1, [32, 32, 32], 0), (long_rows, 1, 4, [31, 32, 32], 0),
                               (short_rows, 4, 1, [32, 32, 32], 1), (long_rows, 64, 1, [25, 10], 1),
                               (long_rows, 33, 32, [32], 1), (long_rows, 1, 600, [2, 2], 1)):
        seeds = oracle.make_seeds(g.rowptr, n * F, 3)
        G = csaw.Graph(g)
        p = csaw.make_params(0, bias, n, F, fan[0], len(fan), fan, 0xD0, schedule=schedule)
        got, kinds = run(G, p, seeds)
        G.close()
        assert kinds["tree"]["launches"] == tree, (g.name, g.rowptr[1], n, F, fan)
        ref = expected(g, seeds, bias, n, F, fan, 0xD0)
        assert got.shape == ref.shape and np.array_equal(got, ref), (n, F, fan)


@pytest.mark.parametrize("bias,schedule", [(0, 0), (0, 1), (1, 1), (2, 1)])
@pytest.mark.parametrize("d", [3, 4, 5, 9, 13, 17, 24, 31, 33])
def test_grouped_draws_of_short_rows(csaw, d, bias, schedule):
    """Rows around N, 2N and 3N edges, where grouped items' first phases fail
    now and then or always, for one slot to sixteen."""
    from csaw import _lib
    g = regular(800, d, 40 + d)
    G = csaw.Graph(g)
    G.set_option(_lib.OPT_TREE, 2)
    for k, fan in enumerate(([1, 3], [2, 4], [4, 2], [8, 2], [12, 1], [16, 2])):
        n, F = 90, 3
        seeds = oracle.make_seeds(g.rowptr, n * F, 7 + k)
        p = csaw.make_params(0, bias, n, F, fan[0], 2, fan, 0xE0 + k, schedule=schedule)
        got, kinds = run(G, p, seeds)
        ref = expected(g, seeds, bias, n, F, fan, 0xE0 + k)
        assert kinds["tree"]["launches"] == 1
        assert got.shape == ref.shape and np.array_equal(got, ref), fan
    G.close()


@pytest.mark.parametrize("schedule", [0, 1])
@pytest.mark.parametrize("d", [20, 33, 200])
def test_unbiased_levels_around_the_warps_of_a_chunk(csaw, d, schedule):
    """Unbiased levels of one item less than the 16 warps of a chunk of few
    roots, as many, and one more: a warp each, or in groups."""
    from csaw import _lib
    g = regular(800, d, 60 + d)
    G = csaw.Graph(g)
    G.set_option(_lib.OPT_TREE, 2)
    for k, fan in enumerate(([15, 4], [16, 4], [17, 4], [1, 16, 2], [5, 3, 2])):
        seeds = oracle.make_seeds(g.rowptr, 20, 9 + k)
        p = csaw.make_params(0, 0, 20, 1, fan[0], len(fan), fan, 0xF0 + k, schedule=schedule)
        got, kinds = run(G, p, seeds)
        ref = expected(g, seeds, 0, 20, 1, fan, 0xF0 + k)
        assert kinds["tree"]["launches"] == 1
        assert got.shape == ref.shape and np.array_equal(got, ref), fan
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
