"""Truss peeling without bitsets: the rounds that look triangles up in the edge
hash table, against the oracle, at the sizes where they can go wrong -- shorter
rows of fewer and more than 256 entries (walked by a warp / dealt to the grid
after a barrier), rounds with a long row right after rounds with others, levels
whose first round has long rows, graphs with one edge -- and against the merge
of sorted rows, which remains where the budget has no room for the table."""
import numpy as np
import pytest

import kt_oracle as O
import kc_cuda_b200 as K
from kc_cuda_b200 import gen

pytestmark = pytest.mark.gpu


def clique(n, base=0):
    i, j = np.triu_indices(n, 1)
    return np.stack([i + base, j + base], axis=1)


def chained_cliques(sizes):
    """Cliques that share one vertex with the next, so levels follow closely."""
    out, base = [], 0
    for s in sizes:
        out.append(clique(s, base))
        base += s - 1
    return np.concatenate(out)


def two_hubs(leaves):
    """Two adjacent hubs with common leaves on a cycle: rows of `leaves` entries meet."""
    r = np.arange(leaves) + 2
    return np.concatenate([[[0, 1]], np.stack([np.zeros_like(r), r], 1), np.stack([np.ones_like(r), r], 1),
                           np.stack([r, np.roll(r, 1)], 1)])


GRAPHS = {
    "edge": lambda: np.array([[0, 1]]),
    "cliques": lambda: chained_cliques([3, 5, 33, 34, 64, 65, 257, 258, 259, 300]),
    "hubs255": lambda: two_hubs(255),
    "hubs256": lambda: two_hubs(256),
    "hubs900": lambda: np.concatenate([two_hubs(900), clique(40, 300)]),
    "rmat": lambda: gen.Graph(gen.rmat(13, 24, 4, [50])).edge_pairs(),
    "er": lambda: gen.Graph(gen.GraphSpec(kind=gen.KTG_ER, n=1500, draws=150_000, seed=3)).edge_pairs(),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_list_peel_equals_oracle(name):
    with K.Context(0) as ctx:
        ctx.set_option("dense_max_n", 0)
        dg = ctx.load_edges(GRAPHS[name]())
        edges = dg.edges()
        want = O.trussness(edges)
        for _ in range(2):
            assert np.array_equal(dg.trussness(), want)
        k = int(want.max(initial=0))
        answer = (k, int((want == k).sum())) if k >= 3 else (0, 0)
        assert dg.kmax_truss() == answer
        dg.free()


def test_without_room_for_the_table():
    """The same answers under a budget that the table does not fit."""
    g = gen.Graph(gen.rmat(13, 24, 4, [50]))
    with K.Context(0) as ctx:
        ctx.set_option("dense_max_n", 0)
        dg = ctx.load_edges(g.edge_pairs())
        want = dg.trussness()
        dg.free()
        ctx.reset_stats()
        dg = ctx.load_edges(g.edge_pairs())
        dg.trussness()
        peak = ctx.stats()["device_bytes_peak"]
        dg.free()
    ran = 0
    for part in range(60, 100, 4):
        with K.Context(0, hbm_budget=peak * part // 100) as ctx:
            ctx.set_option("dense_max_n", 0)
            try:
                dg = ctx.load_edges(g.edge_pairs())
                assert np.array_equal(dg.trussness(), want)
                ran += 1
                dg.free()
            except K.KtError as e:
                assert e.status == 3  # the budget, refused as such
    assert ran
