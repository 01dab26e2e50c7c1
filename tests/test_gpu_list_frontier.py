"""Rounds of truss peeling without bitsets at the line between the two ways of
dealing a frontier: up to 1,024 edges by windows of their rows, above that a
warp per batch of edges.  Disjoint triangles on top of a star give first rounds
of an exact number of edges; the star's hub makes some of their rows long."""
import numpy as np
import pytest

import kt_oracle as O
import kc_cuda_b200 as K

pytestmark = pytest.mark.gpu


def first_round(edges):
    """A 12-clique, a fan of hub triangles, and pendants: `edges` edges without a triangle."""
    i, j = np.triu_indices(12, 1)
    hub, at = 0, 12
    fan = np.arange(at, at + 600)
    at += 600
    pend = np.arange(at, at + edges)
    tri = np.stack([fan[0::2], fan[1::2]], 1)
    spread = np.where(np.arange(edges) % 2, hub, fan[np.arange(edges) % len(fan)])
    return np.concatenate([np.stack([i, j], 1), np.stack([np.full_like(fan, hub), fan], 1), tri,
                           np.stack([spread, pend], 1)])


@pytest.mark.parametrize("edges", [1, 1023, 1024, 1025, 2048])
@pytest.mark.parametrize("persistent", [0, 1])
def test_rounds_at_the_line(edges, persistent):
    with K.Context(0) as ctx:
        ctx.set_option("dense_max_n", 0)
        ctx.set_option("persistent", persistent)
        dg = ctx.load_edges(first_round(edges))
        e = dg.edges()
        want = O.trussness(e)
        assert int((want == 2).sum()) == edges
        assert np.array_equal(dg.trussness(), want)
        dg.free()


@pytest.mark.parametrize("budget", [0, 1])
def test_rows_packed_as_edges_leave(budget):
    """Many levels over which the edges halve several times, with room for the
    rows' copies and (a budget just below the peak with them) without."""
    rng = np.random.default_rng(8)
    parts = [np.stack(np.triu_indices(n, 1), 1) + off for n, off in
             [(20, 0), (40, 10), (80, 30), (120, 70), (160, 150)]]
    parts.append(rng.integers(0, 3000, (60_000, 2)))
    e = np.concatenate(parts)
    with K.Context(0) as ctx:
        ctx.set_option("dense_max_n", 0)
        dg = ctx.load_edges(e)
        want = O.trussness(dg.edges())
        ctx.reset_stats()
        assert np.array_equal(dg.trussness(), want)
        peak = ctx.stats()["device_bytes_peak"]
        dg.free()
    if budget:
        with K.Context(0, hbm_budget=peak - (1 << 16)) as ctx:
            ctx.set_option("dense_max_n", 0)
            dg = ctx.load_edges(e)
            assert np.array_equal(dg.trussness(), want)
            dg.free()
