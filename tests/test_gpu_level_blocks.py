"""Truss levels over long bitset rows, where a block has 256 or 128 threads
instead of 512 (the rows' shared memory), at both sides of the lines and up to
the most vertices that have bitsets, with common neighbours dealt to a warp's
lanes and closed by the lanes whose words hold them; and when a round counts
anew."""
import re

import numpy as np
import pytest

import kt_oracle as O
import kc_cuda_b200 as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16_200, 16_384, 50_000, 57_000, 60_001, 65_536])
def test_levels_over_long_rows(n, capfd):
    rng = np.random.default_rng(n)
    ring = np.stack([np.arange(n), (np.arange(n) + 1) % n])  # every vertex has an edge
    parts = [ring, rng.integers(0, n, (2, 150_000))]
    for size in (60, 45, 45, 30):
        c = rng.permutation(n)[:size]
        i, j = np.triu_indices(size, 1)
        keep = rng.random(len(i)) < 0.9
        parts.append(np.stack([c[i[keep]], c[j[keep]]]))
    x, y = np.concatenate(parts, 1).astype(np.uint64)
    with K.Context(0) as ctx:
        ctx.set_option("dense_min_fill", 1_000_000)
        ctx.set_option("recount_gamma", 1000)  # both kinds of rounds
        g = ctx.load_pairs((x << np.uint64(32)) | y)
        want = O.trussness(g.edges())
        ctx.set_option("verbose", 1)
        assert np.array_equal(g.trussness(), want)
        assert "(n %d, W %d)" % (n, ((n + 31) // 32 + 3) & ~3) in capfd.readouterr().err
        ctx.set_option("recount_gamma", 1)
        assert np.array_equal(g.trussness(), want)
        g.free()


def test_one_graph_counts_anew_where_decrements_cost_more(capfd):
    """Rounds that take a few per cent of a graph's edges: counting the others
    anew costs less than closing the triangles of those (with the factor that a
    union's largest threshold asks for, the last climb counted in no round)."""
    rng = np.random.default_rng(4000)
    u, v = np.nonzero(np.triu(rng.random((4000, 4000), dtype=np.float32) < 0.08, 1))
    with K.Context(0) as ctx:
        g = ctx.load_edges(np.stack([u, v], 1))
        ctx.set_option("verbose", 1)
        got = g.kmax_truss()
        recounts = [int(x) for x in re.findall(r"rounds \((\d+) recount\)", capfd.readouterr().err)]
        assert got == O.solve_edges(g.edges())
        assert sum(recounts) >= 4
        g.free()
