"""Supports from the product of the adjacency rows, against the square of the
adjacency matrix: just past the shortest rows, at and around whole tiles of 256,
more tiles than blocks, sparse and empty parts of a dense matrix."""
import numpy as np
import pytest

import kt_oracle as O
import kc_cuda_b200 as K

pytestmark = pytest.mark.gpu


def dense(n, p, seed, hole=0):
    """A random graph, or one with `hole` vertices that only a few edges reach."""
    rng = np.random.default_rng(seed)
    a = np.triu(rng.random((n, n)) < p, 1)
    if hole:
        a[:, n - hole:] &= rng.random((n, hole)) < 0.02
    return a | a.T


@pytest.mark.parametrize("n,p,hole", [
    (2049, 0.9, 0), (2304, 0.6, 0), (2305, 0.6, 0), (2400, 0.7, 300), (2560, 1.0, 0), (4400, 0.3, 0), (4700, 0.4, 700)])
def test_support_is_the_square(n, p, hole):
    a = dense(n, p, n, hole)
    u, v = np.nonzero(np.triu(a))
    b = a.astype(np.float32)
    square = (b @ b).astype(np.uint32)  # sums below 2^24
    with K.Context(0) as ctx:
        d = ctx.load_edges(np.stack([u, v], 1))
        e = d.edges()
        got = d.tricount()
        assert np.array_equal(got, square[e >> 32, e & 0xffffffff])
        d.free()


@pytest.mark.parametrize("n", [5, 40, 127, 129, 1000, 1025, 2048])
def test_short_rows(n):
    """Rows of 4 to 64 words, by popcounts: both vectors of a lane, runs of edges
    that share a row and ends of the list within a group."""
    a = dense(n, 0.3 if n > 200 else 0.8, n)
    u, v = np.nonzero(np.triu(a))
    b = a.astype(np.float32)
    square = (b @ b).astype(np.uint32)
    with K.Context(0) as ctx:
        ctx.set_option("dense_min_fill", 1000)
        d = ctx.load_edges(np.stack([u, v], 1))
        e = d.edges()
        assert np.array_equal(d.tricount(), square[e >> 32, e & 0xffffffff])
        assert np.array_equal(d.trussness(), O.trussness(e))
        d.free()


def test_union_of_dense_and_sparse_graphs():
    """A batch whose union has graphs for both ways of counting, one of them
    empty of triangles: every answer equals the graph's alone."""
    graphs = []
    for n, p, hole in [(2100, 0.7, 0), (40, 0.5, 0), (3000, 0.04, 0), (2700, 0.5, 400), (300, 0.9, 0), (2304, 0.6, 0)]:
        u, v = np.nonzero(np.triu(dense(n, p, n, hole)))
        graphs.append(np.stack([u, v], 1))
    graphs.append(np.stack([np.zeros(500, np.int64), np.arange(1, 501)], 1))
    with K.Context(0) as ctx:
        ctx.set_option("dense_min_fill", 1000)
        want = []
        for e in graphs:
            d = ctx.load_edges(e)
            want.append(d.kmax_truss())
            d.free()
        b = ctx.batch()
        for e in graphs:
            b.add_edges(e)
        b.run()
        k, c = b.results()
        assert list(zip(k.tolist(), c.tolist())) == want
