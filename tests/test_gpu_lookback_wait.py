"""Scans and compactions whose look-back waits give up: with timeout_ms = 0 a
tile waits for no predecessor that has not published its sum, and adds up that
tile's items itself.  Nothing fails then, so the answers are the usual ones --
of the graph build (scans in place and apart, compactions, sorts of one and of
many tiles) and of host-stepped solves, which have no other wait."""
import numpy as np
import pytest

import kt_oracle as O
import kc_cuda_b200 as K

pytestmark = pytest.mark.gpu


def records(count, ids, seed):
    rng = np.random.default_rng(seed)
    x = rng.integers(0, ids, count, dtype=np.uint64)
    y = rng.integers(0, ids, count, dtype=np.uint64)
    return (x << np.uint64(32)) | y


@pytest.mark.parametrize("count,ids", [(1, 3), (2048, 200), (2049, 5000), (4097, 70_000), (65_537, 3000),
                                       (300_001, 70_000), (3_000_001, 400_009)])
def test_waits_that_give_up_leave_the_sums_right(count, ids):
    xy = records(count, ids, count)
    want = O.clean(xy)
    with K.Context(0) as ctx:
        ctx.set_option("timeout_ms", 0)
        ctx.set_option("persistent", 0)
        ctx.set_option("dense_max_n", 0)
        for _ in range(3):
            g = ctx.load_pairs(xy)
            assert np.array_equal(g.edges(), want)
            if count <= 300_001:
                assert np.array_equal(g.tricount(), O.support(want))
                assert g.kmax_truss() == O.solve_edges(want)
            g.free()


def test_more_launches_than_epochs():
    """The look-back words' epochs (2^14, one for each compaction and each scan
    of several tiles) come round, with and without waits that give up."""
    xy = records(9000, 5000, 11)
    want = O.clean(xy)
    answer = O.solve_edges(want)
    with K.Context(0) as ctx:
        for i in range(2200):  # eight epochs or more each
            g = ctx.load_pairs(xy)
            assert g.kmax_truss() == answer
            g.free()
        ctx.set_option("timeout_ms", 0)
        for i in range(9000):  # two epochs each
            g = ctx.load_pairs(xy)
            if i % 500 < 2:
                assert np.array_equal(g.edges(), want)
            g.free()
