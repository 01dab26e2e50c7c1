"""The one-pass sort, scans and compactions at the edges of their tiles, through
the graph build: records around the 2,048-item tiles of the scans and
compactions and the 4,096-key tile of the sort (one block below, look-back over
many tiles above), random order, repeats and self-loops, ids of one and several
digits, and contexts whose look-back words are reused and grown."""
import numpy as np
import pytest

import kt_oracle as O
import kc_cuda_b200 as K

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with K.Context(0) as c:
        yield c


def records(count, ids, seed):
    rng = np.random.default_rng(seed)
    x = rng.integers(0, ids, count, dtype=np.uint64)
    y = rng.integers(0, ids, count, dtype=np.uint64)
    return (x << np.uint64(32)) | y


@pytest.mark.parametrize("ids", [3, 200, 70_000, (1 << 24) + 3])
@pytest.mark.parametrize("count", [1, 2, 31, 255, 2047, 2048, 2049, 4095, 4096, 4097, 8191, 8192, 8193, 300_001])
def test_edges_sorted_and_distinct(ctx, count, ids):
    xy = records(count, ids, count + ids)
    want = O.clean(xy)
    g = ctx.load_pairs(xy)
    assert np.array_equal(g.edges(), want)
    if ids <= 70_000:
        assert np.array_equal(g.tricount(), O.support(want))
    g.free()


def test_large_ids_and_many_launches(ctx):
    """Ids up to 2^32 - 2 (every bit of a key counts), and enough small launches
    for the look-back words to serve many epochs."""
    xy = records(5000, 2_000, 9)
    top = np.uint64((1 << 32) - 2)
    u, v = xy >> np.uint64(32), xy & np.uint64(0xFFFFFFFF)
    g = None
    try:
        g = ctx.load_pairs(((top - u) << np.uint64(32)) | v)
        assert np.array_equal(g.edges(), O.clean(((top - u) << np.uint64(32)) | v))
    except K.KtError as e:  # 2^32 vertices need more memory than a context may have
        assert e.status == 3
    finally:
        if g is not None:
            g.free()
    small = records(9000, 300, 11)
    want = O.solve_edges(O.clean(small))
    for _ in range(40):
        g = ctx.load_pairs(small)
        assert g.kmax_truss() == want
        g.free()
