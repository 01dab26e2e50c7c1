"""Truss levels over the longest bitset rows, where a block has 128 threads
instead of 512 (the rows' shared memory), at both sides of that line and up to
the most vertices that have bitsets."""
import numpy as np
import pytest

import kt_oracle as O
import kc_cuda_b200 as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [50_000, 57_000, 60_001, 65_536])
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
