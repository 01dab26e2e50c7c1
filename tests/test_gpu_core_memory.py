"""Device memory of the maximum-core search, which counts against a context's
budget: seven words a vertex (degree, tag, alive list, two frontiers, long rows,
the degrees before a probe), and what a solve needs later is not added to it."""
import numpy as np
import pytest

import kt_oracle as O
import kc_cuda_b200 as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count", [(700_001, 1_500_000), (2_000_003, 3_000_000)])
def test_search_scratch(n, count):
    rng = np.random.default_rng(n)
    x = rng.integers(0, n, count, dtype=np.uint64)
    y = rng.integers(0, n, count, dtype=np.uint64)
    x[-1] = n - 1
    with K.Context(0) as ctx:
        g = ctx.load_pairs((x << np.uint64(32)) | y)
        want = O.core_numbers(g.edges(), n)
        ctx.reset_stats()
        before = ctx.stats()["device_bytes_peak"]  # what the graph holds
        member, cmax = g.kmax_core(2)
        peak = ctx.stats()["device_bytes_peak"] - before
        assert cmax == want.max() and np.array_equal(member, want >= 2)
        assert peak <= 7 * 4 * n + (1 << 18)
        g.free()
