"""Large copies from and to pageable memory: a new context's first call does not
pay for pinned memory, and the slots that later copies share among contexts and
threads keep their bytes apart."""
import threading
import time

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


def test_first_large_copy_of_a_context():
    """Pinning 16 MB takes 2 ms at the least (median 15); a first call on 2.4 MB
    differs from the second by less than 1 without it (small allocations)."""
    xy = records(300_000, 20_000, 3)
    with K.Context(0) as warm:  # the process's own first use of the kernels
        warm.load_pairs(xy).free()
    more = []
    for _ in range(9):
        with K.Context(0) as ctx:
            t = [time.perf_counter()]
            for _ in range(2):
                g = ctx.load_pairs(xy)
                t.append(time.perf_counter())
                g.free()
            more.append((t[1] - t[0]) - (t[2] - t[1]))
    assert np.median(more) < 2e-3


def test_contexts_and_threads_share_slots():
    cases = [records(n, n // 8, n) for n in (140_000, 600_001, 1_300_003, 2_000_000, 900_000, 530_000)]
    want = [O.clean(xy) for xy in cases]
    wrong = []

    def work(i):
        with K.Context(0) as ctx:
            for k in range(16):  # 128 MB or more in all after a few rounds
                j = (i + k) % len(cases)
                g = ctx.load_pairs(cases[j])
                e = g.edges()
                if not np.array_equal(e, want[j]) or len(g.tricount()) != len(e):
                    wrong.append((i, k))
                g.free()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    # All contexts are gone, and the slots with them; a new one starts over.
    with K.Context(0) as ctx:
        for k in range(20):
            g = ctx.load_pairs(cases[3])
            assert np.array_equal(g.edges(), want[3])
            g.free()
