"""The synchronisation protocol of the one-launch maximum-core search
(k_core_search in kc_cuda_b200/csrc/kcore.cu), checked on the CPU.

The blocks share rotating frontier counters, big-row counts and a level's
figures, which one thread resets while others may still be between a barrier
and their read of what it ended; the even rounds' frontier is the alive list
not in use, which the next list overwrites.  This runs a block-level
transcription -- same slots, resets and barriers, one read of the counters per
block some time after a barrier, every access a scheduling point -- under
random, skewed interleavings of 1 to 7 blocks, and checks that every block
leaves, the maximum core, its list in order, its degrees, and the tags of the
vertices outside."""
import random

import numpy as np
import pytest

import kt_oracle as O
from kc_cuda_b200 import gen

ALIVE = 0xffffffff
BIG = 4     # rows longer than this go to the dealt-window phase (the kernel's big_row)
WIN = 2     # entries per dealt window
MAXU = (1 << 64) - 1


def search(rows, B, seed, lo, hi, ramp, fixed=False, compact_below=0, most_probes=64):
    rng = random.Random(seed)
    n = len(rows)
    deg = [len(r) for r in rows]
    rem = [ALIVE if d else 0 for d in deg]
    snap = [None] * n
    alive = [[v for v in range(n) if deg[v]] + [None] * sum(d == 0 for d in deg), [None] * n]
    n_alive = sum(d > 0 for d in deg)
    odd = [None] * n
    big = [None] * n
    cnt = [0] * 7
    kept = [None] * B
    out = {"k": [], "left": []}
    bar = {"in": 0, "phase": 0}

    def push(to, slot, v):
        at = cnt[slot]
        cnt[slot] += 1
        assert at < n
        to[at] = v

    def barrier(*slots):
        yield
        phase = bar["phase"]
        bar["in"] += 1
        if bar["in"] == B:
            bar["in"], bar["phase"] = 0, phase ^ 1
        while bar["phase"] == phase:
            yield
        got = []
        for s in slots:  # one thread reads them, some time later
            yield
            got.append(cnt[s])
        return got

    def drop(ws, k, tag, to, slot):
        for w in ws:
            yield
            if rem[w] == ALIVE:
                old = deg[w]
                deg[w] -= 1
                if old == k:
                    rem[w] = tag
                    push(to, slot, w)

    def block(b):
        l, h, r, na, use, probes, tag, i, undo = lo, hi, ramp, n_alive, 0, 0, 1, 0, False

        def front(rnd):
            return odd if rnd & 1 else alive[use ^ 1]

        compact = False
        while (h - l > 1 or fixed) and na and probes < most_probes:
            k = l if fixed else (min(2 * l, h - 1) if r else l + (h - l) // 2)
            if not fixed and k <= l:
                k = l + 1
            if b == 0:
                cnt[(i + 2) % 3] = 0
                cnt[3 + ((i + 1) & 1)] = 0
                cnt[5], cnt[6] = MAXU, 0
            mine = alive[use]
            for j in range(b, na, B):
                v = mine[j]
                yield
                if undo:
                    d = deg[v] = snap[v]
                    rem[v] = ALIVE
                else:
                    d = deg[v]
                    if not fixed:
                        snap[v] = d
                if d < k:
                    rem[v] = tag
                    push(front(i + 1), (i + 1) % 3, v)
            undo = False
            i += 1
            sh = yield from barrier(i % 3)
            removed, empty = 0, False
            while sh[0]:
                nf = sh[0]
                removed += nf
                if not fixed and na - removed < k + 1:
                    empty = True
                    break
                now, to, nc, bc = front(i), front(i + 1), (i + 1) % 3, 3 + (i & 1)
                for f in range(b, nf, B):
                    v = now[f]
                    yield
                    if len(rows[v]) > BIG:
                        push(big, bc, v)
                    else:
                        yield from drop(rows[v], k, tag, to, nc)
                if b == 0:
                    cnt[(i + 2) % 3] = 0
                    yield
                    cnt[3 + ((i + 1) & 1)] = 0
                sh = yield from barrier(nc, bc)
                if sh[1]:
                    x = 0
                    for q in range(sh[1]):
                        v = big[q]
                        for w0 in range(0, len(rows[v]), WIN):
                            if x % B == b:
                                yield from drop(rows[v][w0:w0 + WIN], k, tag, to, nc)
                            x += 1
                    sh = yield from barrier(nc, bc)
                i += 1
            left = 0 if empty else na - removed
            if b == 0:
                out["k"].append(k)
                out["left"].append(left)
            probes += 1
            if not left:
                if fixed:
                    na = 0
                    break
                h, r, undo = k, False, True
                continue
            tag += 1
            stretch = -(-na // B)
            s0, s1 = min(na, b * stretch), min(na, (b + 1) * stretch)
            mn, total, count = MAXU, 0, 0
            for j in range(s0, s1):
                v = mine[j]
                yield
                if rem[v] == ALIVE:
                    count, total, mn = count + 1, total + deg[v], min(mn, deg[v])
            cnt[5] = min(cnt[5], mn)
            yield
            cnt[6] += total
            kept[b] = count
            dmin, dsum = yield from barrier(5, 6)
            at = 0
            for q in range(b):
                yield
                at += kept[q]
            to = alive[use ^ 1]
            for j in range(s0, s1):
                v = mine[j]
                yield
                if rem[v] == ALIVE:
                    to[at] = v
                    at += 1
            use, na, l = use ^ 1, left, k
            if dmin > l:
                l = min(dmin, h - 1)
            if fixed:
                break
            if dsum < compact_below:
                compact = True
                break
            yield from barrier()
        if undo:
            mine = alive[use]
            for j in range(b, na, B):
                yield
                deg[mine[j]] = snap[mine[j]]
                rem[mine[j]] = ALIVE
        if b == 0:
            out.update(lo=l, hi=h, ramp=r, n_alive=na, use=use, compact=compact)

    live = {b: block(b) for b in range(B)}
    weight = {b: rng.random() ** 4 + 1e-3 for b in live}
    steps = 0
    while live:
        if rng.random() < 0.002:
            weight = {b: rng.random() ** 4 + 1e-3 for b in range(B)}
        b = rng.choices(list(live), [weight[x] for x in live])[0]
        try:
            next(live[b])
        except StopIteration:
            del live[b]
        steps += 1
        assert steps < 4_000_000, "blocks wait for one that has left"
    assert bar["in"] == 0
    return out, deg, rem, alive[out["use"]][:out["n_alive"]]


def adjacency(e, n):
    rows = [[] for _ in range(n)]
    for a, b in zip((e >> np.uint64(32)).tolist(), (e & np.uint64(0xffffffff)).tolist()):
        rows[a].append(b)
        rows[b].append(a)
    return rows


GRAPHS = {
    "rmat7_k8": lambda: gen.Graph(gen.rmat(7, 4, 5, [8])).edges(),
    "er200_k9": lambda: gen.Graph(gen.GraphSpec(kind=gen.KTG_ER, n=200, draws=700, seed=4, cliques=[9])).edges(),
    "path": lambda: np.array([(a << 32) | (a + 1) for a in range(40)], dtype=np.uint64),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_search_protocol(name):
    e = GRAPHS[name]()
    n = int(max((e >> np.uint64(32)).max(), (e & np.uint64(0xffffffff)).max())) + 3
    rows = adjacency(e, n)
    core = O.core_numbers(e, n)
    top = int(core.max())

    def check(k, out, deg, rem, members, levels):
        assert members == [v for v in range(n) if core[v] >= k]
        for v in range(n):
            if core[v] >= k:
                assert rem[v] == ALIVE and deg[v] == sum(core[w] >= k for w in rows[v])
            elif rows[v]:  # removed by the first probe beyond its core number
                assert levels[rem[v] - 1] > core[v] and (rem[v] == 1 or levels[rem[v] - 2] <= core[v])

    for seed in range(10):
        B = [1, 2, 3, 5, 7][seed % 5]
        hi = max(len(r) for r in rows) + 1
        out, deg, rem, members = search(rows, B, seed, 1, hi, seed % 2 == 0)
        assert (out["lo"], out["hi"]) == (top, top + 1)
        check(top, out, deg, rem, members, [k for k, left in zip(out["k"], out["left"]) if left])
        k = 1 + seed % (top + 1)
        out, deg, rem, members = search(rows, B, seed, k, k + 1, False, fixed=True)
        check(k, out, deg, rem, members, [k])
        # Ends for a compaction, and for the launch's most probes.
        out, deg, rem, members = search(rows, B, seed, 1, hi, True, compact_below=len(e))
        if out["compact"]:
            check(out["k"][-1], out, deg, rem, members, [k for k, left in zip(out["k"], out["left"]) if left])
        out, deg, rem, members = search(rows, B, seed, 1, hi, False, most_probes=2)
        assert out["lo"] <= top < out["hi"]
        check(max([1] + [k for k, left in zip(out["k"], out["left"]) if left]), out, deg, rem, members,
              [k for k, left in zip(out["k"], out["left"]) if left])
