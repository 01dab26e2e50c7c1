"""The dealing of common neighbours in the peel's bitset rounds (close_common in
kc_cuda_b200/csrc/peel.cu), transcribed and checked on the CPU for chunks of 1 to
32 words: the words' popcounts are scanned over the warp, each lane finds its
task's word with a 5-step search over all 32 lanes and its bit with a select, so
every set bit of the chunk is visited exactly once.  Also the choice of the
chunk length: the units cover every row once, and fill the grid at most once
where chunks shorter than eight words are used."""
import random

import pytest

from test_peel_split_logic import select_bit

MOST = 8  # kSplitWords


def deal(words):
    c = [bin(w).count("1") for w in words] + [0] * (32 - len(words))
    excl = [sum(c[:i]) for i in range(32)]
    total = sum(c)
    visits = []
    for base in range(0, total, 32):
        for lane in range(32):
            t, lo = base + lane, 0
            for st in (16, 8, 4, 2, 1):
                if excl[lo + st] <= t:
                    lo += st
            if t < total:
                visits.append((lo, select_bit(words[lo], t - excl[lo])))
    return visits


@pytest.mark.parametrize("cw", [1, 2, 4, 8, 31, 32])
def test_every_common_neighbour_once(cw):
    rng = random.Random(cw)
    for trial in range(400):
        density = rng.choice([0.0, 0.03, 0.5, 0.97, 1.0])
        words = [sum(1 << b for b in range(32) if rng.random() < density) for _ in range(rng.randint(1, cw))]
        want = [(w, b) for w in range(len(words)) for b in range(32) if words[w] >> b & 1]
        got = deal(words)
        assert sorted(got) == want and len(got) == len(want), (trial, words)


@pytest.mark.parametrize("W", [2, 4, 8, 44, 60, 136, 1736])
def test_chunk_choice(W):
    rng = random.Random(W)
    for _ in range(300):
        gwarps = rng.choice([8, 64, 1184, 4736])
        nf = rng.randint(1, max(1, 16 * gwarps // -(-W // MOST)))
        cw = 1
        while cw < MOST and nf * -(-W // cw) > gwarps:
            cw *= 2
        chunks = -(-W // cw)
        covered = sorted(w for ch in range(chunks) if ch * cw < W for w in range(ch * cw, min(W, ch * cw + cw)))
        assert covered == list(range(W))
        assert cw == MOST or nf * chunks <= gwarps
