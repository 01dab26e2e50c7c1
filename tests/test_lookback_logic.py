"""The rule by which a tile of a one-pass scan finds its prefix when a
predecessor's word does not come (csrc/lookback.cuh), stepped on the CPU: tiles
run in any order of steps, any wait may give up at once, blocks may stop for
good after any step, and the output may overwrite the input.  Every tile that
ends must have the sum of the items before it.

Left out on purpose, each makes a schedule below fail: the second look at the
word after adding up the items (in place), and publishing before writing."""
import random

import pytest

TILE = 4


class Pass:
    def __init__(self, data, in_place, rng, second_look=True, publish_first=True):
        self.inp = list(data)
        self.out = self.inp if in_place else [None] * len(data)
        self.in_place = in_place
        self.tiles = (len(data) + TILE - 1) // TILE
        self.word = [None] * self.tiles  # ("sum" | "prefix", value)
        self.rng = rng
        self.second_look, self.publish_first = second_look, publish_first

    def items(self, t):
        return self.inp[t * TILE:(t + 1) * TILE]

    def write(self, t, own, prefix):
        for i, x in enumerate(own):
            self.out[t * TILE + i] = prefix
            prefix += x

    def run_tile(self, t):
        """A tile's steps; yields between any two accesses that others may see."""
        own = list(self.items(t))
        yield
        total = sum(own)
        if self.publish_first:
            self.word[t] = ("prefix" if t == 0 else "sum", total)
        yield
        prefix, p = 0, t - 1
        while p >= 0:
            w = self.word[p]
            while w is None and self.rng.random() < 0.5:  # waits, or gives up
                yield
                w = self.word[p]
            if w is None:
                added = 0
                for i in range(p * TILE, min((p + 1) * TILE, len(self.inp))):
                    added += self.inp[i]
                    yield
                w = self.word[p] if self.second_look else None
                if w is None:
                    w = ("sum", added)
            prefix += w[1]
            if w[0] == "prefix":
                break
            p -= 1
            yield
        if self.publish_first:
            self.word[t] = ("prefix", prefix + total)
            yield
            self.write(t, own, prefix)
        else:
            self.write(t, own, prefix)
            yield
            self.word[t] = ("prefix", prefix + total)


def wrong_sums(in_place, seeds, **rule):
    wrong = 0
    for seed in range(seeds):
        rng = random.Random(seed)
        data = [rng.randint(0, 9) for _ in range(rng.randint(1, 40))]
        want = [sum(data[:i]) for i in range(len(data))]
        P = Pass(data, in_place, rng, **rule)
        live = {t: P.run_tile(t) for t in range(P.tiles)}
        for t in rng.sample(range(P.tiles), rng.randint(0, P.tiles // 2)):  # these stop for good
            for _ in range(rng.randint(0, 3)):
                next(live[t], None)
            del live[t]
        ended = []
        while live:
            t = rng.choice(list(live))
            try:
                next(live[t])
            except StopIteration:
                ended.append(t)
                del live[t]
        for t in ended:
            a, b = t * TILE, min((t + 1) * TILE, len(data))
            wrong += P.out[a:b] != want[a:b]
    return wrong


@pytest.mark.parametrize("in_place", [False, True])
def test_every_tile_that_ends_has_its_prefix(in_place):
    assert wrong_sums(in_place, 3000) == 0


@pytest.mark.parametrize("rule", [dict(second_look=False), dict(publish_first=False)])
def test_the_steps_that_in_place_scans_need(rule):
    assert wrong_sums(True, 3000, **rule) > 0
