"""The parser's word-at-a-time route against the oracle's parse: every length of
both numbers from 1 to 10 digits, separators of one and several bytes, letters
(which count as digits), high bytes, carriage returns, extra columns, blank
lines, line starts at every offset of a word, and lines near the ends of the
9,216-byte blocks and of the input."""
import numpy as np
import pytest

import kt_oracle as O
import kc_cuda_b200 as K

pytestmark = pytest.mark.gpu


def check(ctx, data):
    g = ctx.load_tsv(data)
    assert np.array_equal(g.edges(), O.clean(O.parse(data)))
    g.free()


@pytest.fixture(scope="module")
def ctx():
    with K.Context(0) as c:
        yield c


@pytest.mark.parametrize("sep", [b"\t", b" ", b",", b"\t\t", b" \t ", b"\xc3\xa9", b"-"])
def test_lengths_and_separators(ctx, sep):
    ids = [7, 42, 123, 9876, 54321, 999_999, 1_234_567, 7_654_321]
    lines = [b"%d%s%d" % (x, sep, y) for x in ids for y in ids]
    pad = b"#\n"
    for shift in range(4):
        for end in (b"\n", b"\r\n", b"\t1\n"):
            check(ctx, pad[:0] + b"1" * shift + b"5\t2\n" + end.join(lines) + end)


def test_long_numbers_wrap_and_zeros(ctx):
    # Leading zeros make long runs without large ids (9 and more characters).
    lines = [b"%s\t%s" % (b"0" * i + b"12", b"0" * j + b"345") for i in range(12) for j in range(12)]
    check(ctx, b"\n".join(lines) + b"\n")
    check(ctx, b"\n".join(lines))  # no newline at the end


def test_letters_are_digits(ctx):
    lines = [b"1:\t2", b"A\t3", b"9z\t1", b"12\tZ", b"a1\tb", b"7\t~"]
    check(ctx, b"\n".join(lines * 3) + b"\n")


@pytest.mark.parametrize("width", [1, 5, 8])
def test_block_edges(ctx, width):
    """Lines of varying lengths over several blocks, ending at every byte around a block's end."""
    rng = np.random.default_rng(width)
    top = 10 ** width
    rows = rng.integers(0, min(top, 4_000_000), (6000, 2))
    body = b"".join(b"%0*d\t%d\n" % (1 + i % width, x, y) for i, (x, y) in enumerate(rows.tolist()))
    for cut in list(range(9216 - 30, 9216 + 30)) + [len(body)]:
        data = body[:cut]
        nl = data.rfind(b"\n") + 1
        tail = data[nl:]
        if tail.count(b"\t") == 0 or tail.endswith(b"\t"):
            data = data[:nl]  # a line cut inside its first number is an error by the grammar
        check(ctx, data)
