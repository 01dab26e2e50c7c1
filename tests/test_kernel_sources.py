"""Rules that the kernels' sources keep, where breaking one shows in no answer
until a compiler or a schedule makes it."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "kc_cuda_b200", "csrc")


def sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            yield os.path.basename(path), f.read()


def test_collectives_name_their_lanes():
    """A ballot and the shuffle after it take the same lanes: none of them takes
    whichever happen to run together at that point."""
    assert [name for name, text in sources() if "__activemask" in text] == []


def test_lists_that_a_launch_rewrites_are_not_restrict():
    """Counting groups take an alive list, edge states and rows which the truss
    levels rewrite between two calls in one launch."""
    text = dict(sources())["dense.cuh"]
    for name, rewritten in (("dense_group", ("list", "state")), ("dense_group_short", ("list", "state")),
                            ("dense_load_row", ("p",))):
        args = re.search(r"void %s\(([^)]*)\)" % name, text).group(1)
        for arg in rewritten:
            assert re.search(r"const uint32_t\* %s\b" % arg, args), (name, arg)
