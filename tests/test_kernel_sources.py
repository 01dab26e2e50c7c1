"""Rules that the kernels' sources keep, where breaking one shows in no answer
until a compiler or a schedule makes it."""
import glob
import os

CSRC = os.path.join(os.path.dirname(__file__), "..", "kc_cuda_b200", "csrc")


def sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            yield os.path.basename(path), f.read()


def test_collectives_name_their_lanes():
    """A ballot and the shuffle after it take the same lanes: none of them takes
    whichever happen to run together at that point."""
    assert [name for name, text in sources() if "__activemask" in text] == []
