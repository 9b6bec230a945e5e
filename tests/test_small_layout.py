"""Where the levels of the one-launch tree keep their split candidates (csrc/small_layout.h), on the CPU."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "legate-boost_b200", "csrc")


@pytest.fixture(scope="module")
def layout(tmp_path_factory):
    d = tmp_path_factory.mktemp("small_layout")
    (d / "t.cpp").write_text('#include "small_layout.h"\n'
                             'extern "C" int begin(int depth, int D) { return lbk::SmallCandBegin(depth, D); }\n'
                             'extern "C" int nodes(int D) { return lbk::SmallCandNodes(D); }\n')
    subprocess.run(["g++", "-shared", "-fPIC", "-I", CSRC, str(d / "t.cpp"), "-o", str(d / "t.so")], check=True)
    return ctypes.CDLL(str(d / "t.so"))


@pytest.mark.parametrize("D", range(1, 13))
def test_a_level_does_not_overwrite_the_one_that_slower_blocks_still_read(layout, D):
    """A block may write level d + 1 while another reads level d: their candidates do not overlap, and lie inside what is
    allocated."""
    spans = [(layout.begin(d, D), layout.begin(d, D) + 2 ** d) for d in range(D)]
    for d, (b, e) in enumerate(spans):
        assert 0 <= b and e <= layout.nodes(D)
        if d > 0:
            assert e <= spans[d - 1][0] or b >= spans[d - 1][1], (d, spans)
