"""Which bytes of a row the lanes of k_hist_smem load and which words of a bin they add to (csrc/hist_units.h), on the CPU."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "legate-boost_b200", "csrc")
GROUP = 32  # features per group: the bins of a row are padded to whole groups


@pytest.fixture(scope="module")
def units(tmp_path_factory):
    d = tmp_path_factory.mktemp("hist_units")
    (d / "t.cpp").write_text('#include "hist_units.h"\n'
                             'using namespace lbk;\n'
                             'extern "C" int word(int fl, int W, int several, int nt, int w) { return FeatureOfWord(W, FormOf(fl, W, several, nt), w); }\n'
                             'extern "C" int bytes(int fl, int W, int several, int nt) { return LaneBytes(FormOf(fl, W, several, nt)); }\n'
                             'extern "C" int piece(int fl, int W, int several, int nt, int groups, int q)\n'
                             '{ return PieceOfLane(W, FormOf(fl, W, several, nt), groups, q); }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "t.cpp"), "-o", str(d / "t.so")], check=True)
    return ctypes.CDLL(str(d / "t.so"))


def _units_of(F):
    """(width, groups of the matrix, first group, groups, features) of the units of a row."""
    G = -(-F // GROUP)
    W = 1 if G == 1 else 2
    for g0 in range(0, G, W):
        yield W, G, g0, min(W, G - g0), min(GROUP * W, F - g0 * GROUP)


@pytest.mark.parametrize("floats", [0, 1])
def test_no_lane_reads_beyond_its_row(units, floats):
    """A caller's matrix ends with its last row: no lane's bytes lie outside the G x 32 of a row, or beyond its unit."""
    for F in range(1, 257):
        for W, G, g0, groups, nt in _units_of(F):
            n = units.bytes(floats, W, G > 2, nt)
            for q in range(2 * W):
                begin = g0 * GROUP + units.piece(floats, W, G > 2, nt, groups, q) * n
                assert begin % n == 0 and g0 * GROUP <= begin and begin + n <= (g0 + groups) * GROUP <= G * GROUP, (F, g0, q)


@pytest.mark.parametrize("floats", [0, 1])
def test_every_feature_has_one_word(units, floats):
    for F in range(1, 257):
        for W, G, g0, groups, nt in _units_of(F):
            words = [units.word(floats, W, G > 2, nt, w) for w in range(GROUP * W)]
            own = sorted(w for w in words if 0 <= w < nt)
            assert own == list(range(nt)), (F, g0)
