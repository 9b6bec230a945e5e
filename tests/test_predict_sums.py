"""How many sums a row of several outputs has in registers (csrc/predict_sums.h), on the CPU."""
import ctypes
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "legate-boost_b200", "csrc")


def test_no_number_of_outputs_has_more_than_one_sum_too_many(tmp_path):
    (tmp_path / "t.cpp").write_text('#include "predict_sums.h"\nextern "C" int sums(int K) { return lbk::SumsOf(K); }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t.so")], check=True)
    sums = ctypes.CDLL(str(tmp_path / "t.so")).sums
    assert sums(1) == 0 and sums(17) == sums(1000) == -1
    for K in range(2, 17):
        assert K <= sums(K) <= K + 1 and (K <= 4 or sums(K) % 2 == 0), K
