"""How many blocks share the rows of a table of the binning kernels (csrc/bin_grid.h), on the CPU."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "legate-boost_b200", "csrc")


@pytest.fixture(scope="module")
def blocks_of(tmp_path_factory):
    d = tmp_path_factory.mktemp("bin_grid")
    (d / "t.cpp").write_text('#include "bin_grid.h"\n'
                             'extern "C" int64_t blocks(int64_t rows, int64_t tables, int64_t resident, int64_t fill)\n'
                             '{ return lbk::BinGridBlocks(rows, tables, resident, fill); }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "t.cpp"), "-o", str(d / "t.so")], check=True)
    f = ctypes.CDLL(str(d / "t.so")).blocks
    f.restype, f.argtypes = ctypes.c_int64, [ctypes.c_int64] * 4
    return f


@pytest.mark.parametrize("resident,fill", [(148, 2048), (444, 512), (592, 512), (1184, 0), (132, 2048)])
def test_no_wave_of_blocks_is_nearly_empty(blocks_of, resident, fill):
    """Waves times the rows (and the table) of a block, against a device that is full to the end.  Rounded up, three tables on
    148 places are 150 blocks: twice the time."""
    for rows in (200_000, 1_000_003, 10_000_000, 100_000_000, 2_000_000_000):
        for tables in list(range(1, 33)) + [64, 100, 128]:
            b = blocks_of(rows, tables, resident, fill)
            assert 1 <= b <= (rows + 63) // 64
            waves = -(-b * tables // resident)
            took, full = waves * (rows / b + fill), rows * tables / resident + fill
            # (one wave of whole blocks per table leaves at most tables - 1 places empty: 13 of 148 for 15 tables, the worst of 16)
            assert took <= (1.1 if tables <= 16 else 1.3) * full, (rows, tables, b)


@pytest.mark.parametrize("rows", [1, 63, 64, 65, 1000])
def test_few_rows_and_many_tables(blocks_of, rows):
    for tables in (1, 3, 148, 149, 5000):
        b = blocks_of(rows, tables, 148, 2048)
        assert 1 <= b <= max(1, (rows + 63) // 64)
