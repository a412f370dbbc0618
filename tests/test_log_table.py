"""The logarithm's table (neofiz_gb300/csrc/nf_ilog.h) is read 16 bytes at a time on the device:
its rows ask for that alignment themselves."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "neofiz_gb300", "csrc")

CHECK = """
#include "nf_ilog.h"
static_assert(alignof(nf_log_row) == 16 && sizeof(nf_log_row) == 32, "a row is two 16-byte loads");
int main() { return (uintptr_t)nf_log_rows_h % 16 != 0 || sizeof nf_log_rows_h != 128 * 32; }
"""


def test_table_rows_are_aligned_for_16_byte_loads(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    source, program = tmp_path / "rows.cpp", tmp_path / "rows"
    source.write_text(CHECK)
    subprocess.run([cxx, "-std=c++17", "-I", CSRC, str(source), "-o", str(program)], check=True)
    assert subprocess.run([str(program)]).returncode == 0
