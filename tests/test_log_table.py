"""The integer logarithm (neofiz_gb300/csrc/nf_ilog.h): its table is read 16 bytes at a time on the
device, and its rows ask for that alignment themselves; its sum lies as close to nf_log_dd's as
the rounding test takes for granted."""
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


# The two roundings' bounds are 240 and 115 units of 2^-84, so the sums' distance is below 355; a
# unit more for the magnitude, which is formed by complement.
SUMS = """
#include <cstdio>
#include "nf_ilog.h"
typedef __int128 Wide;
static Wide fixed84(double x) {                     // x 2^84, rounded
    if (x == 0.0) return 0;
    int e;
    const Wide m = (Wide)(int64_t)ldexp(frexp(x, &e), 53);
    const int s = e - 53 + 84;
    return s >= 0 ? m << s : s < -80 ? 0 : (m + ((Wide)1 << (-s - 1))) >> -s;
}
int main() {
    uint64_t state = 7;
    long used = 0;
    double most = 0.0;
    for (int i = 0; i < 4000000; i++) {
        uint64_t z = (state += 0x9E3779B97F4A7C15ULL);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
        const uint64_t field = 1023 + (i & 1 ? (int)(z >> 58) % 17 - 8 : (int)(z >> 57) - 64);
        double x;
        const uint64_t bits = (field << 52) | (z & 0xfffffffffffffULL);
        memcpy(&x, &bits, 8);
        nf_ilog v;
        if (!nf_ilog_of(x, &v)) continue;
        const unsigned __int128 w = ((unsigned __int128)v.w2 << 64) | ((uint64_t)v.w1 << 32) | v.w0;
        const Wide sum = v.neg ? -(Wide)(w >> v.n) : (Wide)(w >> v.n);
        double hi, lo;
        nf_log_dd(x, &hi, &lo);
        const Wide d = sum - (fixed84(hi) + fixed84(lo));
        most = fmax(most, (double)(d < 0 ? -d : d));
        used++;
    }
    printf("%ld %.0f", used, most);
}
"""


def test_the_sum_lies_within_its_bound_of_the_double_double(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    source, program = tmp_path / "sums.cpp", tmp_path / "sums"
    source.write_text(SUMS)
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, str(source), "-o",
                    str(program)], check=True)
    used, most = subprocess.run([str(program)], capture_output=True, text=True,
                                check=True).stdout.split()
    assert int(used) > 3900000 and float(most) <= 356
