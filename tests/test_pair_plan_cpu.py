"""The launches that the direct sum's pair kernel is cut into, at sizes no GPU
test reaches: every launch fits its partials, the launches cover every row, and
the kernel's 32-bit count of units is the exact one wherever the kernel counts."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ROW, ROW_TILES, CAP = 1024, 8, (1 << 30) // 16

SOURCE = r"""
#include "nb_pair_plan.hpp"
#include <cstdio>
#include <cstdlib>
using namespace nb;
// each launch of a state: per row0 rows units entries, the 64-bit unit count at
// some rows and the 32-bit one
int main(int argc, char** argv) {
    const int sms = atoi(argv[1]), n_pad = atoi(argv[2]), most = atoi(argv[4]);
    const size_t cap = strtoull(argv[3], nullptr, 10);
    const int rows = n_pad / kPairRow;
    int row = 0;
    for (int launch = 0; row < rows && launch < most; ++launch) {
        const PairFold p = pair_plan(sms, n_pad, row, cap, true);
        printf("L %d %d %d %lld %zu\n", p.per, p.row0, p.rows, pair_units(p, n_pad), pair_entries(p, n_pad));
        for (int k = 0; k <= p.rows; k += p.rows > 8 ? p.rows / 8 : 1)
            printf("U %d %lld %d\n", k, pair_units_before<long long>(row + k, row, rows, p.per),
                   pair_units_before<int>(row + k, row, rows, p.per));
        row += p.rows;
    }
    printf("E %d %zu\n", row, kPairMax);
    return 0;
}
"""


@pytest.fixture(scope="module")
def planner(tmp_path_factory):
    d = tmp_path_factory.mktemp("pair_plan")
    (d / "plan.cpp").write_text(SOURCE)
    exe = str(d / "plan")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I",
                    os.path.join(ROOT, "procedural-universe_gb300", "csrc"), str(d / "plan.cpp"), "-o", exe], check=True)
    return exe


def units(row0, rows_of_launch, rows, per):
    """Row q has (rows - q) * ROW_TILES source tiles, in units of `per`."""
    return sum(-(-(rows - q) * ROW_TILES // per) for q in range(row0, row0 + rows_of_launch))


@pytest.mark.parametrize("cap", [CAP, CAP // 64])
@pytest.mark.parametrize("n_pad", [10240, 20480, 262144, 378880, 1 << 20, 5_000_192, 1 << 24, 23_700_480, 40_001_536,
                                   50_001_920, 60_000_256, (1 << 31) - 4096])
def test_launches_fit_and_cover_the_rows(planner, n_pad, cap):
    rows, most = n_pad // ROW, 1 << 20 if n_pad <= 1 << 24 else 3
    out = subprocess.run([planner, "152", str(n_pad), str(cap), str(most)], capture_output=True, text=True, check=True).stdout
    row, checked = 0, 0
    for line in out.splitlines():
        f = [int(x) for x in line.split()[1:]]
        if line[0] == "L":
            per, row0, r, u, entries = f
            assert row0 == row and 1 <= r <= rows - row
            if checked < 50:   # (the exact count walks the rows)
                assert u == units(row0, r, rows, per)
                checked += 1
            # a row's targets, and its sources: the bodies behind it
            need = u * ROW + r * n_pad - ROW * (r * row0 + r * (r + 1) // 2)
            assert entries == need
            assert entries <= cap or r == 1   # (one row is taken whatever it needs)
            row += r
        elif line[0] == "U":
            if n_pad <= 1 << 24:   # the sizes that the kernel takes
                assert f[1] == f[2]
        else:
            assert f[1] == 1 << 24
            assert f[0] == row
            if n_pad <= 1 << 24:
                assert row == rows
