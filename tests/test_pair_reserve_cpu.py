"""The direct sum's partials where the device has no room for the usual ones:
the launches are planned within less, down to single rows, and only then does
the step fail."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CAP = (1 << 30) // 16

SOURCE = r"""
#include "nb_pair_plan.hpp"
#include <cstdio>
#include <cstdlib>
using namespace nb;
// an allocator with room for argv[3] entries
int main(int argc, char** argv) {
    const int n_pad = atoi(argv[1]);
    const size_t cap = strtoull(argv[2], nullptr, 10), room = strtoull(argv[3], nullptr, 10);
    size_t largest = 0, got = 0;
    int tries = 0;
    const size_t used = pair_reserve(152, n_pad, cap, &largest, [&](size_t need) {
        ++tries;
        if (need > room) return false;
        got = need;
        return true;
    });
    size_t most = 0;   // what the launches planned with it need
    int launches = 0;
    for (int r0 = 0; used && r0 < n_pad / kPairRow; ++launches) {
        const PairFold p = pair_plan(152, n_pad, r0, used, true);
        most = std::max(most, pair_entries(p, n_pad));
        r0 += p.rows;
    }
    printf("%zu %zu %zu %zu %d %d\n", used, got, largest, most, launches, tries);
    return 0;
}
"""


@pytest.fixture(scope="module")
def reserve(tmp_path_factory):
    d = tmp_path_factory.mktemp("pair_reserve")
    (d / "reserve.cpp").write_text(SOURCE)
    exe = str(d / "reserve")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "procedural-universe_gb300", "csrc"),
                    str(d / "reserve.cpp"), "-o", exe], check=True)
    return lambda n_pad, room: [int(x) for x in subprocess.run(
        [exe, str(n_pad), str(CAP), str(room)], capture_output=True, text=True, check=True).stdout.split()]


@pytest.mark.parametrize("n_pad", [22528, 100352, 262144, 1 << 20])
def test_usual_partials_where_there_is_room(reserve, n_pad):
    used, got, largest, most, launches, tries = reserve(n_pad, 1 << 40)
    assert used == CAP and tries == 1 and most == largest
    assert got == largest + (2 * n_pad if launches > 1 else 0)


@pytest.mark.parametrize("n_pad", [22528, 100352, 262144, 1 << 20])
@pytest.mark.parametrize("part", [2, 3, 8, 20])
def test_less_where_there_is_not(reserve, n_pad, part):
    full = reserve(n_pad, 1 << 40)[1]
    room = max(full // part, 6 * n_pad)   # (six entries a body hold a row's partials and the carried sums)
    used, got, largest, most, launches, tries = reserve(n_pad, room)
    assert 0 < used <= CAP and most == largest
    assert got == largest + (2 * n_pad if launches > 1 else 0) and got <= room


def test_no_room_at_all(reserve):
    used, got, _, _, _, tries = reserve(262144, 1000)
    assert used == 0 and got == 0 and tries < 40
