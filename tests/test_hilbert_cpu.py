"""The order of octant paths along the Hilbert curve, with paths that a gap
between float child bounds cut short: the map is undone exactly, every cell's
bodies stay together, and a path that ends in a cell comes before those that go
on, so that the cells' nodes start where they would in octant order."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "nb_hilbert.cuh"
#include <algorithm>
#include <cstdio>
#include <map>
#include <random>
#include <vector>
using namespace nb;
struct Body {
    uint64_t path, key;
    int depth;
};
int main() {
    static const HilbertTables t = make_hilbert();
    std::mt19937_64 rng(5);
    for (int trial = 0; trial < 400; ++trial) {
        const int D = trial % 2 ? 21 : 4 + trial % 7, n = 400;
        std::vector<Body> b(n);
        for (Body& x : b) {
            x.depth = rng() % 5 == 0 ? (int)(rng() % D) : D;   // one in five is cut
            x.path = 0;
            for (int l = 0; l < D; ++l) {   // few octants a level: cells hold many bodies
                const uint64_t o = rng() % 3 ? rng() % 2 * 7 : rng() % 8;
                x.path = (x.path << 3) | (l < x.depth ? o : 0);
            }
            x.key = hilbert_map_cut(x.path, x.depth, D, t.forward);
            if (hilbert_map_cut(x.key, x.depth, D, t.inverse) != x.path) return std::printf("not undone\n"), 1;
            if (x.depth == D && x.key != hilbert_map(x.path, D, t.forward)) return std::printf("full path\n"), 1;
        }
        std::stable_sort(b.begin(), b.end(), [](const Body& x, const Body& y) { return x.key < y.key; });
        for (int level = 1; level <= D; ++level) {
            // the bodies that reach a cell of this level follow one another
            std::map<uint64_t, int> last;
            for (int s = 0; s < n; ++s) {
                if (b[s].depth < level) continue;
                const uint64_t cell = b[s].path >> (3 * (D - level));
                const auto f = last.find(cell);
                // bodies cut above the cell may share its first key only at the finest cells
                for (int q = f == last.end() ? s : f->second + 1; q < s; ++q)
                    if (b[q].key != b[f->second].key) return std::printf("cell parted: level %d of %d\n", level, D), 1;
                last[cell] = s;
            }
        }
    }
    std::printf("ok\n");
    return 0;
}
"""


def test_cut_paths_come_first_in_their_cell(tmp_path):
    (tmp_path / "hilbert.cpp").write_text(SOURCE)
    exe = str(tmp_path / "hilbert")
    subprocess.run(["g++", "-std=c++17", "-O2", "-x", "c++", "-I",
                    os.path.join(ROOT, "procedural-universe_gb300", "csrc"), str(tmp_path / "hilbert.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
