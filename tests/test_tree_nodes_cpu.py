"""What a failed allocation of the octree's node arrays leaves behind: whichever
array is not to be had, on one call and on the next, no capacity is larger than
the arrays it stands for, and a call that succeeds has replaced them all."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "nb_tree_nodes.hpp"
#include <cstdio>
#include <cstdlib>
#include <map>
struct Tree {
    size_t int_cap = 0, cell_cap = 0, hash_cap = 0;
    char *int_level = 0, *int_first = 0, *int_parent = 0, *int_mask = 0, *int_nint = 0, *int_pending = 0, *int_block = 0,
         *int_cell = 0, *int_code = 0, *popc_status = 0, *hkeys = 0, *hvals = 0;
    char *cell_com = 0, *cell_meta = 0, *cell_mass = 0, *cell_count = 0, *cell_lo = 0, *cell_hi = 0, *cell_code = 0;
};
static std::map<void*, size_t> bytes;
static int calls, fail_at;
static int grow(void** p, size_t n) {
    bytes.erase(*p);
    std::free(*p);
    *p = nullptr;
    if (++calls == fail_at) return 2;
    *p = std::malloc(1);
    bytes[*p] = n;
    return 0;
}
static size_t of(void* p) { return p ? bytes.at(p) : 0; }
static bool sound(const Tree& t, size_t tile) {
    for (void* p : {t.int_level, t.int_first, t.int_parent, t.int_mask, t.int_nint, t.int_pending, t.int_block, t.int_cell})
        if (of(p) < t.int_cap * 4) return false;
    if (of(t.int_code) < t.int_cap * 8 || of(t.popc_status) < (t.int_cap + tile - 1) / tile * 8) return false;
    if (of(t.hkeys) < t.hash_cap * 8 || of(t.hvals) < t.hash_cap * 4 || t.hash_cap < 2 * t.int_cap) return false;
    if (t.hash_cap & (t.hash_cap - 1)) return false;
    for (void* p : {t.cell_com, t.cell_meta, t.cell_lo, t.cell_hi})
        if (of(p) < t.cell_cap * 16) return false;
    for (void* p : {t.cell_mass, t.cell_code})
        if (of(p) < t.cell_cap * 8) return false;
    return of(t.cell_count) >= t.cell_cap * 4;
}
int main() {
    const size_t tile = 4096, first = 20000;
    int tried = 0, failed = 0;
    for (size_t second : {30000u, 500000u})
        for (size_t third : {40u, 3000u, 25000u, 600000u})
            for (int i = 0; i <= 20; ++i)
                for (int j = 0; j <= 20; ++j) {
                    Tree t;
                    bytes.clear();
                    const size_t sizes[4] = {first, second, third, third};
                    const int at[4] = {0, i, j, 0};
                    for (int k = 0; k < 4; ++k) {
                        calls = 0;
                        fail_at = at[k];
                        const int e = nb::grow_nodes(t, sizes[k], 2 * sizes[k], tile, grow);
                        if (e) ++failed;
                        if (!sound(t, tile) || (!e && (t.int_cap < sizes[k] || t.cell_cap < 2 * sizes[k]))) {
                            std::printf("unsound: %zu then %zu, failures at %d and %d, call %d\n", second, third, i, j, k);
                            return 1;
                        }
                        ++tried;
                    }
                }
    std::printf("%d %d\n", tried, failed);
    return failed > 1000 ? 0 : 1;
}
"""


def test_no_capacity_exceeds_its_arrays(tmp_path):
    (tmp_path / "nodes.cpp").write_text(SOURCE)
    exe = str(tmp_path / "nodes")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "procedural-universe_gb300", "csrc"),
                    str(tmp_path / "nodes.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
