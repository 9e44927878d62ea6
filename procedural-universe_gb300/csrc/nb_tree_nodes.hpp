// nb_tree_nodes.hpp -- growing the octree's node arrays (nb_tree.cu).  Plain C++,
// so that what a failed allocation leaves behind is tested on the host.
#pragma once
#include <cstddef>
#include <cstdint>

namespace nb {

// Makes room for n_int internal nodes and n_cells cells, a quarter more each, by
// grow(pointer, bytes), which replaces the buffer at the pointer and returns 0, or
// an error that is returned here.  A capacity is zero from before its first
// array is replaced until the last one is there: after a failure no later build
// takes the arrays (or the table of internal nodes) for larger than they are, and
// the next call replaces them all.  scan_tile: nodes a tile of the child-count scan.
template <class Tree, class Grow>
auto grow_nodes(Tree& t, size_t n_int, size_t n_cells, size_t scan_tile, Grow grow)
    -> decltype(grow((void**)nullptr, (size_t)0)) {
#define NB_GROW(p, bytes) \
    if (const auto e = grow((void**)&(p), (bytes))) return e
    if (n_int > t.int_cap) {
        const size_t cap = n_int + n_int / 4 + 64;
        t.int_cap = t.hash_cap = 0;
        NB_GROW(t.int_level, cap * 4);
        NB_GROW(t.int_first, cap * 4);
        NB_GROW(t.int_parent, cap * 4);
        NB_GROW(t.int_mask, cap * 4);
        NB_GROW(t.int_nint, cap * 4);
        NB_GROW(t.int_pending, cap * 4);
        NB_GROW(t.int_block, cap * 4);
        NB_GROW(t.int_cell, cap * 4);
        NB_GROW(t.int_code, cap * 8);
        // internal nodes can outnumber bodies (chains of one-child nodes above
        // close pairs): the child-count scan's status is sized by them
        NB_GROW(t.popc_status, (cap + scan_tile - 1) / scan_tile * sizeof(unsigned long long));
        size_t h = 1024;
        while (h < 2 * cap) h <<= 1;
        NB_GROW(t.hkeys, h * 8);
        NB_GROW(t.hvals, h * 4);
        t.hash_cap = h;
        t.int_cap = cap;
    }
    if (n_cells > t.cell_cap) {
        const size_t cap = n_cells + n_cells / 4 + 64;
        t.cell_cap = 0;
        NB_GROW(t.cell_com, cap * 16);
        NB_GROW(t.cell_meta, cap * 16);
        NB_GROW(t.cell_mass, cap * 8);
        NB_GROW(t.cell_count, cap * 4);
        NB_GROW(t.cell_lo, cap * 16);
        NB_GROW(t.cell_hi, cap * 16);
        NB_GROW(t.cell_code, cap * 8);
        t.cell_cap = cap;
    }
#undef NB_GROW
    return {};
}

}  // namespace nb
