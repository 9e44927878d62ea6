// nb_hilbert.cuh -- octant paths in Hilbert order (shared by the octree's keys
// and the gather after their sort).
//
// The traversals walk the tree for up to 64 bodies that are consecutive in the
// sorted order.  In Morton order a run of 64 often jumps between cells that do
// not touch, which widens its bounding box; along the Hilbert curve consecutive
// cells share a face.  The map below rewrites a path of 3-bit octants digit by
// digit, the same map for every body of a cell, so paths that share their first
// levels still do: the sorted order holds every cell's bodies together either
// way, and the tree built from it is the same.
//
// The digits follow C. Hamilton, "Compact Hilbert Indices" (2006): a state is
// the entry corner e and direction d of the curve in a cell; octant l is the
// w-th cell visited, w = gray^-1(rotr(l ^ e, d + 1)), and the cell's own state
// is e ^ rotl(entry(w), d + 1), (d + direction(w) + 1) mod 3.
#pragma once
#include <cstdint>

namespace nb {

constexpr int kHilbertStates = 24;

// Per state, for each octant (forward) or digit (inverse): the digit (octant)
// and the cell's state << 3, in one byte.
struct HilbertTables {
    uint32_t forward[2 * kHilbertStates];
    uint32_t inverse[2 * kHilbertStates];
};

constexpr int rot3(int v, int by) { return ((v << (by % 3)) | (v >> (3 - by % 3))) & 7; }   // left rotation of 3 bits
constexpr int trailing_ones(int v) {
    int n = 0;
    while (v & 1) { ++n; v >>= 1; }
    return n;
}

constexpr HilbertTables make_hilbert() {
    HilbertTables t{};
    for (int state = 0; state < kHilbertStates; ++state) {
        const int e = state & 7, d = state >> 3;
        for (int l = 0; l < 8; ++l) {
            const int g = rot3((l ^ e), 3 - (d + 1) % 3);   // right rotation by d + 1
            const int w = g ^ (g >> 1) ^ (g >> 2);          // inverse Gray code
            const int even = w == 0 ? 0 : 2 * ((w - 1) / 2);
            const int entry = even ^ (even >> 1);
            const int dir = (w == 0 ? 0 : (w & 1) ? trailing_ones(w) : trailing_ones(w - 1)) % 3;
            const int e2 = e ^ rot3(entry, d + 1), d2 = (d + dir + 1) % 3;
            const uint32_t next = (uint32_t)((d2 * 8 + e2) << 3);
            t.forward[2 * state + (l >> 2)] |= (next | (uint32_t)w) << (8 * (l & 3));
            t.inverse[2 * state + (w >> 2)] |= (next | (uint32_t)l) << (8 * (w & 3));
        }
    }
    return t;
}

#ifdef __CUDACC__
#define NB_HILBERT __host__ __device__ __forceinline__
#else
#define NB_HILBERT inline
#endif

// Rewrites the last D digits of a path by the table, the ones before them as
// they are (the batched forest's galaxy slot).
NB_HILBERT uint64_t hilbert_map(uint64_t path, int D, const uint32_t* table) {
    uint64_t out = path >> (3 * D);
    uint32_t state = 0;
    for (int shift = 3 * (D - 1); shift >= 0; shift -= 3) {
        const uint32_t l = (uint32_t)(path >> shift) & 7u;
        const uint32_t b = (table[2 * state + (l >> 2)] >> (8 * (l & 3))) & 255u;
        out = (out << 3) | (uint64_t)(b & 7u);
        state = b >> 3;
    }
    return out;
}

// The same for a path that a gap between float child bounds cut after `depth` of
// its D digits: the rest stays zero, here as in octant order the first place of
// the last cell that holds the body.  (Mapped as octant 0, it would fall between
// the bodies of that cell's child 0, and the child would be emitted twice.)
NB_HILBERT uint64_t hilbert_map_cut(uint64_t path, int depth, int D, const uint32_t* table) {
    const int rest = 3 * (D - depth);
    return hilbert_map(path, D, table) >> rest << rest;
}

#ifdef __CUDACC__
__constant__ HilbertTables c_hilbert = make_hilbert();

// Copies one direction's table to shared memory (divergent states would
// serialise constant reads); the caller synchronises.
__device__ __forceinline__ void load_hilbert(uint32_t* sh, bool inverse) {
    if (threadIdx.x < 2 * kHilbertStates)
        sh[threadIdx.x] = inverse ? c_hilbert.inverse[threadIdx.x] : c_hilbert.forward[threadIdx.x];
}
#endif

}  // namespace nb
