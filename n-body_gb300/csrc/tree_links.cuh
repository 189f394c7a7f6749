// How the records of the octree find their parents (bh.cu; plain functions of
// the radix tree's arrays, so that they also run on the host).
#pragma once

#include "bh.h"

namespace nbody {

constexpr int kMaxLevel = 21;

__host__ __device__ __forceinline__ int bits_set(uint32_t x) {
#ifdef __CUDA_ARCH__
    return __popc(x);
#else
    return __builtin_popcount(x);
#endif
}

__host__ __device__ __forceinline__ int level_of(int delta) {
    const int l = delta / 3;
    return l < kMaxLevel ? l : kMaxLevel;
}

// Several systems packed back to back (an ensemble) are told apart by the
// per-body system id sv.seg. The radix tree then runs over the composite keys
// (system id as 32 leading bits, then the 63-bit key, then the index), so
// delta between bodies of different systems is below 32 and inside a system it
// is 32 + the key's delta. Nodes with delta < 32 join systems and are no
// octree cell (level -1); below them each system's subtree is exactly the tree
// of that system alone. sv.seg == nullptr is the single-system solver.
__host__ __device__ __forceinline__ int level_c(int delta, int base) {
    return delta < base ? -1 : level_of(delta - base);
}

// Whether body i + 1 comes before body i in the order that the tree is built on:
// the sort has not left sorted keys.
__host__ __device__ __forceinline__ bool out_of_order(const uint64_t *__restrict__ k, const int *__restrict__ seg,
                                                      int64_t i) {
    return k[i] > k[i + 1] && (seg == nullptr || seg[i] == seg[i + 1]);
}

// Record index of the cell whose top radix-tree node is p.
__host__ __device__ __forceinline__ int record_of(const BinaryTree &t, const uint32_t *__restrict__ mask,
                                                  const uint32_t *__restrict__ P, int p, int base) {
    const int L = level_c(t.delta[p], base);
    const int lo = t.lo[p];
    return static_cast<int>(P[lo] + bits_set(mask[lo] & ((1u << L) - 1u)));
}

// Octree parent of a record: the nearest radix-tree ancestor that is a cell
// top (the nodes in between split the same cell; at most 6 of them), or -1.
__host__ __device__ __forceinline__ int parent_top(const BinaryTree &t, int p) {
    // At most 6 nodes per octree level inside a system, and at most 32 joining
    // nodes (strictly decreasing delta < 32) above a system's subtree.
    for (int guard = 0; p >= 0 && !t.top[p] && guard < 160; ++guard) p = t.iparent[p];
    return p >= 0 && t.top[p] ? p : -1;
}

constexpr int kNoParent = -1;   // a root
constexpr int kMisplaced = -2;  // the parent's record does not lie before the child's: a broken tree

// Record idx, whose bodies' first key is `key`, into its parent's row of the
// child table (8 places per cell, by key digit, -1 before). p: its radix-tree
// parent. Returns the parent record. A row names only records behind its own,
// whatever the arrays hold, so that no walk down the rows comes round to where
// it was.
__host__ __device__ __forceinline__ int link_child(const BinaryTree &t, const uint32_t *__restrict__ mask,
                                                   const uint32_t *__restrict__ P, int p, int base, uint64_t key,
                                                   int idx, int *__restrict__ kids) {
    p = parent_top(t, p);
    if (p < 0) return kNoParent;
    const int par = record_of(t, mask, P, p, base);
    if (par < 0 || idx <= par) return kMisplaced;
    const int digit = static_cast<int>(key >> (63 - 3 * (level_c(t.delta[p], base) + 1))) & 7;
    kids[8 * static_cast<int64_t>(par) + digit] = idx;
    return par;
}

}  // namespace nbody
