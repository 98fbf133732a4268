// Packed tree over the faces of a mesh: an eight-way box hierarchy without
// pointers, used by the intersection queries.
//
// The faces are ordered by the Morton code of their box centres
// (morton_order, lbvh.cuh); leaf p is the p-th of them.  Node n of level l covers
// the leaves [n 8^l, (n + 1) 8^l), so a node's children are the eight nodes
// 8 n .. 8 n + 7 one level down, and neither the build nor the refit has any
// structure to compute: the build is the sort, the refit one launch.  A level's
// boxes lie one after another (two float4 each), so the eight lanes of a group
// read a node's children as one 256-byte run and test one box each: a walk has a
// third of the levels of a binary one, and its length in dependent loads is what
// bounds a query (k_query states both times).
//
// The leaf set is fixed per build; a caller that removes and renumbers faces
// keeps the order by rewriting vals (-1 for a removed face).  A leaf without a
// live face has the empty box lo = +inf, hi = -inf, which overlaps nothing.
#pragma once

#include "common.cuh"
#include "lbvh.cuh"
#include "scan.cuh"

namespace pamo {

constexpr int kTreeTile = 512;     // leaves per refit block: three levels
constexpr int kTreeMaxLevels = 9;  // levels 0 .. 8; level 8 may hold several groups of eight

struct TreeView {
    float4 *boxes;  // node i of level l: boxes[2 (off[l] + i)] = lo, [.. + 1] = hi
    int4 *leaf;     // per leaf: corner indices, and in .w the face (see leaf_code)
    const int *vals;
    int L;          // leaves
    int top;        // top level
    int top_groups; // groups of eight nodes there (one unless top == kTreeMaxLevels - 1)
    int off[kTreeMaxLevels];
    int count[kTreeMaxLevels];  // nodes that cover a leaf or its tile's padding

    // A block's copy of what a walk needs of each level: where its boxes start, and the
    // last node that covers a leaf.  A walk enters none beyond: the nodes of the levels'
    // padding (which it may read) are empty, but a query box that is NaN or infinite on
    // all axes is apart from none, and the children of padding lie outside the tree.
    __device__ __forceinline__ void levels(int2 *shared) const
    {
#pragma unroll
        for (int l = 0; l < kTreeMaxLevels; ++l)
            if (threadIdx.x == l) shared[l] = make_int2(off[l], (L - 1) >> (3 * l));
        __syncthreads();
    }
};

// leaf_code: the face of a leaf, and whether it is selected (queries, and not
// queried twice for one pair): f >= 0 selected, -2 - f not selected, kLeafDead none.
constexpr int kLeafDead = (int)0x80000000;
__device__ __forceinline__ int leaf_face(int code) { return code >= 0 ? code : -2 - code; }

constexpr long long tree_nodes(long long n)  // box slots for n leaves, the levels' padding included
{
    const long long p0 = (n + kTreeTile - 1) / kTreeTile * kTreeTile;
    return p0 + p0 / 8 + p0 / 64 + (p0 / 512 + 8) + (p0 / 512 + 64) / 7 + 64;
}

struct PackedTree {
    long long cap = 0;    // faces
    void *mem = nullptr;  // owned by ensure()
    uint32_t *keys = nullptr, *keys2 = nullptr;
    int *vals = nullptr, *vals2 = nullptr;  // face of each leaf (and the sort's other buffer)
    int *hist = nullptr, *hist_scratch = nullptr;
    float4 *boxes = nullptr;
    int4 *leaf = nullptr;
    int *scene = nullptr;  // [16]: the scene box, dead faces; [10] the refit's ticket
    int leaves = 0;        // of the last build

    cudaError_t ensure(long long n_faces);
    // the arrays in the caller's memory (bytes(n) of it, 256-byte aligned) instead
    cudaError_t place(void *memory, long long n_faces, cudaStream_t s);
    static constexpr size_t bytes(long long n);
    void release();
    TreeView view() const;
};

constexpr size_t tree_align(size_t x) { return (x + 255) & ~size_t(255); }
constexpr long long tree_hist(long long n) { return 256 * ((n + kLbvhSortTile - 1) / kLbvhSortTile); }

constexpr size_t PackedTree::bytes(long long n)
{
    return 4 * tree_align(4 * (size_t)n) + tree_align(4 * (size_t)tree_hist(n)) +
           tree_align(4 * (size_t)scan_scratch_ints(tree_hist(n))) +
           tree_align(2 * sizeof(float4) * (size_t)tree_nodes(n)) + tree_align(sizeof(int4) * (size_t)n) + 256;
}

// Orders the faces [0, m) of the round input.  For a batch of meshes, vslot
// gives each vertex's mesh rank (< n_ranks): a mesh's leaves are then one run,
// written to ranges[rank] (first leaf, end).
cudaError_t tree_build(PackedTree &t, const float4 *pts, const int4 *tris, int m, cudaStream_t s,
                       const int *vslot = nullptr, int n_ranks = 0, int2 *ranges = nullptr);

// Every box and leaf record from the current geometry.  sel (per face, may be
// null: all) selects the faces that query; the leaves of the live ones are
// appended to qlist and counted in n_query (zero before).  flags[0, m) are
// cleared if given.
cudaError_t tree_refit(PackedTree &t, const float4 *pts, const int4 *tris, const uint8_t *sel, int *qlist,
                       int *n_query, uint8_t *flags, int m, cudaStream_t s);

// A group of eight lanes walks the tree depth first: at each step it stands at
// a group of eight sibling nodes (level lvl, nodes 8 g .. 8 g + 7), one lane per
// node; the hits of levels 1 .. 8 not yet entered are bits of `pend` (eight per
// level), so the lowest set bit is the deepest pending node and no stack is
// needed.  Every node is entered at most once, so a walk always ends.
struct TreeWalk {
    int lvl, g, topg;
    unsigned long long pend;
    bool run;

    __device__ __forceinline__ void start(const TreeView &T, bool has)
    {
        lvl = T.top;
        g = 0;
        topg = 0;
        pend = 0;
        run = has;
    }
    // hits: this group's eight bits for the nodes just tested
    __device__ __forceinline__ void advance(const TreeView &T, unsigned hits)
    {
        if (lvl > 0) pend |= (unsigned long long)hits << (8 * (lvl - 1));
        if (pend == 0) {
            run = ++topg < T.top_groups;
            lvl = T.top;
            g = topg;
            return;
        }
        const int b = __ffsll((long long)pend) - 1;
        const int up = (b >> 3) + 1;  // the level of the pending node, >= lvl
        pend &= pend - 1;
        g = ((g >> (3 * (up - lvl))) << 3) + (b & 7);
        lvl = up - 1;
    }
};

}  // namespace pamo
