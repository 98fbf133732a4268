// Morton order of a mesh's faces, and the linear BVH over it (stage 3 and the mesh
// distance of many samples).
//
// Build: 30-bit Morton code of each face's box centre (10 bits per axis over the
// scene box) -> stable LSD radix sort (4 x 8-bit digits, hand written) ->
// Karras hierarchy over 64-bit keys (code << 32 | sorted position) -> bottom-up
// refit.  Internal node i (0 <= i < L-1) stores both child boxes inline (64 B),
// so traversal reads one node per step and tests the two children.
//
// The leaf set is fixed per build (faces live at the build, sorted by their
// geometry then).  Refit recomputes every leaf box from the current geometry (a dead
// face gets the empty box lo=+inf, hi=-inf, which overlaps nothing) and rebuilds the
// inner boxes.
#pragma once

#include "common.cuh"

namespace pamo {

constexpr int kRefitTile = 256;  // leaves per refit block
// radix-sort tile of lbvh_build (threads x items per thread); Lbvh::hist holds
// 256 counts per tile
constexpr int kLbvhSortThreads = 256;
constexpr int kLbvhSortItems = 8;
constexpr int kLbvhSortTile = kLbvhSortThreads * kLbvhSortItems;
constexpr int kRefitTileShift = 8;
static_assert(kRefitTile == 1 << kRefitTileShift, "refit tile");

struct __align__(16) BvhNode {
    float4 llo;  // .w = left child (int bits): >= 0 internal node, < 0 leaf ~position
    float4 lhi;
    float4 rlo;  // .w = right child
    float4 rhi;
};

struct Lbvh {
    long long cap = 0;        // faces
    uint32_t *keys = nullptr;  // morton keys (ping)
    uint32_t *keys2 = nullptr;
    int *vals = nullptr;  // face index per sorted position (ping)
    int *vals2 = nullptr;
    int *hist = nullptr;        // radix digit counts [256 * tiles]
    int *hist_scratch = nullptr;
    BvhNode *nodes = nullptr;   // [cap]
    // [2*cap]: internal nodes then leaves; (p << 2) | tile << 1 | is_right, -1 for
    // the root, where `tile` says that the parent's leaves all lie in one aligned
    // run of kRefitTile leaves (merged in shared memory by k_refit)
    int *parent = nullptr;
    int *flags = nullptr;       // [cap] refit arrival counters
    int *scene = nullptr;       // 6 ordered ints + n_dead + n_leaves
    int sort_tiles = 0;
    long long leaves_built = 0;  // faces of the last build: bound on the leaf count

    cudaError_t ensure(long long n_faces);
    // the arrays in the caller's memory (bytes(n) of it, 256-byte aligned) instead;
    // such a hierarchy is not released
    cudaError_t place(void *memory, long long n_faces, cudaStream_t s);
    static size_t bytes(long long n_faces);
    void release();
};

// The order of the faces [0, m) by the Morton code of their box centre, 10 bits
// per axis over the scene box (written to scene[0..5], the removed faces' count
// to scene[6]), by a stable radix sort: keys and vals (face indices) ascending,
// removed faces last.  For a batch of meshes (vslot: each vertex's mesh rank <
// n_ranks) the rank is the top of the key, from bit rank_shift up, and the codes
// have fewer bits.  hist: 256 counts per tile of kLbvhSortTile faces.
cudaError_t morton_order(const float4 *pts, const int4 *tris, int m, int *scene, uint32_t *keys, uint32_t *keys2,
                         int *vals, int *vals2, int *hist, int *hist_scratch, const int *vslot, int n_ranks,
                         int &rank_shift, cudaStream_t s);

// Builds the hierarchy for faces [0, m): leaves are the faces live in `tris`
// (the round input), ordered by the Morton code of their box centre.
cudaError_t lbvh_build(Lbvh &b, const float4 *pts, const int4 *tris, int m, cudaStream_t s);

// Recomputes all boxes from the current geometry (pts, tris).
cudaError_t lbvh_refit(Lbvh &b, const float4 *pts, const int4 *tris, int m, cudaStream_t s);

}  // namespace pamo
