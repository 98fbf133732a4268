#include "ptree.cuh"

#include "lbvh.cuh"
#include "scan.cuh"

namespace pamo {

namespace {

// The run of leaves of each mesh of a batch: the sorted keys' rank bits change
// at its ends.  Removed faces sort last (their key has a rank no mesh has).
__global__ void k_tree_ranges(const uint32_t *keys, int m, int shift, int n_ranks, int2 *ranges)
{
    chain_wait();
    PAMO_GRID_STRIDE(i, m)
    {
        const uint32_t r = keys[i] >> shift;
        if (r >= (uint32_t)n_ranks) continue;
        if (i == 0 || (keys[i - 1] >> shift) != r) ranges[r].x = (int)i;
        if (i + 1 == m || (keys[i + 1] >> shift) != r) ranges[r].y = (int)i + 1;
    }
}

struct Box {
    float lx, ly, lz, hx, hy, hz;
};

__device__ __forceinline__ void store_box(float4 *boxes, long long node, const Box &b)
{
    boxes[2 * node] = make_float4(b.lx, b.ly, b.lz, 0.f);
    boxes[2 * node + 1] = make_float4(b.hx, b.hy, b.hz, 0.f);
}

__device__ __forceinline__ Box empty_box() { return {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY}; }

// the union over each aligned run of eight lanes, in all of its lanes
__device__ __forceinline__ Box union8(Box b)
{
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        b.lx = fminf(b.lx, __shfl_xor_sync(0xffffffffu, b.lx, o));
        b.ly = fminf(b.ly, __shfl_xor_sync(0xffffffffu, b.ly, o));
        b.lz = fminf(b.lz, __shfl_xor_sync(0xffffffffu, b.lz, o));
        b.hx = fmaxf(b.hx, __shfl_xor_sync(0xffffffffu, b.hx, o));
        b.hy = fmaxf(b.hy, __shfl_xor_sync(0xffffffffu, b.hy, o));
        b.hz = fmaxf(b.hz, __shfl_xor_sync(0xffffffffu, b.hz, o));
    }
    return b;
}

// The whole refit in one launch: a block's 512 leaves give its 64, 8 and 1
// nodes of levels 1-3 (unions over eight lanes at a time), and the last block to
// finish (a ticket, no waiting) does the levels above, one launch's worth of
// latency instead of one atomic per node on the way up.  Bound by latency on
// small meshes, by the leaves' gathers on large ones: 9 / 12 / 18 us a pass with
// the query list, mean over the rounds of meshes of 5k / 200k / 2M faces, against
// 29 / 44 / 83 us for the bottom-up refit of the binary hierarchy.
__global__ void __launch_bounds__(kTreeTile) k_tree_refit(const __grid_constant__ TreeView T,
                                                          const float4 *__restrict__ pts,
                                                          const int4 *__restrict__ tris,
                                                          const uint8_t *__restrict__ sel, int *qlist, int *n_query,
                                                          uint8_t *flags, int m, int *ticket)
{
    chain_wait();
    __shared__ Box s1[64], s2[8];
    __shared__ int s_cnt[kTreeTile / 32], s_first;
    __shared__ bool s_last;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long p = (long long)blockIdx.x * kTreeTile + tid;
    const int f = p < T.L ? T.vals[p] : -1;
    int4 t = f >= 0 ? tris[f] : make_int4(-1, -1, -1, 0);
    Box b = empty_box();
    bool query = false;
    t.w = kLeafDead;
    if (!face_dead(t)) {
        const float4 a = pts[t.x], c = pts[t.y], d = pts[t.z];
        b = {fminf(a.x, fminf(c.x, d.x)), fminf(a.y, fminf(c.y, d.y)), fminf(a.z, fminf(c.z, d.z)),
             fmaxf(a.x, fmaxf(c.x, d.x)), fmaxf(a.y, fmaxf(c.y, d.y)), fmaxf(a.z, fmaxf(c.z, d.z))};
        query = !sel || sel[f];
        t.w = query ? f : -2 - f;
    }
    if (flags && p < m) flags[p] = 0;
    store_box(T.boxes, p, b);  // level 0 starts at node 0 and is padded to whole tiles
    if (p < T.L) T.leaf[p] = t;
    // the querying leaves, a block at a time, in leaf order within the block
    const unsigned ball = __ballot_sync(0xffffffffu, query);
    if (lane == 0) s_cnt[warp] = __popc(ball);
    b = union8(b);
    if ((tid & 7) == 0) {
        s1[tid >> 3] = b;
        store_box(T.boxes, T.off[1] + (long long)blockIdx.x * 64 + (tid >> 3), b);
    }
    __syncthreads();
    if (warp < 2) {
        Box u = union8(s1[tid]);
        if ((tid & 7) == 0) {
            s2[tid >> 3] = u;
            store_box(T.boxes, T.off[2] + (long long)blockIdx.x * 8 + (tid >> 3), u);
        }
    } else if (tid == 64) {
        int n = 0;
        for (int w = 0; w < kTreeTile / 32; ++w) {
            const int c = s_cnt[w];
            s_cnt[w] = n;
            n += c;
        }
        s_first = n && qlist ? atomicAdd(n_query, n) : 0;
    }
    __syncthreads();
    if (query && qlist) qlist[s_first + s_cnt[warp] + __popc(ball & ((1u << lane) - 1u))] = (int)p;
    if (warp == 0) {
        Box u = union8(s2[lane & 7]);
        if (lane == 0) {
            store_box(T.boxes, T.off[3] + (long long)blockIdx.x, u);
            __threadfence();
            s_last = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
        }
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int l = 3; l <= T.top; ++l) {  // level l's nodes padded to whole groups, and their parents
        const int n = T.count[l], padded = (n + 7) & ~7;
        for (int i0 = 0; i0 < padded; i0 += kTreeTile) {
            const int i = i0 + tid;
            Box u = empty_box();
            if (i < n) {
                const float4 lo = __ldcg(&T.boxes[2 * ((long long)T.off[l] + i)]);
                const float4 hi = __ldcg(&T.boxes[2 * ((long long)T.off[l] + i) + 1]);
                u = {lo.x, lo.y, lo.z, hi.x, hi.y, hi.z};
            } else if (i < padded) {
                store_box(T.boxes, (long long)T.off[l] + i, u);
            }
            u = union8(u);
            if (l < T.top && (tid & 7) == 0 && i < padded) store_box(T.boxes, (long long)T.off[l + 1] + (i >> 3), u);
        }
        __syncthreads();
    }
    if (tid == 0) *ticket = 0;
}

}  // namespace

cudaError_t PackedTree::place(void *memory, long long n, cudaStream_t s)
{
    unsigned char *at = static_cast<unsigned char *>(memory);
    auto take = [&](size_t b) {
        void *p = at;
        at += tree_align(b);
        return p;
    };
    keys = static_cast<uint32_t *>(take(4 * (size_t)n));
    keys2 = static_cast<uint32_t *>(take(4 * (size_t)n));
    vals = static_cast<int *>(take(4 * (size_t)n));
    vals2 = static_cast<int *>(take(4 * (size_t)n));
    hist = static_cast<int *>(take(4 * (size_t)tree_hist(n)));
    hist_scratch = static_cast<int *>(take(4 * (size_t)scan_scratch_ints(tree_hist(n))));
    boxes = static_cast<float4 *>(take(2 * sizeof(float4) * (size_t)tree_nodes(n)));
    leaf = static_cast<int4 *>(take(sizeof(int4) * (size_t)n));
    scene = static_cast<int *>(take(64));
    cap = n;
    leaves = 0;
    return scan_scratch_init(hist_scratch, scan_scratch_ints(tree_hist(n)), s);
}

cudaError_t PackedTree::ensure(long long n)
{
    if (n <= cap && keys) return cudaSuccess;
    release();
    const long long c = n > 16 ? n : 16;
    cudaError_t e = cudaMalloc(&mem, bytes(c));
    if (e != cudaSuccess) {
        mem = nullptr;
        return e;
    }
    return place(mem, c, 0);
}

void PackedTree::release()
{
    if (mem) cudaFree(mem);
    *this = PackedTree{};
}

TreeView PackedTree::view() const
{
    TreeView v{};
    v.boxes = boxes;
    v.leaf = leaf;
    v.vals = vals;
    v.L = leaves;
    const int blocks = (leaves + kTreeTile - 1) / kTreeTile;
    int n = blocks * kTreeTile, off = 0, l = 0;
    for (;; ++l) {
        v.off[l] = off;
        v.count[l] = n;
        const int padded = (n + 7) & ~7;
        off += padded;
        if (l >= 3 && (padded <= 8 || l == kTreeMaxLevels - 1)) {
            v.top_groups = padded / 8;
            break;
        }
        n = padded / 8;
    }
    v.top = l;
    return v;
}

cudaError_t tree_build(PackedTree &t, const float4 *pts, const int4 *tris, int m, cudaStream_t s, const int *vslot,
                       int n_ranks, int2 *ranges)
{
    cudaError_t e = t.ensure(m);
    if (e != cudaSuccess) return e;
    t.leaves = m;
    int shift = 0;
    if ((e = morton_order(pts, tris, m, t.scene, t.keys, t.keys2, t.vals, t.vals2, t.hist, t.hist_scratch, vslot,
                          n_ranks, shift, s)) != cudaSuccess)
        return e;
    if (ranges) {
        if ((e = cudaMemsetAsync(ranges, 0, (size_t)n_ranks * sizeof(int2), s)) != cudaSuccess) return e;
        if (m > 0) launch_chained(k_tree_ranges, grid_for(m), kThreads, 0, s, (const uint32_t *)t.keys, m, shift, n_ranks, ranges);
    }
    return cudaGetLastError();
}

cudaError_t tree_refit(PackedTree &t, const float4 *pts, const int4 *tris, const uint8_t *sel, int *qlist,
                       int *n_query, uint8_t *flags, int m, cudaStream_t s)
{
    if (t.leaves <= 0) return cudaSuccess;
    launch_chained(k_tree_refit, (t.leaves + kTreeTile - 1) / kTreeTile, kTreeTile, 0, s, t.view(), pts, tris, sel, qlist,
           n_query, flags, m, t.scene + 10);
    return cudaGetLastError();
}

}  // namespace pamo
