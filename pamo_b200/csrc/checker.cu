// Acceptance checks of a simplified mesh, on the device:
//   * pamo_check_mesh: exact-predicate self-intersection test of every pair of
//     faces whose closed bounding boxes overlap, degenerate faces, and the
//     manifold / watertight checks (edges in exactly two faces, once each way;
//     one closed fan of faces around every vertex);
//   * pamo_mesh_distance: one-sided distance from a mesh's surface to another
//     mesh by dense sampling (the Hausdorff and Chamfer terms of the
//     reference's metrics.py:31-51), with an upper bound from the sampling
//     density.
// The role model of the first is the reference's CGAL self-intersection script
// (simp_cuda/safe_project/scripts/cgal_intersect/main.cpp:19-111): faces that
// share a vertex or an edge intersect only beyond what they share.
//
// Both walk the faces' packed tree (ptree.cuh), a group of eight lanes per face or
// sample; many samples walk a binary hierarchy (lbvh.cuh) instead, one thread each.
// A call's scratch is one allocation from the device's stream-ordered
// pool: with a dozen cudaMalloc / cudaFree pairs a call, which synchronise the
// device, the check of a 350k-face mesh took 12 to 60 ms, of which its kernels 5.
#include <cfloat>
#include <vector>

#include "exact.cuh"
#include "lbvh.cuh"
#include "ptree.cuh"
#include "scan.cuh"

namespace pamo {
namespace {

using exact::P3;

enum CheckCounter {
    C_PAIRS = 0,       // intersecting pairs
    C_FACES,           // faces in an intersecting pair
    C_DEGENERATE,      // faces with a repeated index or collinear corners
    C_BOUNDARY,        // half-edges without a reverse half-edge
    C_NONMANIFOLD,     // half-edges of an edge in more than two faces or twice one way
    C_BAD_VERTEX,      // vertices whose faces do not form one closed fan
    C_UNREFERENCED,    // vertices in no live face
    C_CANDIDATES,      // face pairs with overlapping boxes
    C_DEAD,            // faces (-1, -1, -1)
    C_ERROR,           // always 0 (a walk of the tree ends by itself)
    C_BAD_INDEX,       // an index outside [0, n_pts) in a live face
    C_COUNT
};

__global__ void k_ck_convert(const float *pts, int n, const int *tris, int m, float4 *p4, int4 *t4)
{
    const long long N = n > m ? n : m;
    PAMO_GRID_STRIDE(i, N)
    {
        if (i < n) p4[i] = make_float4(pts[3 * i], pts[3 * i + 1], pts[3 * i + 2], 0.f);
        if (i < m) t4[i] = make_int4(tris[3 * i], tris[3 * i + 1], tris[3 * i + 2], 0);
    }
}

__global__ void k_ck_validate(const int4 *tris, int m, int n, unsigned long long *cnt)
{
    PAMO_GRID_STRIDE(f, m)
    {
        const int4 t = tris[f];
        if (face_dead(t)) {
            atomicAdd(&cnt[C_DEAD], 1ULL);
            continue;
        }
        if (t.x < 0 || t.x >= n || t.y < 0 || t.y >= n || t.z < 0 || t.z >= n) atomicAdd(&cnt[C_BAD_INDEX], 1ULL);
    }
}

__device__ __forceinline__ void load_tri(const float4 *p, int4 t, P3 *T, int *idx)
{
    idx[0] = t.x; idx[1] = t.y; idx[2] = t.z;
    for (int k = 0; k < 3; ++k) {
        const float4 q = p[idx[k]];
        T[k] = {q.x, q.y, q.z};
    }
}

// whether a face is live and not degenerate (those are tested); counts
__global__ void k_ck_degenerate(const float4 *p, const int4 *tris, int m, uint8_t *ok, unsigned long long *cnt)
{
    PAMO_GRID_STRIDE(f, m)
    {
        const int4 t = tris[f];
        uint8_t good = 0;
        if (!face_dead(t)) {
            P3 T[3];
            int idx[3];
            load_tri(p, t, T, idx);
            good = exact::tri_degenerate(T, idx) ? 0 : 1;
            if (!good) atomicAdd(&cnt[C_DEGENERATE], 1ULL);
        }
        ok[f] = good;
    }
}

__device__ __noinline__ bool pair_intersects(const float4 *p, int4 ta, int4 tb)
{
    P3 A[3], B[3];
    int ia[3], ib[3];
    load_tri(p, ta, A, ia);
    load_tri(p, tb, B, ib);
    return exact::faces_intersect(A, ia, B, ib);
}

// Every pair f < g of tested faces with overlapping closed boxes: a group of eight
// lanes walks the tree for each f, and a warp's pairs gather in shared memory
// until 32 of them can be tested, one a lane.  With one thread per face, testing
// each leaf as it met it on a binary hierarchy, most lanes of a warp waited while
// one evaluated a predicate: 5.0 ms on a 350k-face torus; the whole check of that
// mesh takes 1.4 ms so.
constexpr int kPairThreads = 128;

__global__ void __launch_bounds__(kPairThreads) k_ck_pairs(const __grid_constant__ TreeView T,
                                                           const int *__restrict__ qlist, const int *n_query,
                                                           const float4 *__restrict__ p, uint8_t *flags,
                                                           unsigned long long *cnt)
{
    __shared__ int2 s_pairs[kPairThreads / 32][64];  // leaves of f and g
    __shared__ int2 s_lvl[kTreeMaxLevels];
    T.levels(s_lvl);
    int2 *buf = s_pairs[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31, gl = lane & 7, shift = lane & 24;
    const unsigned below = (1u << lane) - 1u;
    const int N = *n_query;
    int held = 0;
    unsigned long long cand = 0, found = 0;
    auto test = [&](int n) {
        bool hit = false;
        if (lane < n) {
            const int4 a = T.leaf[buf[lane].x], b = T.leaf[buf[lane].y];
            hit = pair_intersects(p, a, b);
            if (hit) flags[a.w] = flags[b.w] = 1;
        }
        cand += n;
        found += __popc(__ballot_sync(0xffffffffu, hit));
    };
    const long long warps = (long long)gridDim.x * (kPairThreads / 32);
    for (long long w = ((long long)blockIdx.x * kPairThreads + threadIdx.x) >> 5; w * 4 < N; w += warps) {
        const long long k = w * 4 + (lane >> 3);
        const bool has = k < N;
        const int q = has ? qlist[k] : 0;
        const int f = T.leaf[q].w;
        const float4 qlo = T.boxes[2 * (size_t)q], qhi = T.boxes[2 * (size_t)q + 1];
        TreeWalk wk;
        wk.start(T, has);
        while (__any_sync(0xffffffffu, wk.run)) {
            bool hit = false, emit = false;
            const int node = 8 * wk.g + gl;
            if (wk.run) {
                const int2 level = s_lvl[wk.lvl];
                const size_t b = 2 * ((size_t)level.x + node);
                const float4 lo = T.boxes[b], hi = T.boxes[b + 1];
                const bool leaf = wk.lvl == 0 && node < T.L;
                const int g = leaf ? T.leaf[node].w : kLeafDead;
                hit = !(hi.x < qlo.x || qhi.x < lo.x || hi.y < qlo.y || qhi.y < lo.y || hi.z < qlo.z || qhi.z < lo.z) &&
                      node <= level.y;
                emit = hit && g > f;  // selected leaves have their face's number, the others a negative one
            }
            const unsigned hits = __ballot_sync(0xffffffffu, hit), em = __ballot_sync(0xffffffffu, emit);
            if (em) {
                if (emit) buf[held + __popc(em & below)] = make_int2(q, node);
                held += __popc(em);
                __syncwarp();
                if (held >= 32) {
                    test(32);
                    held -= 32;
                    const int2 rest = buf[32 + lane];
                    __syncwarp();
                    buf[lane] = rest;
                    __syncwarp();
                }
            }
            if (wk.run) wk.advance(T, (hits >> shift) & 255u);
        }
    }
    if (held > 0) test(held);
    if (lane == 0 && cand) atomicAdd(&cnt[C_CANDIDATES], cand);
    if (lane == 0 && found) atomicAdd(&cnt[C_PAIRS], found);
}

__global__ void k_ck_flagged(const uint8_t *flags, int m, unsigned long long *cnt)
{
    int n = 0;
    PAMO_GRID_STRIDE(f, m) n += flags[f];
    n = __reduce_add_sync(0xffffffffu, n);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(&cnt[C_FACES], (unsigned long long)n);
}

__global__ void k_ck_count(const int4 *tris, int m, int *deg_v)
{
    PAMO_GRID_STRIDE(f, m)
    {
        const int4 t = tris[f];
        if (face_dead(t)) continue;
        atomicAdd(&deg_v[t.x], 1);
        atomicAdd(&deg_v[t.y], 1);
        atomicAdd(&deg_v[t.z], 1);
    }
}

__global__ void k_ck_fill(const int4 *tris, int m, const int *first, int *cursor, int *faces_of)
{
    PAMO_GRID_STRIDE(f, m)
    {
        const int4 t = tris[f];
        if (face_dead(t)) continue;
        faces_of[first[t.x] + atomicAdd(&cursor[t.x], 1)] = (int)f;
        faces_of[first[t.y] + atomicAdd(&cursor[t.y], 1)] = (int)f;
        faces_of[first[t.z] + atomicAdd(&cursor[t.z], 1)] = (int)f;
    }
}

__device__ __forceinline__ int corner(int4 t, int k) { return k == 0 ? t.x : (k == 1 ? t.y : t.z); }

// does face t contain the directed edge a -> b
__device__ __forceinline__ bool has_directed(int4 t, int a, int b)
{
    return (t.x == a && t.y == b) || (t.y == a && t.z == b) || (t.z == a && t.x == b);
}

// per half-edge a -> b of every live face: the faces around a holding a -> b
// (itself included) and b -> a
__global__ void k_ck_edges(const int4 *tris, int m, const int *first, const int *faces_of, unsigned long long *cnt)
{
    PAMO_GRID_STRIDE(h, 3LL * m)
    {
        const int f = (int)(h / 3), k = (int)(h % 3);
        const int4 t = tris[f];
        if (face_dead(t)) continue;
        const int a = corner(t, k), b = corner(t, (k + 1) % 3);
        int same = 0, back = 0;
        for (int s = first[a]; s < first[a + 1]; ++s) {
            const int4 u = tris[faces_of[s]];
            same += has_directed(u, a, b);
            back += has_directed(u, b, a);
        }
        if (same > 1 || back > 1) atomicAdd(&cnt[C_NONMANIFOLD], 1ULL);
        else if (back == 0) atomicAdd(&cnt[C_BOUNDARY], 1ULL);
    }
}

// per vertex: following the faces around v across their shared edges (face
// (v, x, y) is followed by the face holding v -> y) must run through all of
// them once and come back
__global__ void k_ck_fans(const int4 *tris, int n, const int *first, const int *faces_of, unsigned long long *cnt)
{
    PAMO_GRID_STRIDE(vv, n)
    {
        const int v = (int)vv;
        const int s0 = first[v], d = first[v + 1] - s0;
        if (d == 0) {
            atomicAdd(&cnt[C_UNREFERENCED], 1ULL);
            continue;
        }
        auto next_of = [&](int4 t) {  // y of the rotation (v, x, y)
            return t.x == v ? t.z : (t.y == v ? t.x : t.y);
        };
        const int start = faces_of[s0];
        int cur = start, steps = 0;
        bool ok = true;
        while (true) {
            const int y = next_of(tris[cur]);
            int nxt = -1, found = 0;
            for (int s = s0; s < s0 + d; ++s) {
                const int g = faces_of[s];
                if (has_directed(tris[g], v, y)) {
                    nxt = g;
                    ++found;
                }
            }
            if (found != 1) {
                ok = false;
                break;
            }
            ++steps;
            cur = nxt;
            if (cur == start || steps > d) break;
        }
        if (!ok || cur != start || steps != d) atomicAdd(&cnt[C_BAD_VERTEX], 1ULL);
    }
}

// ------------------------------------------------------------------ distances
struct D3 {
    double x, y, z;
};
__device__ __forceinline__ D3 dsub(D3 a, D3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ double ddot(D3 a, D3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ D3 dat(float4 p) { return {p.x, p.y, p.z}; }

// squared distance from p to the closed triangle abc: the closest point by the
// Voronoi regions of the triangle's vertices, edges and face (Ericson,
// Real-Time Collision Detection, 2005, sec. 5.1.5)
__device__ double point_tri_d2(D3 p, D3 a, D3 b, D3 c)
{
    const D3 ab = dsub(b, a), ac = dsub(c, a), ap = dsub(p, a);
    const double d1 = ddot(ab, ap), d2 = ddot(ac, ap);
    D3 q;
    if (d1 <= 0.0 && d2 <= 0.0) {
        q = a;
    } else {
        const D3 bp = dsub(p, b);
        const double d3 = ddot(ab, bp), d4 = ddot(ac, bp);
        if (d3 >= 0.0 && d4 <= d3) {
            q = b;
        } else {
            const double vc = d1 * d4 - d3 * d2;
            if (vc <= 0.0 && d1 >= 0.0 && d3 <= 0.0) {
                const double v = d1 / (d1 - d3);
                q = {a.x + v * ab.x, a.y + v * ab.y, a.z + v * ab.z};
            } else {
                const D3 cp = dsub(p, c);
                const double d5 = ddot(ab, cp), d6 = ddot(ac, cp);
                if (d6 >= 0.0 && d5 <= d6) {
                    q = c;
                } else {
                    const double vb = d5 * d2 - d1 * d6;
                    if (vb <= 0.0 && d2 >= 0.0 && d6 <= 0.0) {
                        const double w = d2 / (d2 - d6);
                        q = {a.x + w * ac.x, a.y + w * ac.y, a.z + w * ac.z};
                    } else {
                        const double va = d3 * d6 - d5 * d4;
                        if (va <= 0.0 && (d4 - d3) >= 0.0 && (d5 - d6) >= 0.0) {
                            const double w = (d4 - d3) / ((d4 - d3) + (d5 - d6));
                            q = {b.x + w * (c.x - b.x), b.y + w * (c.y - b.y), b.z + w * (c.z - b.z)};
                        } else {
                            const double den = 1.0 / (va + vb + vc);
                            const double v = vb * den, w = vc * den;
                            q = {a.x + ab.x * v + ac.x * w, a.y + ab.y * v + ac.y * w, a.z + ab.z * v + ac.z * w};
                        }
                    }
                }
            }
        }
    }
    const D3 d = dsub(p, q);
    return ddot(d, d);
}

__device__ __forceinline__ double box_d2(float4 lo, float4 hi, D3 p)
{
    const double dx = fmax(fmax((double)lo.x - p.x, 0.0), p.x - (double)hi.x);
    const double dy = fmax(fmax((double)lo.y - p.y, 0.0), p.y - (double)hi.y);
    const double dz = fmax(fmax((double)lo.z - p.z, 0.0), p.z - (double)hi.z);
    return dx * dx + dy * dy + dz * dz;
}

// Squared distance from the group's point p to the nearest face of the tree's
// mesh.  The eight lanes test a node's children, the walk enters the nearest one
// and leaves the others that could still hold something closer on the group's
// stack (shared memory; at most seven a level).  All lanes of a warp call this
// together; the result is the same in all lanes of a group.  That rests on the
// lanes' distances being ordered: a face with a NaN or infinite corner gives NaN,
// which would stay in its lane's minimum and part the lanes' walks, so a leaf's
// distance is never more than DBL_MAX (box_d2 gives no NaN: fmax drops it).
constexpr int kHdThreads = 128;
constexpr int kHdStack = 64;

struct HdEntry {
    double d2;
    int lvl, g;
};

__device__ __forceinline__ double nearest_d2(bool has, D3 p, const TreeView &T, const int2 *levels, HdEntry *stack,
                                             const float4 *__restrict__ pts)
{
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, gl = lane & 7, shift = lane & 24;
    double best = DBL_MAX;
    int lvl = T.top, g = 0, topg = 0, sp = 0;
    bool run = has;
    while (__any_sync(kAll, run)) {
        const int node = 8 * g + gl;
        double d = DBL_MAX;
        const int2 level = levels[lvl];
        if (run && node <= level.y) {
            const size_t b = 2 * ((size_t)level.x + node);
            d = box_d2(T.boxes[b], T.boxes[b + 1], p);
            if (lvl == 0) {
                const int4 t = d < best ? T.leaf[node] : make_int4(0, 0, 0, kLeafDead);
                d = t.w != kLeafDead ? point_tri_d2(p, dat(pts[t.x]), dat(pts[t.y]), dat(pts[t.z])) : DBL_MAX;
                d = fmin(d, DBL_MAX);
            }
        }
        double m = d;
        int at = gl;  // the nearest of the eight (the lowest lane of equals)
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const double md = __shfl_xor_sync(kAll, m, o);
            const int ma = __shfl_xor_sync(kAll, at, o);
            if (md < m || (md == m && ma < at)) {
                m = md;
                at = ma;
            }
        }
        const bool inner = run && lvl > 0;
        const unsigned others = (__ballot_sync(kAll, inner && d < best && gl != at) >> shift) & 255u;
        if (inner && d < best && gl != at) stack[sp + __popc(others & ((1u << gl) - 1u))] = HdEntry{d, lvl - 1, node};
        __syncwarp();
        if (run) {
            sp += __popc(others);
            if (inner && m < best) {
                g = 8 * g + at;
                --lvl;
            } else {
                if (lvl == 0 && m < best) best = m;
                bool found = false;
                while (sp > 0 && !found) {
                    const HdEntry e = stack[--sp];
                    found = e.d2 < best;
                    lvl = e.lvl;
                    g = e.g;
                }
                if (!found) {
                    run = ++topg < T.top_groups;
                    lvl = T.top;
                    g = topg;
                }
            }
        }
        __syncwarp();
    }
    return best;
}

// A binary hierarchy as a walk needs it.
struct BvhView {
    const BvhNode *nodes;
    const int *parent, *vals, *scene;
};

// The same by one thread, on a binary hierarchy without a stack: the walk enters the
// nearer child first, and the farther one on the way back if its box is still closer
// than the best face so far (the parent array gives the way up).  The loop counts its
// steps, at most two a node and one up: counted, a warp's lanes meet again at each step;
// in a loop without an end they ran apart (7 of 32 lanes an instruction instead of 16,
// 6.8 ms instead of 3.6 for 1.2M samples against 82k faces).
__device__ double nearest_d2(D3 p, const BvhNode *__restrict__ nodes, const int *__restrict__ parent,
                             const int *__restrict__ vals, int L, const float4 *__restrict__ pts,
                             const int4 *__restrict__ tris)
{
    double best = DBL_MAX;
    auto leaf = [&](int pos) {
        const int g = vals[pos];
        if (g < 0) return;
        const int4 t = tris[g];
        const double d2 = point_tri_d2(p, dat(pts[t.x]), dat(pts[t.y]), dat(pts[t.z]));
        best = fmin(best, d2);
    };
    if (L == 1) {
        leaf(0);
        return best;
    }
    int node = 0, from = 0;  // from: 0 parent, 1 left child, 2 right child
    for (long long budget = 4LL * L + 16; budget > 0; --budget) {
        const BvhNode nd = nodes[node];
        const double dl = box_d2(nd.llo, nd.lhi, p), dr = box_d2(nd.rlo, nd.rhi, p);
        const int near_side = dl <= dr ? 1 : 2;
        const int cl = __float_as_int(nd.llo.w), cr = __float_as_int(nd.rlo.w);
        int next = -1;
        // from the parent: the nearer side, then the farther; back from the
        // nearer side: the farther; back from the farther side: done here
        if (from == 0 || from == near_side) {
            for (int k = from == 0 ? 0 : 1; k < 2 && next < 0; ++k) {
                const int side = k == 0 ? near_side : 3 - near_side;
                if ((side == 1 ? dl : dr) >= best) continue;
                const int c = side == 1 ? cl : cr;
                if (c >= 0) next = c;
                else leaf(~c);
            }
        }
        if (next >= 0) {
            node = next;
            from = 0;
            continue;
        }
        const int code = parent[node];
        if (code < 0) break;
        node = code >> 2;
        from = (code & 1) ? 2 : 1;
    }
    return best;
}

// One group of eight lanes, or one thread, per sample (face f of A, barycentric grid
// point (i/k, j/k)): distance to mesh B; the block's largest squared distance and the
// sum of the squared distances go to this block's partials.
//
// A group's walk is short, but its eight lanes test whole groups of leaves in FP64 for
// the one that is nearest; a thread's walk is a longer chain that wastes nothing.  So
// groups serve few samples, which leave the device idle, and threads many
// (kHdGroupSamples).
template <bool GROUP>
__global__ void __launch_bounds__(kHdThreads) k_hd_samples(const float4 *__restrict__ pa, const int4 *__restrict__ fa,
                                                           int nfa, int k, const __grid_constant__ TreeView T,
                                                           BvhView V, const float4 *__restrict__ pb,
                                                           const int4 *__restrict__ fb, double *part_max,
                                                           double *part_sum, double *part_edge)
{
    __shared__ HdEntry s_stack[GROUP ? kHdThreads / 8 : 1][GROUP ? kHdStack : 1];
    __shared__ int2 s_lvl[kTreeMaxLevels];
    if constexpr (GROUP) T.levels(s_lvl);
    constexpr int kPer = GROUP ? 4 : 32;  // samples a warp
    const int lane = threadIdx.x & 31;
    const int S = (k + 1) * (k + 2) / 2;
    const long long total = (long long)nfa * S;
    double mx = 0.0, sum = 0.0, edge = 0.0;
    const long long warps = (long long)gridDim.x * (kHdThreads / 32);
    for (long long w = ((long long)blockIdx.x * kHdThreads + threadIdx.x) >> 5; w * kPer < total; w += warps) {
        const long long i = w * kPer + (GROUP ? lane >> 3 : lane);
        const int f = i < total ? (int)(i / S) : 0;
        int s = (int)(i % S);
        const int4 t = fa[f];
        const bool has = i < total && !face_dead(t);
        // s -> (u, v) with u + v <= k, rows of u
        int u = 0;
        while (s > k - u) {
            s -= k - u + 1;
            ++u;
        }
        const int v = s;
        D3 a{}, b{}, c{};
        if (has) {
            a = dat(pa[t.x]);
            b = dat(pa[t.y]);
            c = dat(pa[t.z]);
        }
        const double su = (double)u / k, sv = (double)v / k;
        const D3 q = {a.x + su * (b.x - a.x) + sv * (c.x - a.x), a.y + su * (b.y - a.y) + sv * (c.y - a.y),
                      a.z + su * (b.z - a.z) + sv * (c.z - a.z)};
        double d2 = 0.0;
        if constexpr (GROUP) d2 = nearest_d2(has, q, T, s_lvl, s_stack[threadIdx.x >> 3], pb);
        else if (has) d2 = nearest_d2(q, V.nodes, V.parent, V.vals, V.scene[7], pb, fb);
        if (!has || (GROUP && (lane & 7) != 0)) continue;
        mx = fmax(mx, d2);
        sum += d2;
        if (u == 0 && v == 0) {  // the face's longest edge, once per face
            const D3 e0 = dsub(b, a), e1 = dsub(c, b), e2 = dsub(a, c);
            edge = fmax(edge, fmax(ddot(e0, e0), fmax(ddot(e1, e1), ddot(e2, e2))));
        }
    }
    __shared__ double sm[3][kHdThreads];
    sm[0][threadIdx.x] = mx;
    sm[1][threadIdx.x] = sum;
    sm[2][threadIdx.x] = edge;
    __syncthreads();
    for (int o = kHdThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            sm[0][threadIdx.x] = fmax(sm[0][threadIdx.x], sm[0][threadIdx.x + o]);
            sm[1][threadIdx.x] += sm[1][threadIdx.x + o];
            sm[2][threadIdx.x] = fmax(sm[2][threadIdx.x], sm[2][threadIdx.x + o]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part_max[blockIdx.x] = sm[0][0];
        part_sum[blockIdx.x] = sm[1][0];
        part_edge[blockIdx.x] = sm[2][0];
    }
}

constexpr int kHdBlocks = kNumSMs * 8;

// Up to this many samples are walked by groups.  Whole calls, ms by groups / by threads,
// for meshes close to each other (a simplified mesh and its input) against 82k faces:
// 0.33/0.30 at 15k samples, 0.40/0.35 at 31k, 0.52/0.30 at 61k, 1.45/0.60 at 307k,
// 15.3/2.8 at 4.9M; for meshes a tenth of their size apart, where the walks of
// neighbouring samples part: 0.40/0.59, 0.51/0.62, 0.73/0.61, 2.21/1.44, 27.3/11.0.
// Against 320 faces they meet near 50k, against 328k near 20k (close) and 50k (apart).
constexpr long long kHdGroupSamples = 40000;

// One stream-ordered allocation, handed out in pieces: sized by a first pass over
// the same take() calls with no memory behind them.
struct Scratch {
    unsigned char *p = nullptr;
    size_t at = 0;
    cudaStream_t s = nullptr;
    explicit Scratch(cudaStream_t st) : s(st) {}
    ~Scratch()
    {
        if (p) cudaFreeAsync(p, s);
    }
    Scratch(const Scratch &) = delete;
    Scratch &operator=(const Scratch &) = delete;
    bool allocate()  // after the sizing pass
    {
        const size_t bytes = at;
        at = 0;
        return cudaMallocAsync((void **)&p, bytes ? bytes : 1, s) == cudaSuccess;
    }
    template <class T> T *take(size_t n)
    {
        T *q = p ? reinterpret_cast<T *>(p + at) : nullptr;
        at += tree_align(n * sizeof(T));
        return q;
    }
};

}  // namespace
}  // namespace pamo

using namespace pamo;

extern "C" int pamo_check_mesh(const float *d_points, const int *d_tris, int n_pts, int n_tris,
                               unsigned char *d_out_flags, long long *h_out, void *stream)
{
    if (!h_out || n_pts < 0 || n_tris < 0 || (n_tris && (!d_points || !d_tris || n_pts == 0))) return PAMO_ERR_INVALID_ARG;
    for (int i = 0; i < C_COUNT; ++i) h_out[i] = 0;
    if (n_tris == 0) {
        h_out[C_UNREFERENCED] = n_pts;
        return PAMO_OK;
    }
    int dev;
    if (cudaGetDevice(&dev) != cudaSuccess) return PAMO_ERR_NO_DEVICE;
    cudaStream_t s = (cudaStream_t)stream;
    PAMO_CUDA_TRY(retain_pool_memory());
    const size_t n = (size_t)n_pts, m = (size_t)n_tris;
    const long long scan_ints = scan_scratch_ints((long long)n_pts + 1);
    Scratch mem(s);
    float4 *p4;
    int4 *t4;
    unsigned long long *c;
    uint8_t *ok, *fl;
    int *qlist, *n_query, *degv, *first, *cursor, *faces_of, *scan_tmp;
    unsigned char *tree_mem;
    for (int pass = 0; pass < 2; ++pass) {
        p4 = mem.take<float4>(n);
        t4 = mem.take<int4>(m);
        c = mem.take<unsigned long long>(C_COUNT + 1);
        ok = mem.take<uint8_t>(m);
        fl = d_out_flags ? d_out_flags : mem.take<uint8_t>(m);
        qlist = mem.take<int>(m);
        degv = mem.take<int>(n + 1);
        first = mem.take<int>(n + 1);
        cursor = mem.take<int>(n);
        faces_of = mem.take<int>(3 * m);
        scan_tmp = mem.take<int>((size_t)scan_ints);
        tree_mem = mem.take<unsigned char>(PackedTree::bytes(n_tris));
        if (pass == 0 && !mem.allocate()) return PAMO_ERR_OOM;
    }
    n_query = reinterpret_cast<int *>(c + C_COUNT);
    PAMO_CUDA_TRY(cudaMemsetAsync(c, 0, (C_COUNT + 1) * 8, s));
    launch(k_ck_convert, grid_for(n_pts > n_tris ? n_pts : n_tris), kThreads, 0, s, d_points, n_pts, d_tris, n_tris, p4,
           t4);
    launch(k_ck_validate, grid_for(n_tris), kThreads, 0, s, (const int4 *)t4, n_tris, n_pts, c);
    unsigned long long h[C_COUNT];
    PAMO_CUDA_TRY(cudaMemcpyAsync(h, c, C_COUNT * 8, cudaMemcpyDeviceToHost, s));
    PAMO_CUDA_TRY(cudaStreamSynchronize(s));
    if (h[C_BAD_INDEX]) return PAMO_ERR_INVALID_ARG;
    launch(k_ck_degenerate, grid_for(n_tris), kThreads, 0, s, (const float4 *)p4, (const int4 *)t4, n_tris, ok, c);
    // self-intersections (the refit clears the flags)
    PackedTree tree;  // its arrays lie in this call's scratch: nothing to release
    PAMO_CUDA_TRY(tree.place(tree_mem, n_tris, s));
    PAMO_CUDA_TRY(tree_build(tree, p4, t4, n_tris, s));
    PAMO_CUDA_TRY(tree_refit(tree, p4, t4, ok, qlist, n_query, fl, n_tris, s));
    launch(k_ck_pairs, grid_for(8LL * n_tris, kPairThreads), kPairThreads, 0, s, tree.view(), (const int *)qlist,
           (const int *)n_query, (const float4 *)p4, fl, c);
    launch(k_ck_flagged, grid_for(n_tris), kThreads, 0, s, (const uint8_t *)fl, n_tris, c);
    // manifold checks over the vertex -> face lists
    PAMO_CUDA_TRY(cudaMemsetAsync(degv, 0, (n + 1) * 4, s));
    PAMO_CUDA_TRY(cudaMemsetAsync(cursor, 0, n * 4, s));
    launch(k_ck_count, grid_for(n_tris), kThreads, 0, s, (const int4 *)t4, n_tris, degv);
    PAMO_CUDA_TRY(scan_scratch_init(scan_tmp, scan_ints, s));
    PAMO_CUDA_TRY(exclusive_scan(degv, first, (long long)n_pts + 1, nullptr, scan_tmp, nullptr, s));
    launch(k_ck_fill, grid_for(n_tris), kThreads, 0, s, (const int4 *)t4, n_tris, (const int *)first, cursor, faces_of);
    launch(k_ck_edges, grid_for(3LL * n_tris), kThreads, 0, s, (const int4 *)t4, n_tris, (const int *)first,
           (const int *)faces_of, c);
    launch(k_ck_fans, grid_for(n_pts), kThreads, 0, s, (const int4 *)t4, n_pts, (const int *)first,
           (const int *)faces_of, c);
    PAMO_CUDA_TRY(cudaGetLastError());
    PAMO_CUDA_TRY(cudaMemcpyAsync(h, c, C_COUNT * 8, cudaMemcpyDeviceToHost, s));
    PAMO_CUDA_TRY(cudaStreamSynchronize(s));
    for (int i = 0; i < C_COUNT; ++i) h_out[i] = (long long)h[i];
    return PAMO_OK;
}

extern "C" int pamo_mesh_distance(const float *d_pa, const int *d_fa, int na, int nfa, const float *d_pb,
                                  const int *d_fb, int nb, int nfb, int subdiv, double *h_out4, void *stream)
{
    if (!h_out4 || na < 0 || nfa < 0 || nb < 0 || nfb < 0 || subdiv < 1 || subdiv > 1024) return PAMO_ERR_INVALID_ARG;
    if ((nfa && (!d_pa || !d_fa || na == 0)) || (nfb && (!d_pb || !d_fb || nb == 0))) return PAMO_ERR_INVALID_ARG;
    for (int i = 0; i < 4; ++i) h_out4[i] = 0.0;
    if (nfa == 0) return PAMO_OK;
    if (nfb == 0) return PAMO_ERR_INVALID_ARG;  // no surface to measure against
    int dev;
    if (cudaGetDevice(&dev) != cudaSuccess) return PAMO_ERR_NO_DEVICE;
    cudaStream_t s = (cudaStream_t)stream;
    PAMO_CUDA_TRY(retain_pool_memory());
    Scratch mem(s);
    float4 *pa4, *pb4;
    int4 *fa4, *fb4;
    double *pm;
    unsigned long long *bad;
    unsigned char *tree_mem;
    const long long total = (long long)nfa * ((subdiv + 1) * (subdiv + 2) / 2);
    const bool groups = total <= kHdGroupSamples;
    for (int pass = 0; pass < 2; ++pass) {
        pa4 = mem.take<float4>((size_t)na);
        fa4 = mem.take<int4>((size_t)nfa);
        pb4 = mem.take<float4>((size_t)nb);
        fb4 = mem.take<int4>((size_t)nfb);
        pm = mem.take<double>(3 * kHdBlocks);
        bad = mem.take<unsigned long long>(2 * C_COUNT);
        tree_mem = mem.take<unsigned char>(groups ? PackedTree::bytes(nfb) : Lbvh::bytes(nfb));
        if (pass == 0 && !mem.allocate()) return PAMO_ERR_OOM;
    }
    double *ps = pm + kHdBlocks, *pe = ps + kHdBlocks;
    launch(k_ck_convert, grid_for(na > nfa ? na : nfa), kThreads, 0, s, d_pa, na, d_fa, nfa, pa4, fa4);
    launch(k_ck_convert, grid_for(nb > nfb ? nb : nfb), kThreads, 0, s, d_pb, nb, d_fb, nfb, pb4, fb4);
    PAMO_CUDA_TRY(cudaMemsetAsync(bad, 0, 2 * C_COUNT * 8, s));
    launch(k_ck_validate, grid_for(nfa), kThreads, 0, s, (const int4 *)fa4, nfa, na, bad);
    launch(k_ck_validate, grid_for(nfb), kThreads, 0, s, (const int4 *)fb4, nfb, nb, bad + C_COUNT);
    unsigned long long hb[2 * C_COUNT];
    PAMO_CUDA_TRY(cudaMemcpyAsync(hb, bad, sizeof(hb), cudaMemcpyDeviceToHost, s));
    PAMO_CUDA_TRY(cudaStreamSynchronize(s));
    if (hb[C_BAD_INDEX] || hb[C_DEAD] == (unsigned long long)nfa) return PAMO_ERR_INVALID_ARG;
    if (hb[C_COUNT + C_BAD_INDEX] || hb[C_COUNT + C_DEAD] == (unsigned long long)nfb) return PAMO_ERR_INVALID_ARG;
    const long long live_a = (long long)nfa - (long long)hb[C_DEAD];  // dead faces of A add no samples
    PackedTree tree;  // the arrays of both lie in this call's scratch: nothing to release
    Lbvh bvh;
    if (groups) {
        PAMO_CUDA_TRY(tree.place(tree_mem, nfb, s));
        PAMO_CUDA_TRY(tree_build(tree, pb4, fb4, nfb, s));
        PAMO_CUDA_TRY(tree_refit(tree, pb4, fb4, nullptr, nullptr, nullptr, nullptr, nfb, s));
        launch(k_hd_samples<true>, kHdBlocks, kHdThreads, 0, s, (const float4 *)pa4, (const int4 *)fa4, nfa, subdiv,
               tree.view(), BvhView{}, (const float4 *)pb4, (const int4 *)fb4, pm, ps, pe);
    } else {
        PAMO_CUDA_TRY(bvh.place(tree_mem, nfb, s));
        PAMO_CUDA_TRY(lbvh_build(bvh, pb4, fb4, nfb, s));
        PAMO_CUDA_TRY(lbvh_refit(bvh, pb4, fb4, nfb, s));
        launch(k_hd_samples<false>, kHdBlocks, kHdThreads, 0, s, (const float4 *)pa4, (const int4 *)fa4, nfa, subdiv,
               TreeView{}, BvhView{bvh.nodes, bvh.parent, bvh.vals, bvh.scene}, (const float4 *)pb4,
               (const int4 *)fb4, pm, ps, pe);
    }
    PAMO_CUDA_TRY(cudaGetLastError());
    std::vector<double> h(3 * kHdBlocks);
    PAMO_CUDA_TRY(cudaMemcpyAsync(h.data(), pm, 3 * kHdBlocks * 8, cudaMemcpyDeviceToHost, s));
    PAMO_CUDA_TRY(cudaStreamSynchronize(s));
    double mx = 0.0, sum = 0.0, edge = 0.0;
    for (int i = 0; i < kHdBlocks; ++i) {  // fixed order: the result does not depend on scheduling
        mx = fmax(mx, h[i]);
        sum += h[kHdBlocks + i];
        edge = fmax(edge, h[2 * kHdBlocks + i]);
    }
    const double samples = (double)live_a * ((subdiv + 1) * (subdiv + 2) / 2);
    h_out4[0] = sqrt(mx);
    // every point of a face lies within (longest edge / k) / sqrt(3) of a sample
    // (a sub-triangle's circumradius, or half its longest edge when obtuse), and
    // the distance to B is 1-Lipschitz
    h_out4[1] = sqrt(mx) + sqrt(edge) / subdiv / sqrt(3.0);
    h_out4[2] = sum / samples;
    h_out4[3] = samples;
    return PAMO_OK;
}
