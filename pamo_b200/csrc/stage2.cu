// Stage-2 collapse round on the device (sm_100a).
//
// One round follows the reference's CUSimp_Free::forward
// (simp_cuda/src/cusimp_free.cu:891-1048) decision for decision, with a B200
// layout and fewer passes:
//   face pass A   plane of every face (fp32, reference order), vertex degrees,
//                 per-face descending-edge counts                 [:276-289,306-317,337-348]
//   2 scans       vertex->face CSR offsets, edge offsets
//   face pass B   CSR fill + edge emission                          [:291-304,319-335]
//   vertex pass   canonical (ascending face) order of each CSR segment, then the
//                 quadric sum in that order                          [:350-366]
//   edge pass     cost (link condition, edge lengths, flip and skinny terms,
//                 quadric at the midpoint, u32 quantisation) fused with the
//                 64-bit key min over each endpoint                  [:382-610]
//   edge pass     independent-set test + collapse + skinny rollback  [:639-774]
//   scan/scatter  collapsed list in edge order
//   face pass     degenerate faces removed                           [:218-232]
//   edge pass     coincident-endpoint collapses                      [:234-274]
//   packed tree   build over the round's faces, refit, query of the faces touched
//                 by collapses, pair tests                           [bvh/self_intersect.cuh]
//   undo passes   candidates, restore, re-check (<= 5)               [:776-878,1015-1040]
//   scan          pts_map = exclusive scan of occupancy              [:1042-1045]
// The key independent set uses a per-vertex minimum: an edge wins iff its key is
// the minimum over every face touching either endpoint (the reference's per-face
// minimum), which equals: key == vmin[u] == vmin[v] and no vertex of those faces
// has a smaller vmin.
#include <cstdio>
#include <cstring>

#include "scan.cuh"
#include "exact.cuh"
#include "stage2.cuh"
#include "tritri.cuh"

namespace pamo {

#define S2_TRY_EARLY(expr)                                \
    do {                                                  \
        cudaError_t _e = (expr);                          \
        if (_e != cudaSuccess) return map_cuda_error(_e); \
    } while (0)

namespace {

constexpr float kCostRange = 10.0f;
constexpr double kRebuildFraction = 0.6;

__device__ __forceinline__ uint32_t quantise_cost(float c)
{
    // the reference converts with a saturating float->u32 conversion
    return (uint32_t)(tclamp(c, 0.0f, kCostRange) / kCostRange * 4294967296.0f);
}

// The round's working copies and everything that starts it at zero.
__global__ void k_round_init(const float4 *__restrict__ opts, const int4 *__restrict__ otris, float4 *pts,
                             int4 *tris, int *occ, int *deg, int *cursor, unsigned long long *vmin, int *first_edge,
                             uint8_t *active, RoundCounters *cnt, int n, int m)
{
    chain_wait();
    constexpr int kCounters = (int)(sizeof(RoundCounters) / sizeof(int));
    const long long N = n + 1 > kCounters ? n + 1 : kCounters;
    PAMO_GRID_STRIDE(i, N > m + 1 ? N : m + 1)
    {
        if (i < n) {
            pts[i] = opts[i];
            occ[i] = 1;
            deg[i] = 0;
            cursor[i] = 0;
            vmin[i] = ~0ull;
        } else if (i == n) {
            occ[n] = 0;
            deg[n] = 0;
        }
        if (i < m) {
            tris[i] = otris[i];
            active[i] = 0;
        } else if (i == m) {
            first_edge[m] = 0;
        }
        if (i < kCounters) reinterpret_cast<int *>(cnt)[i] = 0;
    }
}

__global__ void k_face_a(const float4 *__restrict__ pts, const int4 *__restrict__ tris, int m, int *deg,
                         int *ecount, float4 *plane, float4 *elen)
{
    chain_wait();
    PAMO_GRID_STRIDE(f, m)
    {
        int4 t = tris[f];
        if (face_dead(t)) {
            ecount[f] = 0;
            continue;
        }
        atomicAdd(&deg[t.x], 1);
        atomicAdd(&deg[t.y], 1);
        atomicAdd(&deg[t.z], 1);
        ecount[f] = (t.x > t.y) + (t.y > t.z) + (t.z > t.x);
        V3 v0 = v3(pts[t.x]), v1 = v3(pts[t.y]), v2 = v3(pts[t.z]);
        V3 nrm = vcross(vsub(v1, v0), vsub(v2, v0));
        nrm = vdivs(nrm, vnorm(nrm));
        float d = -vdot(nrm, v0);
        plane[f] = make_float4(nrm.x, nrm.y, nrm.z, d);
        // the three edge lengths in cyclic order, as the cost kernel sums them
        // (cusimp_free.cu:448-485): |P[i]-P[j]|, |P[j]-P[k]|, |P[k]-P[i]|
        elen[f] = make_float4(vnorm(vsub(v0, v1)), vnorm(vsub(v1, v2)), vnorm(vsub(v2, v0)), 0.f);
    }
}

__global__ void k_face_b(const int4 *__restrict__ tris, int m, const int *__restrict__ first_near, int *cursor,
                         int *near_tris, const int *__restrict__ first_edge, int2 *edges)
{
    chain_wait();
    PAMO_GRID_STRIDE(f, m)
    {
        int4 t = tris[f];
        if (face_dead(t)) continue;
        near_tris[first_near[t.x] + atomicAdd(&cursor[t.x], 1)] = (int)f;
        near_tris[first_near[t.y] + atomicAdd(&cursor[t.y], 1)] = (int)f;
        near_tris[first_near[t.z] + atomicAdd(&cursor[t.z], 1)] = (int)f;
        int e = first_edge[f];
        if (t.x > t.y) edges[e++] = make_int2(t.y, t.x);
        if (t.y > t.z) edges[e++] = make_int2(t.z, t.y);
        if (t.z > t.x) edges[e++] = make_int2(t.x, t.z);
    }
}

__device__ __forceinline__ int next_after(int4 t, int v);

// Canonical (ascending) segment order of each vertex's faces, the vertex after it
// in each face, then the quadric sum p p^T in that order.  A group of eight lanes
// per vertex: the faces go to shared memory, each lane finds the rank of its own
// by counting, leaves its plane at that rank, and sums one or two of the ten
// entries over the planes in order.  One thread per vertex sorted its segment by
// insertion in global memory and then followed the faces one by one, which made
// the round's setup 32 / 59 / 94 us on meshes of 5k / 200k / 2M faces (mean over
// the rounds); it was 27 / 52 / 92 us so, and is 21 / 48 / 91 with chained launches.
constexpr int kRing = 32;  // longer segments are sorted and summed by one lane

__global__ void __launch_bounds__(kThreads) k_vertex_quadric(const int *__restrict__ first_near, int *near_tris,
                                                             const float4 *__restrict__ plane,
                                                             const int4 *__restrict__ tris, float *quad, int *nxt,
                                                             int n)
{
    chain_wait();
    __shared__ int s_face[kThreads / 8][kRing];
    __shared__ float4 s_plane[kThreads / 8][kRing];
    const int lane = threadIdx.x & 31, gl = lane & 7;
    int *face = s_face[threadIdx.x >> 3];
    float4 *pl = s_plane[threadIdx.x >> 3];
    // entry gl (and 8 + gl) of the quadric: the product of these two plane components
    const int c0 = gl < 4 ? 0 : gl < 7 ? 1 : 2, c1 = gl < 4 ? gl : gl < 7 ? gl - 3 : 2;
    const int e0 = gl == 0 ? 2 : 3;
    const long long warps = (long long)gridDim.x * (kThreads / 32);
    for (long long w = ((long long)blockIdx.x * kThreads + threadIdx.x) >> 5; w * 4 < n; w += warps) {
        const long long v = w * 4 + (lane >> 3);
        const int a = v < n ? first_near[v] : 0, d = v < n ? first_near[v + 1] - a : 0;
        const bool in_ring = d <= kRing;
        float q = 0.f, q2 = 0.f;
        if (in_ring)
            for (int i = gl; i < d; i += 8) face[i] = near_tris[a + i];
        __syncwarp();
        if (in_ring) {
            for (int i = gl; i < d; i += 8) {
                const int f = face[i];
                int rank = 0;
                for (int j = 0; j < d; ++j) rank += face[j] < f || (face[j] == f && j < i);
                near_tris[a + rank] = f;
                nxt[a + rank] = next_after(tris[f], (int)v);  // vertex after v in face f (i->j->k->i)
                pl[rank] = plane[f];
            }
        } else if (gl == 0) {
            for (int i = a + 1; i < a + d; ++i) {
                int x = near_tris[i], j = i - 1;
                while (j >= a && near_tris[j] > x) {
                    near_tris[j + 1] = near_tris[j];
                    --j;
                }
                near_tris[j + 1] = x;
            }
            for (int s = a; s < a + d; ++s) nxt[s] = next_after(tris[near_tris[s]], (int)v);
        }
        __syncwarp();
        for (int j = 0; j < d; ++j) {
            const float4 x = in_ring ? pl[j] : plane[near_tris[a + j]];
            const float p[4] = {x.x, x.y, x.z, x.w};
            const float x0 = c0 == 0 ? p[0] : c0 == 1 ? p[1] : p[2];
            const float x1 = c1 == 0 ? p[0] : c1 == 1 ? p[1] : c1 == 2 ? p[2] : p[3];
            q += x0 * x1;
            q2 += (e0 == 2 ? p[2] : p[3]) * p[3];
        }
        if (v < n) {
            quad[12 * v + gl] = q;
            if (gl < 4) quad[12 * v + 8 + gl] = gl < 2 ? q2 : 0.f;
        }
        __syncwarp();
    }
}

// Quality mode: each vertex's quadric in FP64, the planes recomputed from the
// positions in FP64 (unit normal n, d = -n . a), summed over the vertex's faces
// in its (sorted) list order, so the result is deterministic.
__global__ void k_vertex_quadric64(const int *__restrict__ first_near, const int *__restrict__ near_tris,
                                   const float4 *__restrict__ pts, const int4 *__restrict__ tris, double *q64, int n)
{
    chain_wait();
    PAMO_GRID_STRIDE(v, n)
    {
        double q[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
        for (int s = first_near[v]; s < first_near[v + 1]; ++s) {
            const int4 t = tris[near_tris[s]];
            const float4 fa = pts[t.x], fb = pts[t.y], fc = pts[t.z];
            const double ax = fa.x, ay = fa.y, az = fa.z;
            const double ux = fb.x - ax, uy = fb.y - ay, uz = fb.z - az;
            const double wx = fc.x - ax, wy = fc.y - ay, wz = fc.z - az;
            double nx = uy * wz - uz * wy, ny = uz * wx - ux * wz, nz = ux * wy - uy * wx;
            const double len = sqrt(nx * nx + ny * ny + nz * nz);
            if (!(len > 0.0)) continue;  // a degenerate face has no plane
            nx /= len;
            ny /= len;
            nz /= len;
            const double d = -(nx * ax + ny * ay + nz * az);
            q[0] += nx * nx; q[1] += nx * ny; q[2] += nx * nz; q[3] += nx * d;
            q[4] += ny * ny; q[5] += ny * nz; q[6] += ny * d;
            q[7] += nz * nz; q[8] += nz * d; q[9] += d * d;
        }
        for (int k = 0; k < 10; ++k) q64[10 * (size_t)v + k] = q[k];
    }
}

// Quality mode: the point minimising v^T (Qu + Qv) v, from the 3 x 3 system
// A x = -b of the summed quadric (Cramer's rule in FP64).  The midpoint is kept
// when the system is close to singular (|det| below 1e-12 of the product of
// A's row norms) or the minimiser lies more than the edge's length from the
// midpoint (a nearly flat, ill-conditioned quadric).
__device__ V3 qem_position(const double *qu, const double *qv, V3 p0, V3 p1)
{
    double q[10];
    for (int k = 0; k < 10; ++k) q[k] = qu[k] + qv[k];
    const double a00 = q[0], a01 = q[1], a02 = q[2], a11 = q[4], a12 = q[5], a22 = q[7];
    const double b0 = -q[3], b1 = -q[6], b2 = -q[8];
    const double c00 = a11 * a22 - a12 * a12, c01 = a02 * a12 - a01 * a22, c02 = a01 * a12 - a02 * a11;
    const double det = a00 * c00 + a01 * c01 + a02 * c02;
    const double r0 = sqrt(a00 * a00 + a01 * a01 + a02 * a02), r1 = sqrt(a01 * a01 + a11 * a11 + a12 * a12);
    const double r2 = sqrt(a02 * a02 + a12 * a12 + a22 * a22);
    const V3 mid = vmid(p0, p1);
    if (!(fabs(det) > 1e-12 * r0 * r1 * r2)) return mid;
    const double c11 = a00 * a22 - a02 * a02, c12 = a01 * a02 - a00 * a12, c22 = a00 * a11 - a01 * a01;
    const double x = (c00 * b0 + c01 * b1 + c02 * b2) / det;
    const double y = (c01 * b0 + c11 * b1 + c12 * b2) / det;
    const double z = (c02 * b0 + c12 * b1 + c22 * b2) / det;
    const double ex = (double)p1.x - p0.x, ey = (double)p1.y - p0.y, ez = (double)p1.z - p0.z;
    const double dx = x - mid.x, dy = y - mid.y, dz = z - mid.z;
    if (!(dx * dx + dy * dy + dz * dz <= ex * ex + ey * ey + ez * ez)) return mid;
    return {(float)x, (float)y, (float)z};
}

__device__ __forceinline__ int next_after(int4 t, int v)
{
    if (t.x == v) return t.y;
    if (t.y == v) return t.z;
    if (t.z == v) return t.x;
    return -2;
}

__device__ __forceinline__ float skinny_term(V3 n0, V3 n1, V3 n2)
{
    // edge_length / triangle_area (cusimp_free.cu:368-380) and the penalty with
    // the reference's precedence: only the first square divides (:533,573)
    float l01 = vnorm(vsub(n0, n1));
    float l12 = vnorm(vsub(n1, n2));
    float l20 = vnorm(vsub(n2, n0));
    float s = (l01 + l12 + l20) / 2.0f;
    float area = sqrtf(s * (s - l01) * (s - l12) * (s - l20));
    // pow(float, 2) in the reference resolves to std::pow's promoting overload:
    // the squares and the sum after the fp32 numerator are doubles, rounded once
    const float c4s3 = 4.0f * sqrtf(3.0f);
    float num = c4s3 * area;
    // Shortcut: every term is non-negative, so the same sum in fp32 (five
    // roundings, relative error < 4e-7 while l01^2 is a normal float; an fp32
    // overflow to +inf only happens when the double sum is far above 1) bounds
    // the double sum from below within 4e-7.  At or above 1 + 2^-18 the double
    // sum is above 1, its float rounding is >= 1, and the clamped penalty is
    // exactly 0 -- the value the double path returns.  Well-shaped triangles
    // (sum near 3) take this path; NaN and near-1 sums fall through.
    const float q01 = l01 * l01;
    if (q01 >= 1.17549435e-38f) {
        float ef = num / q01 + l12 * l12 + l20 * l20 + 0.0000001f;
        if (ef >= 1.0f + 0x1p-18f) return 0.0f;
    }
    // Second shortcut: CUDA's double pow(x, 2.0) is within one double ulp of the
    // exact square x*x for every float x (an exhaustive check over all finite
    // floats on a B200; it differs for ~6% of them).  The same sum with exact
    // squares therefore lies within 8 ulp of the one with pow (each term is
    // non-negative); when a 16-ulp neighbourhood of it rounds to one float, that
    // float is the reference's.  Otherwise (NaN, inf, or a sum next to a float
    // rounding boundary) the pow form is evaluated as the reference writes it.
    const double sq = (double)num / ((double)l01 * (double)l01) + (double)l12 * (double)l12 +
                      (double)l20 * (double)l20 + (double)0.0000001f;
    const double margin = sq * 0x1p-48;
    const float fq = (float)sq;
    if (fq == (float)(sq - margin) && fq == (float)(sq + margin)) return 1.0f - tclamp(fq, 0.0f, 1.0f);
    double e = (double)num / pow((double)l01, 2.0) + pow((double)l12, 2.0) + pow((double)l20, 2.0) +
               (double)0.0000001f;
    return 1.0f - tclamp((float)e, 0.0f, 1.0f);
}

// Whether the moved face's unit normal c / |c| points against `on`, i.e. the
// reference's dot(on, c / |c|) < 0 with c normalised by three divisions.
// Shortcut: with |c|^2 in the normal range and |on . c| well above the
// rounding error of either dot product (1e-5 of sum |on_i c_i|, against a few
// 2^-24 for both forms), the two dot products have the same, non-zero sign, and
// dot(on, c) / |c| stays far from underflow (dc^2 > 1e-30 |c|^2).  Otherwise
// the reference's expression is evaluated.
__device__ __forceinline__ bool normal_flips(V3 on, V3 c)
{
    const float s2 = c.x * c.x + c.y * c.y + c.z * c.z;
    const float dc = vdot(on, c);
    const float mag = fabsf(on.x * c.x) + fabsf(on.y * c.y) + fabsf(on.z * c.z);
    if (s2 > 1e-30f && s2 < 1e30f && fabsf(dc) > 1e-5f * mag && dc * dc > 1e-30f * s2) return dc < 0.f;
    const V3 nn = vdivs(c, vnorm(c));
    return vdot(on, nn) < 0;
}

struct CostArgs {
    const int2 *edges;
    const int *n_edges;
    const float4 *pts;
    const int4 *tris;
    const int *first_near;
    const int *near_tris;
    const int *nxt;
    const float4 *plane;
    const float4 *elen;
    const float4 *quad;
    const uint8_t *invalid;
    uint32_t *edge_cost;
    unsigned long long *vmin;
    float tres, edge_s;
    int is_stuck;
    // batch mode (null otherwise): per-mesh parameters and stale state
    const SlotInfo *slots;
    const SlotCounters *scnt;
    const int *vslot;
    // quality mode (null otherwise): FP64 quadrics in, collapse positions out
    const double *quad64;
    float4 *epos;
};

// What both forms of the edge cost make of the sums over an edge's one-rings.
// The length term: the mean of the nedge edges there, whose lengths add up to sum, and
// the edge's own.
__device__ __forceinline__ float edge_length_term(float sum, int nedge, V3 v0, V3 v1, float tres, float edge_s)
{
    const float mean = sum / (float)nedge / edge_s * tres;
    return mean + vnorm(vsub(v0, v1)) / edge_s * tres;
}

// The cost: the quadric's error at mid, the length term and the ntri skinny terms,
// which add up to Qa.
template <bool QUALITY>
__device__ __forceinline__ uint32_t edge_cost_sum(const CostArgs &A, int u, int v, V3 mid, float elen, float Qa,
                                                  int ntri, float tres, float edge_s)
{
    Qa = 5.0f * Qa;
    if constexpr (QUALITY) {  // the quadric error in FP64 at the chosen position
        const double *qu = A.quad64 + 10 * (size_t)u, *qv = A.quad64 + 10 * (size_t)v;
        double q[10];
        for (int k = 0; k < 10; ++k) q[k] = qu[k] + qv[k];
        const double x = mid.x, y = mid.y, z = mid.z;
        const double qe = x * (q[0] * x + q[1] * y + q[2] * z + q[3]) + y * (q[1] * x + q[4] * y + q[5] * z + q[6]) +
                          z * (q[2] * x + q[5] * y + q[7] * z + q[8]) + (q[3] * x + q[6] * y + q[8] * z + q[9]);
        const float cost = (float)(qe / ((double)edge_s * (double)edge_s));
        return quantise_cost(cost + elen + Qa / (float)ntri * tres);
    }
    float4 a0 = A.quad[3 * u], a1 = A.quad[3 * u + 1], a2 = A.quad[3 * u + 2];
    float4 b0 = A.quad[3 * v], b1 = A.quad[3 * v + 1], b2 = A.quad[3 * v + 2];
    float m00 = a0.x + b0.x, m01 = a0.y + b0.y, m02 = a0.z + b0.z, m03 = a0.w + b0.w;
    float m11 = a1.x + b1.x, m12 = a1.y + b1.y, m13 = a1.z + b1.z, m22 = a1.w + b1.w;
    float m23 = a2.x + b2.x, m33 = a2.y + b2.y;
    float x = mid.x, y = mid.y, z = mid.z, w = 1.0f;
    float r0 = m00 * x + m01 * y + m02 * z + m03 * w;
    float r1 = m01 * x + m11 * y + m12 * z + m13 * w;
    float r2 = m02 * x + m12 * y + m22 * z + m23 * w;
    float r3 = m03 * x + m13 * y + m23 * z + m33 * w;
    float qe = r0 * x + r1 * y + r2 * z + r3 * w;
    float cost = qe / (edge_s * edge_s);
    return quantise_cost(cost + elen + Qa / (float)ntri * tres);
}

// Returns true when the reference writes a new cost for the edge.  QUALITY:
// quality mode (FP64 quadric terms and the chosen collapse position in epos);
// compiled separately so the reference's path carries none of it.
template <bool QUALITY>
__device__ bool edge_cost_value(const CostArgs &A, int u, int v, bool inv_u, bool inv_v, float tres, float edge_s,
                                int is_stuck, uint32_t &out, int e = -1)
{
    if constexpr (QUALITY) {  // an edge whose cost is not rewritten collapses to its midpoint
        const V3 m0 = vmid(v3(A.pts[u]), v3(A.pts[v]));
        A.epos[e] = make_float4(m0.x, m0.y, m0.z, 0.f);
    }
    if (inv_u && inv_v) {
        out = 0xFFFFFFFFu;
        return true;
    }
    if (is_stuck) return false;
    const int ua = A.first_near[u], ub = A.first_near[u + 1];
    const int va = A.first_near[v], vb = A.first_near[v + 1];
    int dup = 0;
    for (int a = ua; a < ub; ++a) {
        int iu = A.nxt[a];
        for (int b = va; b < vb; ++b) {
            int iv = A.nxt[b];
            if (iu == iv) dup++;
            if (dup > 2) {
                out = 0xFFFFFFFFu;
                return true;
            }
        }
    }
    if (dup != 2) return false;

    float elen = 0.0f;
    int nedge = 0;
    for (int pass = 0; pass < 2; ++pass) {
        int lo = pass ? va : ua, hi = pass ? vb : ub;
        for (int a = lo; a < hi; ++a) {
            const int f = A.near_tris[a];
            int4 t = A.tris[f];
            float4 l = A.elen[f];
            if (t.x > t.y) { elen += l.x; nedge++; }
            if (t.y > t.z) { elen += l.y; nedge++; }
            if (t.z > t.x) { elen += l.z; nedge++; }
        }
    }
    V3 v0 = v3(A.pts[u]), v1 = v3(A.pts[v]);
    elen = edge_length_term(elen, nedge, v0, v1, tres, edge_s);
    // the collapse position: the midpoint (the reference), or in quality mode
    // the FP64 quadric's minimiser
    V3 mid;
    if constexpr (QUALITY) {
        mid = qem_position(A.quad64 + 10 * (size_t)u, A.quad64 + 10 * (size_t)v, v0, v1);
        A.epos[e] = make_float4(mid.x, mid.y, mid.z, 0.f);
    } else {
        mid = vmid(v0, v1);
    }

    float Qa = 0.0f;
    int ntri = 0;
    for (int pass = 0; pass < 2; ++pass) {
        int w = pass ? v : u, other = pass ? u : v;
        int lo = pass ? va : ua, hi = pass ? vb : ub;
        for (int a = lo; a < hi; ++a) {
            const int f = A.near_tris[a];
            int4 t = A.tris[f];
            if (face_has(t, other)) continue;
            V3 o0 = v3(A.pts[t.x]), o1 = v3(A.pts[t.y]), o2 = v3(A.pts[t.z]);
            V3 n0 = t.x == w ? mid : o0;
            V3 n1 = t.y == w ? mid : o1;
            V3 n2 = t.z == w ? mid : o2;
            // the unchanged face's unit normal is the face plane's (same expression)
            V3 on = v3(A.plane[f]);
            const V3 c = vcross(vsub(n1, n0), vsub(n2, n0));
            if (normal_flips(on, c)) {
                out = 0xFFFFFFFFu;
                return true;
            }
            Qa += skinny_term(n0, n1, n2);
            ntri++;
        }
    }
    out = edge_cost_sum<QUALITY>(A, u, v, mid, elen, Qa, ntri, tres, edge_s);
    return true;
}

// The edge-cost pass runs in the hierarchy's leaf (Morton) order: a block takes
// kChunkFaces consecutive leaves, lists their faces' edges in shared memory
// (each face owns its 0-2 descending edges) and its threads take the list in
// turn, so neighbouring lanes gather neighbouring vertices and every lane has an
// edge.  Costs are indexed by edge, so the order of work does not change them.
constexpr int kChunkFaces = kThreads;
constexpr int kChunkEdges = 3 * kChunkFaces;

__device__ __forceinline__ int chunk_edges(const int *order, const int *first_edge, int L, long long base,
                                           int *s_list)
{
    long long p = base + threadIdx.x;
    int f = p < L ? order[p] : -1;  // -1: past the end, or a face removed since the build
    int fe = f >= 0 ? first_edge[f] : 0;
    int c = f >= 0 ? first_edge[f + 1] - fe : 0;
    int total;
    int off = block_excl_scan<kThreads>(c, total);
    for (int j = 0; j < c; ++j) s_list[off + j] = fe + j;
    __syncthreads();
    return total;
}

template <bool QUALITY>
__global__ void __launch_bounds__(kThreads) k_edge_cost(CostArgs A, const int *order, int L,
                                                        const int *first_edge)
{
    chain_wait();
    __shared__ int s_list[kChunkEdges];
    for (long long base = (long long)blockIdx.x * kChunkFaces; base < L; base += (long long)gridDim.x * kChunkFaces) {
        const int total = chunk_edges(order, first_edge, L, base, s_list);
        for (int q = threadIdx.x; q < total; q += kThreads) {
            const int e = s_list[q];
            int2 ed = A.edges[e];
            uint32_t c;
            if (!A.slots) {
                if (edge_cost_value<QUALITY>(A, ed.x, ed.y, A.invalid[ed.x], A.invalid[ed.y], A.tres, A.edge_s,
                                             A.is_stuck, c, e))
                    A.edge_cost[e] = c;
                else
                    c = A.edge_cost[e];  // the reference keeps the previous round's value
            } else {  // the mesh's own parameters, invalid table and stale costs (mesh-local numbers)
                const int r = A.vslot[ed.x];
                const SlotInfo &S = A.slots[r];
                const int el = e - A.scnt[r].edge_off;
                if (edge_cost_value<QUALITY>(A, ed.x, ed.y, S.invalid[ed.x - S.vert_off], S.invalid[ed.y - S.vert_off],
                                             S.tres, *S.scale, S.is_stuck, c))
                    S.edge_cost[el] = c;
                else
                    c = S.edge_cost[el];
            }
            unsigned long long key = ((unsigned long long)c << 32) | (unsigned)e;
            atomicMin(&A.vmin[ed.x], key);
            atomicMin(&A.vmin[ed.y], key);
        }
        __syncthreads();
    }
}

// The cost of an edge, by a group of eight lanes: lane gl takes every eighth face
// of u's one-ring, then of v's, so an edge's dozen faces are two steps instead of
// a chain of twelve.  What the reference adds up face by face is added in that
// order: each lane leaves its face's terms in `terms` (the group's eight entries
// in shared memory; a term that is not counted is 0, which changes no
// non-negative sum) and every lane adds the eight entries one after another.
// All 32 lanes of a warp call this together (has: the group holds an edge), and
// a group's results are the same in all of its lanes.  Returns true when the
// reference writes a new cost for the edge.  QUALITY: quality mode (FP64 quadric
// terms and the chosen collapse position in epos); compiled separately so the
// reference's path carries none of it.
template <bool QUALITY>
__device__ __forceinline__ bool edge_cost_group(const CostArgs &A, bool has, int u, int v, bool inv_u, bool inv_v,
                                                float tres, float edge_s, int is_stuck, uint32_t &out, int e,
                                                float4 *terms)
{
    constexpr unsigned kAll = 0xffffffffu;
    const int gl = threadIdx.x & 7, shift = threadIdx.x & 24;
    bool written = false, live = has;
    out = 0xFFFFFFFFu;
    V3 v0 = {0.f, 0.f, 0.f}, v1 = v0;
    int ua = 0, ub = 0, va = 0, vb = 0;
    if (has) {
        v0 = v3(A.pts[u]);
        v1 = v3(A.pts[v]);
        if constexpr (QUALITY) {  // an edge whose cost is not rewritten collapses to its midpoint
            const V3 m0 = vmid(v0, v1);
            if (gl == 0) A.epos[e] = make_float4(m0.x, m0.y, m0.z, 0.f);
        }
        if (inv_u && inv_v) {
            written = true;
            live = false;
        } else if (is_stuck) {
            live = false;
        } else {
            ua = A.first_near[u];
            ub = A.first_near[u + 1];
            va = A.first_near[v];
            vb = A.first_near[v + 1];
        }
    }
    // the link condition: pairs of equal next vertices, exactly two wanted
    int dup = 0;
    for (int a0 = ua; __any_sync(kAll, live && a0 < ub); a0 += 8) {
        const int a = a0 + gl;
        const bool ha = live && a < ub;
        const int iu = ha ? A.nxt[a] : 0;
        for (int b0 = va; __any_sync(kAll, live && a0 < ub && b0 < vb); b0 += 8) {
            const int b = b0 + gl;
            const int iv = live && b < vb ? A.nxt[b] : 0;
            const int n = live ? vb - b0 : 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int x = __shfl_sync(kAll, iv, j, 8);
                dup += ha && j < n && x == iu;
            }
        }
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) dup += __shfl_xor_sync(kAll, dup, o);
    if (live && dup != 2) {
        written = dup > 2;
        live = false;
    }
    // the collapse position: the midpoint (the reference), or in quality mode
    // the FP64 quadric's minimiser
    V3 mid = vmid(v0, v1);
    if constexpr (QUALITY) {
        if (live) {
            mid = qem_position(A.quad64 + 10 * (size_t)u, A.quad64 + 10 * (size_t)v, v0, v1);
            if (gl == 0) A.epos[e] = make_float4(mid.x, mid.y, mid.z, 0.f);
        }
    }
    float elen = 0.0f, Qa = 0.0f;
    int nedge = 0, ntri = 0;
    bool flip = false;
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
        const int w = pass ? v : u, other = pass ? u : v;
        const int lo = pass ? va : ua, hi = pass ? vb : ub;
        for (int a0 = lo; __any_sync(kAll, live && a0 < hi); a0 += 8) {
            const int a = a0 + gl;
            float4 term = make_float4(0.f, 0.f, 0.f, 0.f);
            if (live && a < hi) {
                const int f = A.near_tris[a];
                const int4 t = A.tris[f];
                const float4 l = A.elen[f];
                if (t.x > t.y) { term.x = l.x; nedge++; }
                if (t.y > t.z) { term.y = l.y; nedge++; }
                if (t.z > t.x) { term.z = l.z; nedge++; }
                if (!face_has(t, other)) {
                    const V3 o0 = v3(A.pts[t.x]), o1 = v3(A.pts[t.y]), o2 = v3(A.pts[t.z]);
                    const V3 n0 = t.x == w ? mid : o0;
                    const V3 n1 = t.y == w ? mid : o1;
                    const V3 n2 = t.z == w ? mid : o2;
                    // the unchanged face's unit normal is the face plane's (same expression)
                    const V3 on = v3(A.plane[f]);
                    const V3 c = vcross(vsub(n1, n0), vsub(n2, n0));
                    flip = flip || normal_flips(on, c);
                    term.w = skinny_term(n0, n1, n2);
                    ntri++;
                }
            }
            terms[gl] = term;
            __syncwarp();
            if (live && a0 < hi) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float4 x = terms[j];
                    elen += x.x;
                    elen += x.y;
                    elen += x.z;
                    Qa += x.w;
                }
            }
            __syncwarp();
        }
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        nedge += __shfl_xor_sync(kAll, nedge, o);
        ntri += __shfl_xor_sync(kAll, ntri, o);
    }
    const bool any_flip = (__ballot_sync(kAll, flip) >> shift & 255u) != 0;
    if (!live) return written;
    if (any_flip) return true;
    elen = edge_length_term(elen, nedge, v0, v1, tres, edge_s);
    out = edge_cost_sum<QUALITY>(A, u, v, mid, elen, Qa, ntri, tres, edge_s);
    return true;
}

// The edge-cost pass by groups, in leaf order too: a warp takes kGroupLeaves
// consecutive leaves, lists their faces' edges in shared memory (each face owns
// its 0-3 descending edges) and its four groups take the list in turn, so
// neighbouring groups gather neighbouring vertices.  Costs are indexed by edge,
// so the order of work does not change them.
constexpr int kGroupLeaves = 8;  // few, so that a small mesh has a warp for every dozen edges

template <bool QUALITY>
__global__ void __launch_bounds__(kThreads, 4) k_edge_cost_group(CostArgs A, const int *order, int L, const int *first_edge)
{
    chain_wait();
    constexpr unsigned kAll = 0xffffffffu;
    __shared__ int s_list[kThreads / 32][3 * kGroupLeaves];
    __shared__ float4 s_terms[kThreads];
    const int lane = threadIdx.x & 31;
    int *list = s_list[threadIdx.x >> 5];
    float4 *terms = s_terms + (threadIdx.x & ~7);
    const long long step = (long long)gridDim.x * (kThreads / 32) * kGroupLeaves;
    for (long long base = (((long long)blockIdx.x * kThreads + threadIdx.x) >> 5) * kGroupLeaves; base < L; base += step) {
        const long long p = base + lane;
        const int f = lane < kGroupLeaves && p < L ? order[p] : -1;  // -1: past the end, or removed since the sort
        const int fe = f >= 0 ? first_edge[f] : 0;
        const int c = f >= 0 ? first_edge[f + 1] - fe : 0;
        const int inc = warp_incl_scan(c), total = __shfl_sync(kAll, inc, 31);
        for (int j = 0; j < c; ++j) list[inc - c + j] = fe + j;
        __syncwarp();
        for (int q0 = 0; q0 < total; q0 += 4) {
            const int q = q0 + (lane >> 3);
            const bool has = q < total;
            const int e = has ? list[q] : 0;
            const int2 ed = has ? A.edges[e] : make_int2(0, 0);
            // a batch has its mesh's own parameters, invalid table and stale costs (mesh-local numbers)
            bool inv_u = false, inv_v = false;
            float tres = A.tres, edge_s = A.edge_s;
            int stuck = A.is_stuck;
            uint32_t *stale = A.edge_cost + e;
            if (has && A.slots) {
                const int r = A.vslot[ed.x];
                const SlotInfo &S = A.slots[r];
                stale = S.edge_cost + (e - A.scnt[r].edge_off);
                inv_u = S.invalid[ed.x - S.vert_off];
                inv_v = S.invalid[ed.y - S.vert_off];
                tres = S.tres;
                edge_s = *S.scale;
                stuck = S.is_stuck;
            } else if (has) {
                inv_u = A.invalid[ed.x];
                inv_v = A.invalid[ed.y];
            }
            uint32_t c;
            const bool written = edge_cost_group<QUALITY>(A, has, ed.x, ed.y, inv_u, inv_v, tres, edge_s, stuck, c, e,
                                                          terms);
            if (has && (lane & 7) < 2) {
                if (!written) c = *stale;  // the reference keeps the previous round's value
                else if ((lane & 7) == 0) *stale = c;
                atomicMin(&A.vmin[(lane & 7) ? ed.y : ed.x], ((unsigned long long)c << 32) | (unsigned)e);
            }
        }
        __syncwarp();
    }
}

__device__ __forceinline__ bool is_skinny(V3 p, V3 q, V3 r)
{
    V3 pq = vsub(q, p), pr = vsub(r, p), qr = vsub(r, q);
    float lpq = sqrtf(vdot(pq, pq)), lpr = sqrtf(vdot(pr, pr)), lqr = sqrtf(vdot(qr, qr));
    float ml = fmaxf(lpq, fmaxf(lpr, lqr));
    V3 c = vcross(pq, pr);
    float thr = (float)(1e-6 * (double)ml * (double)ml);
    float area = 0.5f * sqrtf(c.x * c.x + c.y * c.y + c.z * c.z);
    return area < thr;
}

struct CollapseArgs {
    const int2 *edges;
    const int *n_edges;
    const uint32_t *edge_cost;
    const unsigned long long *vmin;
    const int *first_near;
    const int *near_tris;
    const float4 *opts;
    const int4 *otris;
    float4 *pts;
    int4 *tris;
    int *occ;
    int *eflag;
    uint32_t collapse_t;
    const SlotInfo *slots;  // batch mode (null otherwise)
    const SlotCounters *scnt;
    const int *vslot;
    const float4 *epos;  // quality mode: the position the edge cost chose (null: the midpoint)
};

// The independent set: every lane tests its edge's threshold and key (most edges
// fail at once); the one-rings of those that pass are then checked by groups of
// eight lanes, four edges at a time -- a chain of a dozen faces, three dependent
// loads each, when one thread walks it.  The flags' scan is the collapse list, and
// the winners' collapses run over that list (k_collapse_apply), so no warp carries
// idle lanes through a collapse.  Winners have disjoint one-rings, and the tests
// read only the round input (otris) and the key minima, so splitting the two
// changes nothing.
__global__ void __launch_bounds__(kThreads) k_collapse(CollapseArgs A)
{
    chain_wait();
    constexpr unsigned kAll = 0xffffffffu;
    const int E = *A.n_edges;
    const int lane = threadIdx.x & 31, gl = lane & 7, shift = lane & 24;
    const long long step = (long long)gridDim.x * blockDim.x;
    for (long long base = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < E; base += step) {
        const int e = (int)(base + lane);
        int2 ed = make_int2(0, 0);
        unsigned long long key = 0;
        bool pass = false;
        if (base + lane < E) {
            uint32_t c, collapse_t;
            if (!A.slots) {
                c = A.edge_cost[e];
                collapse_t = A.collapse_t;
            } else {
                const int r = A.vslot[A.edges[e].x];
                c = A.slots[r].edge_cost[e - A.scnt[r].edge_off];
                collapse_t = A.slots[r].collapse_t;
            }
            if (c <= collapse_t) {
                ed = A.edges[e];
                key = ((unsigned long long)c << 32) | (unsigned)e;
                pass = A.vmin[ed.x] == key && A.vmin[ed.y] == key;
            }
        }
        unsigned won = 0;
        for (unsigned todo = __ballot_sync(kAll, pass); todo;) {
            int src = 0;
            bool has = false;
#pragma unroll
            for (int k = 0; k < 4; ++k) {  // the next four edges, one per group
                if (shift == 8 * k && todo) {
                    src = __ffs(todo) - 1;
                    has = true;
                }
                todo &= todo - 1;
            }
            const int u = __shfl_sync(kAll, ed.x, src), v = __shfl_sync(kAll, ed.y, src);
            const unsigned long long k0 = __shfl_sync(kAll, key, src);
            int ua = 0, du = 0, va = 0, d = 0;  // the two rings as one list
            if (has) {
                ua = A.first_near[u];
                du = A.first_near[u + 1] - ua;
                va = A.first_near[v] - du;
                d = A.first_near[v + 1] - va;
            }
            bool less = false;
            for (int i0 = 0; __any_sync(kAll, i0 < d); i0 += 8) {
                const int i = i0 + gl;
                if (i < d) {
                    const int4 t = A.otris[A.near_tris[(i < du ? ua : va) + i]];  // round input: never written here
                    less = less || A.vmin[t.x] < k0 || A.vmin[t.y] < k0 || A.vmin[t.z] < k0;
                }
            }
            const unsigned lost = __ballot_sync(kAll, less);
            const unsigned mine = has && ((lost >> shift) & 255u) == 0 ? 1u << src : 0u;
            won |= __reduce_or_sync(kAll, mine);
        }
        if (base + lane < E) A.eflag[e] = (int)(won >> lane & 1u);
    }
}

// Collapse of each winner (list[0, *n_list)), by a group of eight lanes: u moves to
// the midpoint (the quality mode's chosen position), v goes, faces holding both
// die and v's faces take u; if a surviving one-ring face would be skinny nothing
// is changed, and the edge stays in the collapsed list.  The one-ring's faces are
// marked as those that query the tree.
template <bool QUALITY>
__global__ void __launch_bounds__(kThreads) k_collapse_apply(CollapseArgs A, const int *list, const int *n_list,
                                                             uint8_t *active)
{
    chain_wait();
    constexpr unsigned kAll = 0xffffffffu;
    const int N = *n_list;
    const int lane = threadIdx.x & 31, gl = lane & 7, shift = lane & 24;
    const long long warps = (long long)gridDim.x * (kThreads / 32);
    for (long long w = ((long long)blockIdx.x * kThreads + threadIdx.x) >> 5; w * 4 < N; w += warps) {
        const long long k = w * 4 + (lane >> 3);
        int u = 0, v = 0, ua = 0, du = 0, va = 0, d = 0;
        V3 mid = {0.f, 0.f, 0.f};
        if (k < N) {
            const int e = list[k];
            const int2 ed = A.edges[e];
            u = ed.x;
            v = ed.y;
            ua = A.first_near[u];
            du = A.first_near[u + 1] - ua;
            va = A.first_near[v] - du;
            d = A.first_near[v + 1] - va;
            if constexpr (QUALITY) mid = v3(A.epos[e]);  // the position the edge cost chose
            else mid = vmid(v3(A.opts[u]), v3(A.opts[v]));
        }
        // the one-rings after the collapse, from the round input (no other winner touches
        // them).  A ring lists a face once for each corner there: one that holds v twice
        // goes, as its second turn finds the u that the first one left.
        auto moved = [&](int i, int &f) {
            f = A.near_tris[(i < du ? ua : va) + i];
            int4 t = A.otris[f];
            const int at_v = (t.x == v) + (t.y == v) + (t.z == v);
            if (face_has(t, i < du ? v : u) || at_v > 1) t = make_int4(-1, -1, -1, 0);
            else if (t.x == v) t.x = u;
            else if (t.y == v) t.y = u;
            else if (t.z == v) t.z = u;
            return t;
        };
        bool skinny = false;
        for (int i0 = 0; __any_sync(kAll, i0 < d); i0 += 8) {
            if (i0 + gl >= d) continue;
            int f;
            const int4 t = moved(i0 + gl, f);
            active[f] = 1;
            if (t.x == -1) continue;
            auto at = [&](int x) { return x == u ? mid : v3(A.opts[x]); };
            skinny = skinny || is_skinny(at(t.x), at(t.y), at(t.z));
        }
        if (((__ballot_sync(kAll, skinny) >> shift) & 255u) != 0 || d == 0) d = 0;  // rolled back
        for (int i0 = 0; __any_sync(kAll, i0 < d); i0 += 8) {
            if (i0 + gl >= d) continue;
            int f;
            const int4 t = moved(i0 + gl, f);
            if (t.x == -1 || i0 + gl >= du) A.tris[f] = t;
        }
        if (d > 0 && gl == 0) {
            A.pts[u] = make_float4(mid.x, mid.y, mid.z, 0.f);
            A.pts[v] = make_float4(0.f, 0.f, 0.f, 0.f);
            A.occ[v] = 0;
        }
    }
}

// Coincident-endpoint collapses: positions are read (k_cleanup) before any write;
// the writes are applied in edge order by one thread.  Flagged edges are rare
// (exactly equal coordinates), so one block of kLineThreads finds them chunk by
// chunk and its thread 0 applies each chunk's edges in order.  Other blocks of the
// same launch may have written the faces and flags: these loads bypass the L1.
constexpr int kLineThreads = 256;
constexpr int kLinePerThread = 8;

__device__ __forceinline__ void line_collapse(int u, int v, const int *first_near, const int *near_tris, float4 *pts,
                                              int4 *tris, int *occ)
{
    pts[v] = make_float4(0.f, 0.f, 0.f, 0.f);
    occ[v] = 0;
    for (int a = first_near[u]; a < first_near[u + 1]; ++a) {
        int f = near_tris[a];
        if (face_has(__ldcg(&tris[f]), v)) tris[f] = make_int4(-1, -1, -1, 0);
    }
    for (int a = first_near[v]; a < first_near[v + 1]; ++a) {
        int f = near_tris[a];
        int4 t = __ldcg(&tris[f]);
        if (face_has(t, u)) t = make_int4(-1, -1, -1, 0);
        else if (t.x == v) t.x = u;
        else if (t.y == v) t.y = u;
        else if (t.z == v) t.z = u;
        tris[f] = t;
    }
}

// Calls on_edge(e) on thread 0 for every flagged e < E, in ascending order.
template <typename OnEdge>
__device__ __forceinline__ void for_flagged_in_order(const int *eflag, int E, OnEdge on_edge)
{
    __shared__ int s_idx[kLineThreads * kLinePerThread];
    for (long long base = 0; base < E; base += kLineThreads * kLinePerThread) {
        int local[kLinePerThread];
        int c = 0;
#pragma unroll
        for (int k = 0; k < kLinePerThread; ++k) {
            long long e = base + (long long)threadIdx.x * kLinePerThread + k;
            if (e < E && __ldcg(&eflag[e])) local[c++] = (int)e;
        }
        int total;
        int off = block_excl_scan<kLineThreads>(c, total);
        for (int k = 0; k < c; ++k) s_idx[off + k] = local[k];
        __syncthreads();
        if (threadIdx.x == 0)
            for (int i = 0; i < total; ++i) on_edge(s_idx[i]);
        __syncthreads();
    }
}

// After the collapses: faces with a repeated index go, and edges with coincident
// end points are flagged and counted; the last block to finish (a ticket, no
// waiting) applies those, and sets the prefix of the collapsed list that the
// reference's undo check looks at.  The faces of the considered coincident edges
// join those that query the tree.  A batch applies them in k_b_line_apply.
template <bool BATCH>
__global__ void __launch_bounds__(kLineThreads) k_cleanup(int4 *tris, int m, const int2 *edges, const int *n_edges,
                                                          float4 *pts, int *eflag, const int *first_near,
                                                          const int *near_tris, int *occ, int *collapsed,
                                                          uint8_t *active, RoundCounters *cnt)
{
    chain_wait();
    const int E = *n_edges;
    __shared__ bool s_last;
    int local = 0;
    PAMO_GRID_STRIDE(i, m > E ? m : E)
    {
        if (i < m) {
            const int4 t = tris[i];
            if (!face_dead(t) && (t.x == t.y || t.y == t.z || t.z == t.x)) tris[i] = make_int4(-1, -1, -1, 0);
        }
        if (i < E) {
            const int2 ed = edges[i];
            const float4 p = pts[ed.x], q = pts[ed.y];
            const int f = p.x == q.x && p.y == q.y && p.z == q.z;
            eflag[i] = f;
            local += f;
        }
    }
    if (local) atomicAdd(&cnt->n_line, local);
    if (BATCH) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(&cnt->ticket, 1) == (int)gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    if (!s_last) return;
    const int nm = cnt->n_main, lines = *(volatile int *)&cnt->n_line;
    const int window = ((nm + 511) / 512) * 512;  // grid of the reference's undo-candidate launch
    int k = 0;
    if (lines > 0)
        for_flagged_in_order(eflag, E, [&](int e) {
            const int u = edges[e].x, v = edges[e].y;
            if (nm + k < window)
                for (int side = 0; side < 2; ++side) {
                    const int w = side ? v : u;
                    for (int a = first_near[w]; a < first_near[w + 1]; ++a) active[near_tris[a]] = 1;
                }
            collapsed[nm + k++] = e;
            line_collapse(u, v, first_near, near_tris, pts, tris, occ);
        });
    if (threadIdx.x != 0) return;
    cnt->n_line = k;
    cnt->n_total = nm + k;
    cnt->n_considered = cnt->n_total < window ? cnt->n_total : window;
}

__device__ __forceinline__ bool box_overlap(float4 alo, float4 ahi, float4 qlo, float4 qhi)
{
    return !(ahi.x < qlo.x || qhi.x < alo.x || ahi.y < qlo.y || qhi.y < alo.y || ahi.z < qlo.z || qhi.z < alo.z);
}

__device__ __forceinline__ int shared_indices(int4 a, int4 b)
{
    return (a.x == b.x) + (a.x == b.y) + (a.x == b.z) + (a.y == b.x) + (a.y == b.y) + (a.y == b.z) +
           (a.z == b.x) + (a.z == b.y) + (a.z == b.z);
}

// The leaves whose boxes overlap each listed leaf's, as candidate pairs: a group
// of eight lanes per query (TreeWalk), four queries a warp.  A pair of two
// selected faces is emitted once (by the lower index); pairs sharing
// `skip_shared` or more vertex indices are dropped: 2 for the reference's test,
// which never reports pairs sharing an edge; 4 (none) for the exact test of
// quality mode.  ranges (a batch): a query stays in its own mesh's run of leaves.
//
// A walk is a chain of dependent loads, so its length sets the time: one thread
// per query on a binary hierarchy followed ~100 nodes and loaded each leaf's
// face, flag and corners one after another (90 / 120 / 222 us a pass with its query
// list, mean over the rounds of meshes of 5k / 200k / 2M faces).  Here a step tests
// eight boxes, and a leaf's record comes with its box: 19 / 27 / 83 us.  The pairs gather in
// shared memory and leave 32 at a time, one counter update for each 32.
constexpr int kQueryThreads = 256;

template <bool BATCH>
__global__ void __launch_bounds__(kQueryThreads) k_query(const __grid_constant__ TreeView T,
                                                         const int *__restrict__ qlist,
                                                         RoundCounters *cnt, uint2 *pairs, long long cap_pairs,
                                                         int skip_shared, const int2 *__restrict__ ranges,
                                                         const int *__restrict__ vslot)
{
    chain_wait();
    __shared__ uint2 s_pairs[kQueryThreads / 32][64];
    __shared__ int2 s_lvl[kTreeMaxLevels];  // indexed by a lane's own level
    T.levels(s_lvl);
    uint2 *buf = s_pairs[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31, gl = lane & 7, shift = lane & 24;
    const unsigned below = (1u << lane) - 1u;
    const int N = cnt->n_query;
    int held = 0;  // pairs in buf
    auto flush = [&](int n) {
        int first = 0;
        if (lane == 0) first = atomicAdd(&cnt->n_pairs, n);
        first = __shfl_sync(0xffffffffu, first, 0);
        if (lane < n) {
            const long long pos = (long long)first + lane;
            if (pos < cap_pairs) pairs[pos] = buf[lane];
            else atomicAdd(&cnt->pair_overflow, 1);
        }
    };
    const long long warps = (long long)gridDim.x * (kQueryThreads / 32);
    for (long long w = ((long long)blockIdx.x * kQueryThreads + threadIdx.x) >> 5; w * 4 < N; w += warps) {
        const long long k = w * 4 + (lane >> 3);
        const bool has = k < N;
        const int q = has ? qlist[k] : 0;
        const int4 t = T.leaf[q];
        const float4 qlo = T.boxes[2 * (size_t)q], qhi = T.boxes[2 * (size_t)q + 1];
        int2 rg = make_int2(0, 0);
        if (BATCH && has) rg = ranges[vslot[t.x]];
        TreeWalk wk;
        wk.start(T, has);
        while (__any_sync(0xffffffffu, wk.run)) {
            bool hit = false, emit = false;
            int other = 0;
            const int node = 8 * wk.g + gl;
            if (wk.run) {
                const int2 level = s_lvl[wk.lvl];
                const size_t b = 2 * ((size_t)level.x + node);
                const float4 lo = T.boxes[b], hi = T.boxes[b + 1];
                const bool leaf = wk.lvl == 0 && node < T.L;
                const int4 r = leaf ? T.leaf[node] : make_int4(-1, -1, -1, kLeafDead);
                hit = box_overlap(lo, hi, qlo, qhi) && node <= level.y;
                if (BATCH) {
                    const long long first = (long long)node << (3 * wk.lvl), end = ((long long)node + 1) << (3 * wk.lvl);
                    hit = hit && first < rg.y && end > rg.x;
                }
                if (leaf && hit && node != q && r.w != kLeafDead) {
                    other = leaf_face(r.w);
                    emit = !(r.w >= 0 && other < t.w) && shared_indices(t, r) < skip_shared;
                }
            }
            const unsigned hits = __ballot_sync(0xffffffffu, hit), em = __ballot_sync(0xffffffffu, emit);
            if (em) {
                if (emit) buf[held + __popc(em & below)] = make_uint2((unsigned)t.w, (unsigned)other);
                held += __popc(em);
                __syncwarp();
                if (held >= 32) {
                    flush(32);
                    held -= 32;
                    const uint2 rest = buf[32 + lane];
                    __syncwarp();
                    buf[lane] = rest;
                    __syncwarp();
                }
            }
            if (wk.run) wk.advance(T, (hits >> shift) & 255u);
        }
    }
    if (held > 0) flush(held);
}

__device__ __forceinline__ void load_face(const float4 *pts, int4 t, float out[3][3], int idx[3])
{
    idx[0] = t.x; idx[1] = t.y; idx[2] = t.z;
    float4 p[3] = {pts[t.x], pts[t.y], pts[t.z]};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        out[a][0] = p[a].x; out[a][1] = p[a].y; out[a][2] = p[a].z;
    }
}

template <bool EXACT>
__global__ void __launch_bounds__(kThreads) k_pairs(const uint2 *pairs, RoundCounters *cnt,
                                                    long long cap_pairs, const float4 *__restrict__ pts,
                                                    const int4 *__restrict__ tris, uint8_t *isect, float eps)
{
    chain_wait();
    long long N = cnt->n_pairs < cap_pairs ? cnt->n_pairs : cap_pairs;
    PAMO_GRID_STRIDE(k, N)
    {
        uint2 pr = pairs[k];
        if constexpr (EXACT) {
            // quality mode: the acceptance checker's exact predicate (exact.cuh);
            // a degenerate face counts as intersecting
            exact::P3 P[3], Q[3];
            const int4 ta = tris[pr.x], tb = tris[pr.y];
            const int ia[3] = {ta.x, ta.y, ta.z}, ib[3] = {tb.x, tb.y, tb.z};
            for (int c = 0; c < 3; ++c) {
                const float4 a = pts[ia[c]], b = pts[ib[c]];
                P[c] = {a.x, a.y, a.z};
                Q[c] = {b.x, b.y, b.z};
            }
            const bool da = exact::tri_degenerate(P, ia), db = exact::tri_degenerate(Q, ib);
            const bool hit = !da && !db && exact::faces_intersect(P, ia, Q, ib);
            if (da || hit) isect[pr.x] = 1;
            if (db || hit) isect[pr.y] = 1;
            if (da || db || hit) cnt->n_hit = 1;
            continue;
        }
        float A[3][3], B[3][3];
        int ia[3], ib[3];
        load_face(pts, tris[pr.x], A, ia);
        load_face(pts, tris[pr.y], B, ib);
        if (pair_flag_directed(A, ia, B, ib, eps) || pair_flag_directed(B, ib, A, ia, eps)) {
            isect[pr.x] = 1;
            isect[pr.y] = 1;
            cnt->n_hit = 1;
        }
    }
}

// The considered edges with an intersecting face in their one-rings: flags and
// count.  The host scans the flags into the undo list only if there are any.
__global__ void k_undo_flags(const int *collapsed, RoundCounters *cnt, const int2 *edges,
                             const int *first_near, const int *near_tris, const uint8_t *isect, int *uflag)
{
    chain_wait();
    if (!cnt->n_hit) return;  // no pair intersects (n_undo is 0)
    const int N = cnt->n_considered;
    int local = 0;
    PAMO_GRID_STRIDE(p, N)
    {
        int2 ed = edges[collapsed[p]];
        int hit = 0;
        for (int a = first_near[ed.x]; a < first_near[ed.x + 1] && !hit; ++a) hit = isect[near_tris[a]];
        for (int a = first_near[ed.y]; a < first_near[ed.y + 1] && !hit; ++a) hit = isect[near_tris[a]];
        uflag[p] = hit;
        local += hit;
    }
    if (local) atomicAdd(&cnt->n_undo, local);
}

// The listed collapses taken back (undo_idx: positions in the collapsed list): the
// one-rings restored from the round input and, if `active` is given, selected for
// the next query (they alone: cleared before).  The undo list gets the end
// points' vertices from `first` on, through the previous round's map: pts_map at
// this point (cusimp_free.cu:869-878 runs before :1042-1045).  Thread 0 resets the
// pass's counters.
__global__ void k_undo_apply(const int *undo_idx, int N, const int *collapsed, const int2 *edges,
                             const int *first_near, const int *near_tris, const float4 *opts, const int4 *otris,
                             float4 *pts, int4 *tris, int *occ, uint8_t *active, const int *pts_map, int *undo_list,
                             int first, const SlotInfo *slots, const SlotCounters *scnt, const int *vslot,
                             RoundCounters *cnt)
{
    chain_wait();
    if (blockIdx.x == 0 && threadIdx.x == 0)
        cnt->n_pairs = cnt->pair_overflow = cnt->n_query = cnt->n_hit = cnt->n_undo = 0;
    PAMO_GRID_STRIDE(k, N)
    {
        const int2 ed = edges[collapsed[undo_idx[k]]];
        const int u = ed.x, v = ed.y;
        occ[v] = 1;
        pts[u] = opts[u];
        pts[v] = opts[v];
        for (int side = 0; side < 2; ++side) {
            const int w = side ? v : u;
            for (int a = first_near[w]; a < first_near[w + 1]; ++a) {
                const int f = near_tris[a];
                tris[f] = otris[f];
                if (active) active[f] = 1;
            }
        }
        if (!slots) {
            undo_list[first + 2 * k] = pts_map[u];
            undo_list[first + 2 * k + 1] = pts_map[v];
        } else {  // the mesh's own list and map, in its own numbers
            const int r = vslot[u];
            const SlotInfo &S = slots[r];
            const int j = S.pass_first + 2 * ((int)k - scnt[r].undo_off);
            S.undo_list[j] = S.pts_map[u - S.vert_off];
            S.undo_list[j + 1] = S.pts_map[v - S.vert_off];
        }
    }
}

// undo_list[first + i] = pts_map[tmp_undo[i]], through the previous round's map
__global__ void k_rearrange(const int *tmp_undo, const int *pts_map, int *undo_list, int first, int count)
{
    PAMO_GRID_STRIDE(i, count) undo_list[first + i] = pts_map[tmp_undo[i]];
}

__global__ void k_mark_invalid(const int *undo_in, int n, uint8_t *table)
{
    PAMO_GRID_STRIDE(i, n) table[undo_in[i]] = 1;
}

// Compaction by the scans' positions, and the tree's leaves renumbered: leaf p's
// face gets its compacted index, or -1 if removed.
__global__ void k_compact(const float4 *pts, const int *occ, const int *pts_map, int n, const int4 *tris,
                          const int *fpos, int m, float4 *opts, int4 *otris, int *vals, int L, RoundCounters *cnt)
{
    chain_wait();
    long long N = n > m ? n : m;
    N = N > L ? N : L;
    PAMO_GRID_STRIDE(i, N)
    {
        if (i < n && occ[i]) opts[pts_map[i]] = pts[i];
        if (i < m) {
            const int4 t = tris[i];
            if (t.x >= 0) otris[fpos[i]] = make_int4(pts_map[t.x], pts_map[t.y], pts_map[t.z], 0);
        }
        if (i < L) {
            const int f = vals[i];
            vals[i] = f >= 0 && tris[f].x >= 0 ? fpos[f] : -1;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        cnt->n_pts_next = pts_map[n];
        cnt->n_tris_next = m > 0 ? fpos[m - 1] + (tris[m - 1].x >= 0) : 0;
    }
}

__global__ void k_validate_faces(const int *tris, int m, int n, int *bad)
{
    int local = 0;
    PAMO_GRID_STRIDE(f, m)
    {
        int a = tris[3 * f], b = tris[3 * f + 1], c = tris[3 * f + 2];
        bool dead = a == -1 && b == -1 && c == -1;
        bool ok = a >= 0 && a < n && b >= 0 && b < n && c >= 0 && c < n;
        local += !(dead || ok);
    }
    if (local) atomicAdd(bad, local);
}

__global__ void k_validate_range(const int *v, int count, int hi, int *bad)
{
    int local = 0;
    PAMO_GRID_STRIDE(i, count) local += (v[i] < 0 || v[i] > hi);
    if (local) atomicAdd(bad, local);
}

// ---------------------------------------------------------------------------
// Batch kernels.  Per-mesh loops use blockIdx.y = the mesh's rank and stride
// over the mesh's range with blockIdx.x.
#define SLOT_STRIDE(j, count) \
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < (long long)(count); j += (long long)blockDim.x * gridDim.x)

// Before the round, per mesh, as the single-mesh round does (cusimp_free.cu:899-916):
// stuck: the undo list starts with the previous one mapped through the previous
// vertex map; not stuck with a non-empty list: the invalid table is cleared.
__global__ void k_b_pre_copy(const SlotInfo *slots)
{
    chain_wait();
    const SlotInfo S = slots[blockIdx.y];
    if (S.is_stuck) {
        SLOT_STRIDE(j, S.n_undo_in)
        {
            int x = S.undo_prev[j];
            S.tmp_undo[j] = x;
            S.undo_list[j] = S.pts_map[x];
        }
    } else if (S.clear_invalid) {
        SLOT_STRIDE(j, S.cap_v) S.invalid[j] = 0;
    }
}

__global__ void k_b_pre_mark(const SlotInfo *slots)
{
    chain_wait();
    const SlotInfo S = slots[blockIdx.y];
    SLOT_STRIDE(j, S.n_undo_in) S.invalid[S.undo_prev[j]] = 1;
}

__global__ void k_b_vslot(const SlotInfo *slots, int *vslot)
{
    chain_wait();
    const SlotInfo S = slots[blockIdx.y];
    SLOT_STRIDE(j, S.n) vslot[S.vert_off + j] = (int)blockIdx.y;
}

// first packed edge and edge count of each mesh (first_edge has m + 1 entries)
__global__ void k_b_edge_off(const SlotInfo *slots, const int *first_edge, SlotCounters *scnt, int K)
{
    chain_wait();
    PAMO_GRID_STRIDE(r, K)
    {
        const SlotInfo &S = slots[r];
        scnt[r].edge_off = first_edge[S.face_off];
        scnt[r].n_edges = first_edge[S.face_off + S.m] - first_edge[S.face_off];
    }
}

// pos = exclusive scan over the packed edges of a flag, total = its sum:
// each mesh's first entry and count in the compacted list.
__device__ __forceinline__ void seg_of_scan(const int *pos, int total, int n_all, int first, int count, int &off,
                                            int &cnt)
{
    off = first < n_all ? pos[first] : total;
    int end = first + count < n_all ? pos[first + count] : total;
    cnt = end - off;
}

__global__ void k_b_main(const int *pos, const RoundCounters *cnt, SlotCounters *scnt, int K)
{
    chain_wait();
    PAMO_GRID_STRIDE(r, K)
    {
        int off, c;
        seg_of_scan(pos, cnt->n_main, cnt->n_edges, scnt[r].edge_off, scnt[r].n_edges, off, c);
        scnt[r].main_off = off;
        scnt[r].n_main = c;
    }
}

// Coincident-endpoint collapses over the whole batch (the single-mesh version's
// order: positions read before any write, writes in edge order), and each
// mesh's undo-candidate window: its collapsed edges then its coincident ones,
// cut at the reference's launch-grid roundup of its own collapsed count.
__global__ void __launch_bounds__(kLineThreads) k_b_line_apply(const int2 *edges, const int *n_edges,
                                                               const int *eflag, const int *first_near,
                                                               const int *near_tris, float4 *pts, int4 *tris, int *occ,
                                                               int *line_list, const int *vslot, RoundCounters *cnt,
                                                               SlotCounters *scnt, int K)
{
    chain_wait();
    const int E = *n_edges;
    for (int r = threadIdx.x; r < K; r += blockDim.x) scnt[r].n_line = 0;
    __syncthreads();
    int k = 0;
    if (cnt->n_line > 0)
        for_flagged_in_order(eflag, E, [&](int e) {
            int u = edges[e].x, v = edges[e].y;
            line_list[k++] = e;
            scnt[vslot[u]].n_line++;
            line_collapse(u, v, first_near, near_tris, pts, tris, occ);
        });
    if (threadIdx.x != 0) return;
    cnt->n_line = k;
    cnt->n_total = cnt->n_main + k;
    int line_off = 0, cand_off = 0;
    for (int r = 0; r < K; ++r) {
        SlotCounters &c = scnt[r];
        c.line_off = line_off;
        line_off += c.n_line;
        int total = c.n_main + c.n_line;
        int window = ((c.n_main + 511) / 512) * 512;
        c.n_considered = total < window ? total : window;
        c.cand_off = cand_off;
        cand_off += c.n_considered;
    }
    cnt->n_considered = cand_off;
}

__global__ void k_b_cand_fill(const int *collapsed, const int *line_list, const int2 *edges, const int *vslot,
                              const RoundCounters *cnt, const SlotCounters *scnt, int *cand,
                              const int *first_near, const int *near_tris, uint8_t *active)
{
    chain_wait();
    const int nm = cnt->n_main, nl = cnt->n_line;
    PAMO_GRID_STRIDE(p, (long long)nm + nl)
    {
        int e, r, k;
        if (p < nm) {
            e = collapsed[p];
            r = vslot[edges[e].x];
            k = (int)p - scnt[r].main_off;
        } else {
            int q = (int)p - nm;
            e = line_list[q];
            r = vslot[edges[e].x];
            k = scnt[r].n_main + q - scnt[r].line_off;
            if (k < scnt[r].n_considered)  // its faces query the tree (the collapses marked theirs)
                for (int side = 0; side < 2; ++side) {
                    const int w = side ? edges[e].y : edges[e].x;
                    for (int a = first_near[w]; a < first_near[w + 1]; ++a) active[near_tris[a]] = 1;
                }
        }
        if (k < scnt[r].n_considered) cand[scnt[r].cand_off + k] = e;
    }
}

__global__ void k_b_undo_counts(const int *upos, const RoundCounters *cnt, SlotCounters *scnt, int K)
{
    chain_wait();
    PAMO_GRID_STRIDE(r, K)
    {
        int off, c;
        seg_of_scan(upos, cnt->n_undo, cnt->n_considered, scnt[r].cand_off, scnt[r].n_considered, off, c);
        scnt[r].undo_off = off;
        scnt[r].n_undo = c;
    }
}

// each mesh's vertex map in its own numbers, and the copy of its undo list
__global__ void k_b_local_map(const SlotInfo *slots, const int *gmap)
{
    chain_wait();
    const SlotInfo S = slots[blockIdx.y];
    const int base = gmap[S.vert_off];
    SLOT_STRIDE(j, (long long)S.n + 1) S.pts_map[j] = gmap[S.vert_off + j] - base;
    SLOT_STRIDE(j, S.nvu) S.undo_prev[j] = S.undo_list[j];
}

__global__ void k_b_next(const SlotInfo *slots, const int *gmap, const int *fpos, SlotCounters *scnt, int K)
{
    chain_wait();
    PAMO_GRID_STRIDE(r, K)
    {
        const SlotInfo &S = slots[r];
        scnt[r].vert_off_next = gmap[S.vert_off];
        scnt[r].n_next = gmap[S.vert_off + S.n] - gmap[S.vert_off];
        scnt[r].face_off_next = fpos[S.face_off];
        scnt[r].m_next = fpos[S.face_off + S.m] - fpos[S.face_off];
    }
}

}  // namespace

void Profiler::begin(int phase, cudaStream_t s)
{
    if (!on) return;
    if (open_phase >= 0) end(s);
    if (used + 2 > kPool || n_marks >= kPool / 2) return;  // pool full: drop (collect() frees it)
    for (int k = 0; k < 2; ++k)
        if (!ev[used + k]) cudaEventCreate(&ev[used + k]);
    cudaEventRecord(ev[used], s);
    marks[n_marks][0] = phase;
    marks[n_marks][1] = used;
    open_phase = phase;
    used += 2;
}

void Profiler::end(cudaStream_t s)
{
    if (!on || open_phase < 0) return;
    cudaEventRecord(ev[marks[n_marks][1] + 1], s);
    n_marks++;
    open_phase = -1;
}

void Profiler::collect()
{
    if (!on) return;
    for (int i = 0; i < n_marks; ++i) {
        float t = 0.f;
        if (cudaEventElapsedTime(&t, ev[marks[i][1]], ev[marks[i][1] + 1]) == cudaSuccess) {
            ms[marks[i][0]] += t;
            calls[marks[i][0]]++;
        }
    }
    if (open_phase >= 0) {  // a phase still open keeps its start event, moved to slot 0
        const int slot = marks[n_marks][1];
        cudaEvent_t a = ev[0], b = ev[1];
        ev[0] = ev[slot];
        ev[1] = ev[slot + 1];
        ev[slot] = a;
        ev[slot + 1] = b;
        marks[0][0] = marks[n_marks][0];
        marks[0][1] = 0;
        used = 2;
    } else {
        used = 0;
    }
    n_marks = 0;
}

void Profiler::reset()
{
    for (int i = 0; i < PH_COUNT; ++i) {
        ms[i] = 0;
        calls[i] = 0;
    }
    n_marks = used = 0;
    open_phase = -1;
}

void Profiler::release()
{
    for (int i = 0; i < kPool; ++i)
        if (ev[i]) {
            cudaEventDestroy(ev[i]);
            ev[i] = nullptr;
        }
}

int Stage2::validate(const int *d_tris, int n, int m, const int *d_undo, int n_undo, int undo_hi, cudaStream_t s)
{
    int *bad = dev_misc + 32;
    S2_TRY_EARLY(cudaMemsetAsync(bad, 0, 4, s));
    if (m > 0) launch(k_validate_faces, grid_for(m), kThreads, 0, s, d_tris, m, n, bad);
    if (n_undo > 0) launch(k_validate_range, grid_for(n_undo), kThreads, 0, s, d_undo, n_undo, undo_hi, bad);
    S2_TRY_EARLY(cudaMemcpyAsync(hcnt, bad, 4, cudaMemcpyDeviceToHost, s));
    S2_TRY_EARLY(cudaStreamSynchronize(s));
    return hcnt->n_main == 0 ? PAMO_OK : PAMO_ERR_INVALID_ARG;
}

// ---------------------------------------------------------------------------
// buffers

void Stage2::release()
{
    void *p[] = {edge_cost, pts_map, undo_list, tmp_undo, invalid_table, opts, pts, otris, tris, occ,
                 first_near, cursor, near_tris, first_edge, edges, plane, elen4, nxt, quad, vmin, eflag, collapsed,
                 active, isect, uflag, undo_idx, fpos, qlist, pairs, scan_scratch, scan_scratch2, dev_misc, dcnt, quad64, epos};
    for (void *q : p)
        if (q) cudaFree(q);
    quad64 = nullptr;
    epos = nullptr;
    cap_q64 = cap_epos = 0;
    if (hcnt) cudaFreeHost(hcnt);
    if (h_scalars) cudaFreeHost(h_scalars);
    prof.release();
    edge_cost = nullptr; pts_map = nullptr; undo_list = nullptr; tmp_undo = nullptr; invalid_table = nullptr;
    opts = pts = nullptr; otris = tris = nullptr; occ = nullptr;
    first_near = cursor = near_tris = first_edge = nullptr; edges = nullptr; plane = quad = elen4 = nullptr;
    nxt = nullptr;
    vmin = nullptr; eflag = collapsed = nullptr; active = isect = nullptr; uflag = undo_idx = fpos = qlist = nullptr;
    pairs = nullptr; scan_scratch = scan_scratch2 = nullptr; dev_misc = nullptr; dcnt = nullptr; hcnt = nullptr; h_scalars = nullptr;
    tree.release();
    tree_carried = false;
    cap_pts = cap_tris = cap_edges = cap_undo = cap_pairs = 0;
}

int Stage2::ensure(long long n, long long m)
{
    if (n <= cap_pts && m <= cap_tris && dcnt) return PAMO_OK;
    long long cp = n > cap_pts ? n : cap_pts;
    long long ct = m > cap_tris ? m : cap_tris;
    release();
    cp = cp > 4 ? cp : 4;
    ct = ct > 4 ? ct : 4;
    long long ce = 3 * ct;
    long long cu = 16 * (cp + 1) + 6 * ct + 16;
    long long big = (cp + 1 > ce + 1 ? cp + 1 : ce + 1);
    big = big > ct + 1 ? big : ct + 1;
    scan_scratch_len = scan_scratch_ints(big);
#define ALLOC(ptr, bytes)                                             \
    do {                                                              \
        if (cudaMalloc((void **)&ptr, (size_t)(bytes)) != cudaSuccess) { \
            release();                                                \
            return PAMO_ERR_OOM;                                      \
        }                                                             \
    } while (0)
    ALLOC(edge_cost, (ce + 1) * 4);
    ALLOC(pts_map, (cp + 1) * 4);
    ALLOC(undo_list, cu * 4);
    ALLOC(tmp_undo, cu * 4);
    ALLOC(invalid_table, cp + 1);
    ALLOC(opts, (cp + 1) * 16);
    ALLOC(pts, (cp + 1) * 16);
    ALLOC(otris, (ct + 1) * 16);
    ALLOC(tris, (ct + 1) * 16);
    ALLOC(occ, (cp + 1) * 4);
    ALLOC(first_near, (cp + 1) * 4);
    ALLOC(cursor, (cp + 1) * 4);
    ALLOC(near_tris, 3 * (ct + 1) * 4);
    ALLOC(first_edge, (ct + 1) * 4);
    ALLOC(edges, (ce + 1) * 8);
    ALLOC(plane, (ct + 1) * 16);
    ALLOC(elen4, (ct + 1) * 16);
    ALLOC(nxt, 3 * (ct + 1) * 4);
    ALLOC(quad, 3 * (cp + 1) * 16);
    ALLOC(vmin, (cp + 1) * 8);
    ALLOC(eflag, (ce + 1) * 4);
    ALLOC(collapsed, (ce + 1) * 4);
    ALLOC(active, ct + 1);
    ALLOC(isect, ct + 1);
    ALLOC(uflag, (ce + 1) * 4);
    ALLOC(undo_idx, (ce + 1) * 4);
    ALLOC(fpos, (ct + 1) * 4);
    ALLOC(qlist, (ct + 1) * 4);
    ALLOC(scan_scratch, scan_scratch_len * 4);
    ALLOC(scan_scratch2, scan_scratch_len * 4);
    ALLOC(dev_misc, 256);
    ALLOC(dcnt, sizeof(RoundCounters));
#undef ALLOC
    if (cudaMallocHost((void **)&hcnt, sizeof(RoundCounters)) != cudaSuccess) {
        release();
        return PAMO_ERR_OOM;
    }
    if (cudaMallocHost((void **)&h_scalars, 64) != cudaSuccess) {
        release();
        return PAMO_ERR_OOM;
    }
    scan_scratch_init(scan_scratch, scan_scratch_len);
    scan_scratch_init(scan_scratch2, scan_scratch_len);
    // state the reference reads stale starts at zero
    cudaMemset(edge_cost, 0, (ce + 1) * 4);
    cudaMemset(pts_map, 0, (cp + 1) * 4);
    cudaMemset(undo_list, 0, cu * 4);
    cudaMemset(tmp_undo, 0, cu * 4);
    cudaMemset(invalid_table, 0, cp + 1);
    cap_pts = cp;
    cap_tris = ct;
    cap_edges = ce;
    cap_undo = cu;
    if (tree.ensure(ct) != cudaSuccess) {
        release();
        return PAMO_ERR_OOM;
    }
    if (cudaDeviceSynchronize() != cudaSuccess) return PAMO_ERR_DEVICE;
    return ensure_pairs(16 * ct);
}

int Stage2::ensure_pairs(long long n)
{
    if (n <= cap_pairs && pairs) return PAMO_OK;
    if (pairs) cudaFree(pairs);
    pairs = nullptr;
    cap_pairs = 0;
    if (cudaMalloc((void **)&pairs, (size_t)n * sizeof(uint2)) != cudaSuccess) return PAMO_ERR_OOM;
    cap_pairs = n;
    return PAMO_OK;
}

// ---------------------------------------------------------------------------
// one round

#define S2_TRY(expr)                                  \
    do {                                              \
        cudaError_t _e = (expr);                      \
        if (_e != cudaSuccess) return map_cuda_error(_e); \
    } while (0)

// Flags every face of an intersecting pair that has a selected face, then counts
// the considered edges with such a face in their one-rings (n_undo).  The first
// pass of a round selects the one-rings of all the collapses that the undo check
// considers, a later pass only those of the edges the previous check undid: every
// pair that intersected had a face of such a ring, so all of its one-ring was
// selected again, and a pair of two faces outside them is as it was, apart.  (The
// rings of an independent set's collapses are disjoint, so undoing one moves no
// other face; after coincident-endpoint collapses, which may chain, every pass
// selects what the first one did.)  The pass's counters are zero before.
static cudaError_t isect_pass(Stage2 &S, int m, const int *considered, cudaStream_t s)
{
    cudaError_t e;
    S.prof.begin(PH_REFIT, s);
    if ((e = tree_refit(S.tree, S.pts, S.tris, S.active, S.qlist, &S.dcnt->n_query, S.isect, m, s)) != cudaSuccess)
        return e;
    S.prof.begin(PH_QUERY, s);
    if (S.n_slots > 0)
        launch_chained(k_query<true>, grid_for(8LL * m), kQueryThreads, 0, s, S.tree.view(), (const int *)S.qlist, S.dcnt,
               S.pairs, S.cap_pairs, 2, (const int2 *)S.ranges, (const int *)S.vslot);
    else
        launch_chained(k_query<false>, grid_for(8LL * m), kQueryThreads, 0, s, S.tree.view(), (const int *)S.qlist, S.dcnt,
               S.pairs, S.cap_pairs, S.quality ? 4 : 2, (const int2 *)nullptr, (const int *)nullptr);
    S.prof.begin(PH_PAIRS, s);
    const int pair_grid = grid_for(S.cap_pairs < 8LL * m ? S.cap_pairs : 8LL * m);  // about the pairs there are
    if (S.quality)
        launch_chained(k_pairs<true>, pair_grid, kThreads, 0, s, S.pairs, S.dcnt, S.cap_pairs, S.pts, S.tris,
               S.isect, 1e-3f);
    else
        launch_chained(k_pairs<false>, pair_grid, kThreads, 0, s, S.pairs, S.dcnt, S.cap_pairs, S.pts, S.tris,
               S.isect, 1e-3f);
    if (considered) {
        S.prof.begin(PH_UNDO, s);
        launch_chained(k_undo_flags, grid_for(3LL * m), kThreads, 0, s, considered, S.dcnt, (const int2 *)S.edges,
               (const int *)S.first_near, (const int *)S.near_tris, (const uint8_t *)S.isect, S.uflag);
    }
    S.prof.end(s);
    return cudaGetLastError();
}

// The counters, and with them whatever was copied to the host before, once the
// stream is done; a fault that a scan recorded since the last time ends the round.
int Stage2::read_counters(cudaStream_t s)
{
    S2_TRY(cudaMemcpyAsync(hcnt, dcnt, sizeof(RoundCounters), cudaMemcpyDeviceToHost, s));
    S2_TRY(cudaStreamSynchronize(s));
    prof.collect();
    return hcnt->scan_fault ? PAMO_ERR_DEVICE : PAMO_OK;
}

// isect_pass and the counters' copy; once more with a larger pair buffer if the
// candidates did not fit.
static int checked_pass(Stage2 &S, int m, const int *considered, cudaStream_t s)
{
    for (int attempt = 0;; ++attempt) {
        S2_TRY(isect_pass(S, m, considered, s));
        int rc = S.read_counters(s);
        if (rc) return rc;
        if (S.hcnt->pair_overflow == 0) return PAMO_OK;
        if (attempt > 0) return PAMO_ERR_CAPACITY;
        rc = S.ensure_pairs((long long)S.hcnt->n_pairs + S.hcnt->n_pairs / 2 + 1024);
        if (rc) return rc;
        S2_TRY(cudaMemsetAsync(&S.dcnt->n_undo, 0, 5 * sizeof(int), s));  // n_undo to n_hit
    }
}

// positions of the flagged entries of the considered list, in its order (pos: also
// each entry's prefix, which a batch splits by mesh)
static cudaError_t undo_list_of(Stage2 &S, int *pos, cudaStream_t s)
{
    return scan_job(ScanJob{S.uflag, nullptr, pos, S.undo_idx, S.hcnt->n_considered, nullptr, S.scan_scratch,
                            &S.dcnt->n_undo},
                    s, &S.dcnt->scan_fault);
}

// A thread per edge follows a chain of a dozen faces (45 us a pass at least, however
// few the edges); a group of eight lanes follows it in two steps, but spends more
// instructions, as a ring of six leaves two lanes idle and FP64 terms are repeated.
// The first rounds of a torus take, us a pass by threads / by groups,
//   10k 47/25   34k 48/32   63k 54/53   80k 59/67   100k 60/75   200k 112/132   800k 344/485
//   in quality mode  10k 49/30   34k 50/40   43k 54/57   50k 55/63   100k 63/97   800k 457/651
// and later rounds, whose rings are uneven, favour the groups more.  Over whole loops
// the passes add up, by the limit (all by threads, 50k, 64k, 80k, 100k, 130k, all by
// groups), to 23.8, 22.8, 22.7, 22.6, 22.6, 22.7, 29.4 ms for a torus of 2M faces and
// 4.35, 3.73, 3.72, 3.75, 3.77, 3.82, 4.14 for a sphere of 328k; in quality mode (30k,
// 40k, 50k, 64k) to 30.8, 30.8, 30.7, 30.8 and 4.56, 4.53, 4.54, 4.59: flat about the
// limits chosen.  A batch counts its packed faces, which is what fills the device.
template <bool QUALITY>
static void launch_edge_cost(const CostArgs &A, const int *order, int m, int L, const int *first_edge, cudaStream_t s)
{
    if (m <= (QUALITY ? 50000 : 100000))
        launch_chained(k_edge_cost_group<QUALITY>, grid_for(L, kThreads / 32 * kGroupLeaves), kThreads, 0, s, A, order, L,
               first_edge);
    else
        launch_chained(k_edge_cost<QUALITY>, grid_for(L, kChunkFaces), kThreads, 0, s, A, order, L, first_edge);
}

int Stage2::round(int n, int m, float scale, float threshold, bool is_stuck, const int *d_undo_in, int n_undo_in,
                  int *n_undo_out, cudaStream_t s, bool keep_bvh)
{
    int nvu = 0, first = 0;
    if (is_stuck) {
        if (n_undo_in > 0) {
            S2_TRY(cudaMemcpyAsync(tmp_undo, d_undo_in, (size_t)n_undo_in * 4, cudaMemcpyDeviceToDevice, s));
            launch(k_rearrange, grid_for(n_undo_in), kThreads, 0, s, tmp_undo, pts_map, undo_list, 0, n_undo_in);
        }
        nvu += n_undo_in;
        first += n_undo_in;
    } else if (n_undo_in != 0) {
        S2_TRY(cudaMemsetAsync(invalid_table, 0, (size_t)cap_pts + 1, s));
    }
    if (n_undo_in > 0) launch(k_mark_invalid, grid_for(n_undo_in), kThreads, 0, s, d_undo_in, n_undo_in, invalid_table);

    const float tres = threshold, edge_s = scale;
    // host-side conversion as in the reference (cusimp_free.cu:923): the
    // template clamp, then float -> u32 keeping the low 32 bits when out of range
    float ct = (0.0f > threshold) ? 0.0f : threshold;
    ct = (ct < kCostRange) ? ct : kCostRange;
    const uint32_t collapse_t = (uint32_t)(unsigned long long)(ct / kCostRange * 4294967296.0f);

    prof.begin(PH_SETUP, s);
    launch_chained(k_round_init, grid_for((n > m ? n : m) + 1LL), kThreads, 0, s, (const float4 *)opts, (const int4 *)otris, pts,
           tris, occ, first_near, cursor, vmin, first_edge, active, dcnt, n, m);
    launch_chained(k_face_a, grid_for(m), kThreads, 0, s, pts, tris, m, first_near, first_edge, plane, elen4);
    S2_TRY(scan_jobs(ScanJob{first_near, nullptr, first_near, nullptr, n + 1LL, nullptr, scan_scratch, nullptr},
                     ScanJob{first_edge, nullptr, first_edge, nullptr, m + 1LL, nullptr, scan_scratch2, &dcnt->n_edges},
                     s, &dcnt->scan_fault));
    const int *d_n_edges = &dcnt->n_edges;
    launch_chained(k_face_b, grid_for(m), kThreads, 0, s, tris, m, first_near, cursor, near_tris, first_edge, edges);
    launch_chained(k_vertex_quadric, grid_for(8LL * n), kThreads, 0, s, (const int *)first_near, near_tris, (const float4 *)plane,
           (const int4 *)tris, reinterpret_cast<float *>(quad), nxt, n);
    if (quality) {
        int rc = ensure_quality(n, 3LL * m);
        if (rc) return rc;
        launch_chained(k_vertex_quadric64, grid_for(n), kThreads, 0, s, (const int *)first_near, (const int *)near_tris,
               (const float4 *)pts, (const int4 *)tris, quad64, n);
    }
    // The tree only needs an order of the round input's faces: sort them, or keep
    // the previous round's order (leaves renumbered by compact(), removed faces
    // as empty leaves) while at least kRebuildFraction of its leaves are faces.
    // Queries find every overlapping leaf whatever the order, so the pairs found
    // do not depend on this choice; the refit before each query sets the boxes.
    prof.begin(PH_LBVH_BUILD, s);
    if (!(keep_bvh && tree_carried && m <= tree.leaves && (double)m >= kRebuildFraction * (double)tree.leaves))
        S2_TRY(tree_build(tree, pts, tris, m, s));
    tree_carried = false;

    const long long EMAX = 3LL * m;
    prof.begin(PH_EDGE_COST, s);
    CostArgs ca{edges, d_n_edges, pts, tris, first_near, near_tris, nxt, plane, elen4, quad, invalid_table,
                edge_cost, vmin, tres, edge_s, is_stuck ? 1 : 0, nullptr, nullptr, nullptr,
                quality ? (const double *)quad64 : nullptr, quality ? epos : nullptr};
    if (quality)
        launch_edge_cost<true>(ca, tree.vals, m, tree.leaves, first_edge, s);
    else
        launch_edge_cost<false>(ca, tree.vals, m, tree.leaves, first_edge, s);
    CollapseArgs cl{edges, d_n_edges, edge_cost, vmin, first_near, near_tris, opts, otris, pts, tris, occ, eflag,
                    collapse_t, nullptr, nullptr, nullptr, quality ? (const float4 *)epos : nullptr};
    prof.begin(PH_COLLAPSE, s);
    launch_chained(k_collapse, grid_for(EMAX), kThreads, 0, s, cl);
    S2_TRY(scan_job(ScanJob{eflag, nullptr, nullptr, collapsed, EMAX, d_n_edges, scan_scratch, &dcnt->n_main}, s,
                    &dcnt->scan_fault));
    if (quality)
        launch_chained(k_collapse_apply<true>, grid_for(EMAX), kThreads, 0, s, cl, (const int *)collapsed,
               (const int *)&dcnt->n_main, active);
    else
        launch_chained(k_collapse_apply<false>, grid_for(EMAX), kThreads, 0, s, cl, (const int *)collapsed,
               (const int *)&dcnt->n_main, active);
    prof.begin(PH_CLEANUP, s);
    launch_chained(k_cleanup<false>, grid_for(EMAX), kLineThreads, 0, s, tris, m, (const int2 *)edges, d_n_edges, pts, eflag,
           (const int *)first_near, (const int *)near_tris, occ, collapsed, active, dcnt);
    int rc = checked_pass(*this, m, collapsed, s);
    if (rc) return rc;
    last_stats[0] = hcnt->n_edges;
    last_stats[1] = hcnt->n_main;
    last_stats[2] = hcnt->n_total;
    last_stats[5] = hcnt->n_pairs;
    last_stats[6] = m;
    int cnt_undo = hcnt->n_undo;
    nvu += 2 * cnt_undo;
    if (nvu > cap_undo) return PAMO_ERR_CAPACITY;
    int it = 0;
    while (cnt_undo != 0) {
        it++;
        prof.begin(PH_UNDO, s);
        S2_TRY(undo_list_of(*this, nullptr, s));
        const bool reselect = hcnt->n_line == 0;  // see isect_pass
        if (reselect) S2_TRY(cudaMemsetAsync(active, 0, (size_t)m, s));
        launch_chained(k_undo_apply, grid_for(cnt_undo), kThreads, 0, s, (const int *)undo_idx, cnt_undo,
               (const int *)collapsed, (const int2 *)edges, (const int *)first_near, (const int *)near_tris,
               (const float4 *)opts, (const int4 *)otris, pts, tris, occ, reselect ? active : nullptr,
               (const int *)pts_map, undo_list, first, (const SlotInfo *)nullptr, (const SlotCounters *)nullptr,
               (const int *)nullptr, dcnt);
        first += 2 * cnt_undo;
        if ((rc = checked_pass(*this, m, collapsed, s))) return rc;
        cnt_undo = hcnt->n_undo;
        nvu += 2 * cnt_undo;
        if (nvu > cap_undo) return PAMO_ERR_CAPACITY;
        if (it == 5) break;
    }
    last_stats[3] = it;
    last_stats[4] = nvu;
    // pts_map = exclusive scan of occ[0..n]; the faces' positions for compact()
    prof.begin(PH_COMPACT, s);
    S2_TRY(scan_jobs(ScanJob{occ, nullptr, pts_map, nullptr, n + 1LL, nullptr, scan_scratch, nullptr},
                     ScanJob{nullptr, tris, fpos, nullptr, m, nullptr, scan_scratch2, nullptr}, s, &dcnt->scan_fault));
    prof.end(s);
    *n_undo_out = nvu;
    return PAMO_OK;
}

cudaError_t query_and_test_pairs(PackedTree &tree, const float4 *pts, const int4 *tris, int m, int *qlist,
                                 uint2 *pairs, long long cap_pairs, RoundCounters *cnt, uint8_t *isect,
                                 cudaStream_t s)
{
    cudaError_t e = tree_refit(tree, pts, tris, nullptr, qlist, &cnt->n_query, isect, m, s);
    if (e != cudaSuccess) return e;
    launch_chained(k_query<false>, grid_for(8LL * m), kQueryThreads, 0, s, tree.view(), (const int *)qlist, cnt, pairs,
           cap_pairs, 2, (const int2 *)nullptr, (const int *)nullptr);
    launch_chained(k_pairs<false>, grid_for(cap_pairs), kThreads, 0, s, pairs, cnt, cap_pairs, pts, tris, isect, 1e-3f);
    return cudaGetLastError();
}

int Stage2::ensure_quality(long long n_pts, long long n_edges)
{
    if (n_pts > cap_q64 || !quad64) {
        if (quad64) cudaFree(quad64);
        quad64 = nullptr;
        cap_q64 = 0;
        const long long c = n_pts > cap_pts ? n_pts : cap_pts;
        if (cudaMalloc((void **)&quad64, (size_t)(c + 1) * 10 * sizeof(double)) != cudaSuccess) return PAMO_ERR_OOM;
        cap_q64 = c;
    }
    if (n_edges > cap_epos || !epos) {
        if (epos) cudaFree(epos);
        epos = nullptr;
        cap_epos = 0;
        const long long c = n_edges > cap_edges ? n_edges : cap_edges;
        if (cudaMalloc((void **)&epos, (size_t)(c + 1) * sizeof(float4)) != cudaSuccess) return PAMO_ERR_OOM;
        cap_epos = c;
    }
    return PAMO_OK;
}

int Stage2::self_intersect_all(int n, int m, cudaStream_t s)
{
    tree_carried = false;
    // faces of opts/otris; every live face queries the tree
    launch_chained(k_round_init, grid_for((n > m ? n : m) + 1LL), kThreads, 0, s, (const float4 *)opts, (const int4 *)otris, pts,
           tris, occ, first_near, cursor, vmin, first_edge, active, dcnt, n, m);
    S2_TRY(cudaMemsetAsync(active, 1, (size_t)m, s));
    S2_TRY(tree_build(tree, pts, tris, m, s));
    return checked_pass(*this, m, nullptr, s);
}

int Stage2::compact(int n, int m, cudaStream_t s)
{
    prof.begin(PH_COMPACT, s);
    const bool keep = tree.leaves > 0 && tree.leaves >= m;
    launch_chained(k_compact, grid_for(n > m ? n : m), kThreads, 0, s, (const float4 *)pts, (const int *)occ,
           (const int *)pts_map, n, (const int4 *)tris, (const int *)fpos, m, opts, otris, tree.vals,
           keep ? tree.leaves : 0, dcnt);
    tree_carried = keep;
    prof.end(s);
    return read_counters(s);
}

}  // namespace pamo

// ---------------------------------------------------------------------------
// batch rounds

namespace pamo {

int Stage2::ensure_batch(int K)
{
    if (K <= cap_slots && slots) return PAMO_OK;
    if (cap_pts <= 0 || cap_tris <= 0) return PAMO_ERR_INVALID_ARG;  // ensure() first
    if (slots) cudaFree(slots);
    if (scnt) cudaFree(scnt);
    if (ranges) cudaFree(ranges);
    if (ranges_next) cudaFree(ranges_next);
    if (hslots) cudaFreeHost(hslots);
    if (hscnt) cudaFreeHost(hscnt);
    slots = nullptr; scnt = nullptr; ranges = ranges_next = nullptr; hslots = nullptr; hscnt = nullptr;
    cap_slots = 0;
    int c = K > 16 ? K : 16;
    if (cudaMalloc((void **)&slots, (size_t)c * sizeof(SlotInfo)) != cudaSuccess ||
        cudaMalloc((void **)&scnt, (size_t)c * sizeof(SlotCounters)) != cudaSuccess ||
        cudaMalloc((void **)&ranges, (size_t)c * sizeof(int2)) != cudaSuccess ||
        cudaMalloc((void **)&ranges_next, (size_t)c * sizeof(int2)) != cudaSuccess ||
        cudaMallocHost((void **)&hslots, (size_t)c * sizeof(SlotInfo)) != cudaSuccess ||
        cudaMallocHost((void **)&hscnt, (size_t)c * sizeof(SlotCounters)) != cudaSuccess)
        return PAMO_ERR_OOM;
    if (!vslot && cudaMalloc((void **)&vslot, (size_t)(cap_pts + 1) * 4) != cudaSuccess) return PAMO_ERR_OOM;
    if (!gmap && cudaMalloc((void **)&gmap, (size_t)(cap_pts + 1) * 4) != cudaSuccess) return PAMO_ERR_OOM;
    if (!line_list && cudaMalloc((void **)&line_list, (size_t)(cap_edges + 1) * 4) != cudaSuccess) return PAMO_ERR_OOM;
    if (!cand && cudaMalloc((void **)&cand, (size_t)(cap_edges + 1) * 4) != cudaSuccess) return PAMO_ERR_OOM;
    cap_slots = c;
    return PAMO_OK;
}

static dim3 slot_grid(int K, long long per_slot_max)
{
    long long x = (per_slot_max + kThreads - 1) / kThreads;
    x = x < 1 ? 1 : (x > 64 ? 64 : x);
    return dim3((unsigned)x, (unsigned)K);
}

int Stage2::round_batch(int n, int m, int K, int *nvu_out, cudaStream_t s)
{
    if (K <= 0 || K > cap_slots) return PAMO_ERR_INVALID_ARG;
    n_slots = K;
    std::vector<int> nvu(K), first(K), cnt_undo(K);
    long long max_n = 0, max_undo_in = 0, max_cap_v = 0;
    for (int r = 0; r < K; ++r) {
        SlotInfo &h = hslots[r];
        nvu[r] = first[r] = h.is_stuck ? h.n_undo_in : 0;
        h.pass_first = 0;
        h.nvu = 0;
        max_n = h.n > max_n ? h.n : max_n;
        max_undo_in = h.n_undo_in > max_undo_in ? h.n_undo_in : max_undo_in;
        max_cap_v = h.cap_v > max_cap_v ? h.cap_v : max_cap_v;
    }
    S2_TRY(cudaMemsetAsync(scnt, 0, (size_t)K * sizeof(SlotCounters), s));
    S2_TRY(cudaMemcpyAsync(slots, hslots, (size_t)K * sizeof(SlotInfo), cudaMemcpyHostToDevice, s));
    launch_chained(k_b_pre_copy, slot_grid(K, max_undo_in > max_cap_v ? max_undo_in : max_cap_v), kThreads, 0, s,
           (const SlotInfo *)slots);
    launch_chained(k_b_pre_mark, slot_grid(K, max_undo_in), kThreads, 0, s, (const SlotInfo *)slots);
    launch_chained(k_b_vslot, slot_grid(K, max_n), kThreads, 0, s, (const SlotInfo *)slots, vslot);

    prof.begin(PH_SETUP, s);
    launch_chained(k_round_init, grid_for((n > m ? n : m) + 1LL), kThreads, 0, s, (const float4 *)opts, (const int4 *)otris, pts,
           tris, occ, first_near, cursor, vmin, first_edge, active, dcnt, n, m);
    launch_chained(k_face_a, grid_for(m), kThreads, 0, s, pts, tris, m, first_near, first_edge, plane, elen4);
    S2_TRY(scan_jobs(ScanJob{first_near, nullptr, first_near, nullptr, n + 1LL, nullptr, scan_scratch, nullptr},
                     ScanJob{first_edge, nullptr, first_edge, nullptr, m + 1LL, nullptr, scan_scratch2, &dcnt->n_edges},
                     s, &dcnt->scan_fault));
    const int *d_n_edges = &dcnt->n_edges;
    launch_chained(k_face_b, grid_for(m), kThreads, 0, s, tris, m, first_near, cursor, near_tris, first_edge, edges);
    launch_chained(k_vertex_quadric, grid_for(8LL * n), kThreads, 0, s, (const int *)first_near, near_tris, (const float4 *)plane,
           (const int4 *)tris, reinterpret_cast<float *>(quad), nxt, n);
    launch_chained(k_b_edge_off, grid_for(K), kThreads, 0, s, (const SlotInfo *)slots, (const int *)first_edge, scnt, K);
    prof.begin(PH_LBVH_BUILD, s);
    // the previous round's order while it holds (each mesh's run of leaves stays where
    // it was): sorting every round was a fifth of a batch of 32 meshes
    if (!(tree_carried && m <= tree.leaves && (double)m >= kRebuildFraction * (double)tree.leaves))
        S2_TRY(tree_build(tree, pts, tris, m, s, vslot, K, ranges));
    tree_carried = false;

    const long long EMAX = 3LL * m;
    prof.begin(PH_EDGE_COST, s);
    CostArgs ca{edges, d_n_edges, pts, tris, first_near, near_tris, nxt, plane, elen4, quad, nullptr,
                nullptr, vmin, 0.f, 1.f, 0, slots, scnt, vslot, nullptr, nullptr};
    launch_edge_cost<false>(ca, tree.vals, m, tree.leaves, first_edge, s);
    CollapseArgs cl{edges, d_n_edges, nullptr, vmin, first_near, near_tris, opts, otris, pts, tris, occ, eflag,
                    0u, slots, scnt, vslot, nullptr};
    prof.begin(PH_COLLAPSE, s);
    launch_chained(k_collapse, grid_for(EMAX), kThreads, 0, s, cl);
    S2_TRY(scan_job(ScanJob{eflag, nullptr, uflag, collapsed, EMAX, d_n_edges, scan_scratch, &dcnt->n_main}, s,
                    &dcnt->scan_fault));
    launch_chained(k_collapse_apply<false>, grid_for(EMAX), kThreads, 0, s, cl, (const int *)collapsed,
           (const int *)&dcnt->n_main, active);
    launch_chained(k_b_main, grid_for(K), kThreads, 0, s, (const int *)uflag, (const RoundCounters *)dcnt, scnt, K);
    prof.begin(PH_CLEANUP, s);
    launch_chained(k_cleanup<true>, grid_for(EMAX), kLineThreads, 0, s, tris, m, (const int2 *)edges, d_n_edges, pts, eflag,
           (const int *)first_near, (const int *)near_tris, occ, collapsed, active, dcnt);
    launch_chained(k_b_line_apply, 1, kLineThreads, 0, s, edges, d_n_edges, eflag, first_near, near_tris, pts, tris, occ,
           line_list, (const int *)vslot, dcnt, scnt, K);
    launch_chained(k_b_cand_fill, grid_for(EMAX), kThreads, 0, s, (const int *)collapsed, (const int *)line_list, edges,
           (const int *)vslot, (const RoundCounters *)dcnt, (const SlotCounters *)scnt, cand, (const int *)first_near,
           (const int *)near_tris, active);
    // a check, and where it finds edges to undo their list and each mesh's share of it
    auto pass = [&]() -> int {
        int rc = checked_pass(*this, m, cand, s);
        if (rc) return rc;
        for (int r = 0; r < K; ++r) hscnt[r].n_undo = 0;
        if (hcnt->n_undo == 0) return PAMO_OK;
        S2_TRY(undo_list_of(*this, eflag, s));
        launch_chained(k_b_undo_counts, grid_for(K), kThreads, 0, s, (const int *)eflag, (const RoundCounters *)dcnt, scnt, K);
        S2_TRY(cudaMemcpyAsync(hscnt, scnt, (size_t)K * sizeof(SlotCounters), cudaMemcpyDeviceToHost, s));
        S2_TRY(cudaStreamSynchronize(s));
        return PAMO_OK;
    };
    int rc = pass();
    if (rc) return rc;
    last_stats[0] = hcnt->n_edges;
    last_stats[1] = hcnt->n_main;
    last_stats[2] = hcnt->n_total;
    last_stats[5] = hcnt->n_pairs;
    last_stats[6] = m;
    bool any = false;
    for (int r = 0; r < K; ++r) {
        cnt_undo[r] = hscnt[r].n_undo;
        nvu[r] += 2 * cnt_undo[r];
        if (nvu[r] > hslots[r].cap_undo) return PAMO_ERR_CAPACITY;
        any = any || cnt_undo[r] != 0;
    }
    int it = 0;
    while (any) {
        it++;
        prof.begin(PH_UNDO, s);
        for (int r = 0; r < K; ++r) {
            hslots[r].pass_first = first[r];
            first[r] += 2 * cnt_undo[r];
        }
        S2_TRY(cudaMemcpyAsync(slots, hslots, (size_t)K * sizeof(SlotInfo), cudaMemcpyHostToDevice, s));
        const bool reselect = hcnt->n_line == 0;  // as in the single-mesh round
        if (reselect) S2_TRY(cudaMemsetAsync(active, 0, (size_t)m, s));
        launch_chained(k_undo_apply, grid_for(hcnt->n_undo), kThreads, 0, s, (const int *)undo_idx, hcnt->n_undo,
               (const int *)cand, (const int2 *)edges, (const int *)first_near, (const int *)near_tris,
               (const float4 *)opts, (const int4 *)otris, pts, tris, occ, reselect ? active : nullptr,
               (const int *)nullptr, (int *)nullptr, 0, (const SlotInfo *)slots, (const SlotCounters *)scnt,
               (const int *)vslot, dcnt);
        rc = pass();
        if (rc) return rc;
        any = false;
        for (int r = 0; r < K; ++r) {
            cnt_undo[r] = hscnt[r].n_undo;
            nvu[r] += 2 * cnt_undo[r];
            if (nvu[r] > hslots[r].cap_undo) return PAMO_ERR_CAPACITY;
            any = any || cnt_undo[r] != 0;
        }
        if (it == 5) break;
    }
    last_stats[3] = it;
    // the packed vertex map, each mesh's own map and undo-list copy
    prof.begin(PH_COMPACT, s);
    S2_TRY(scan_jobs(ScanJob{occ, nullptr, gmap, nullptr, n + 1LL, nullptr, scan_scratch, nullptr},
                     ScanJob{nullptr, tris, fpos, nullptr, m, nullptr, scan_scratch2, fpos + m}, s, &dcnt->scan_fault));
    long long max_nvu = 0;
    for (int r = 0; r < K; ++r) {
        hslots[r].nvu = nvu[r];
        max_nvu = nvu[r] > max_nvu ? nvu[r] : max_nvu;
        nvu_out[r] = nvu[r];
    }
    S2_TRY(cudaMemcpyAsync(slots, hslots, (size_t)K * sizeof(SlotInfo), cudaMemcpyHostToDevice, s));
    launch_chained(k_b_local_map, slot_grid(K, (max_n + 1 > max_nvu ? max_n + 1 : max_nvu)), kThreads, 0, s,
           (const SlotInfo *)slots, (const int *)gmap);
    prof.end(s);
    return PAMO_OK;
}

int Stage2::compact_batch(int n, int m, int K, cudaStream_t s)
{
    prof.begin(PH_COMPACT, s);
    launch_chained(k_compact, grid_for(n > m ? n : m), kThreads, 0, s, (const float4 *)pts, (const int *)occ,
                   (const int *)gmap, n, (const int4 *)tris, (const int *)fpos, m, opts, otris, tree.vals, tree.leaves,
                   dcnt);
    tree_carried = true;  // until a mesh is admitted; the caller renumbers what it moves
    launch_chained(k_b_next, grid_for(K), kThreads, 0, s, (const SlotInfo *)slots, (const int *)gmap, (const int *)fpos, scnt,
           K);
    prof.end(s);
    S2_TRY(cudaMemcpyAsync(hscnt, scnt, (size_t)K * sizeof(SlotCounters), cudaMemcpyDeviceToHost, s));
    return read_counters(s);
}

}  // namespace pamo
