// Stage 1 of PaMO.run: remeshing (simp_cuda/pamo/__init__.py:60-120,130-142).
//
// The reference normalises the triangles into the unit cube, asks
// torchcumesh2sdf for a narrow-band signed distance field on an R^3 grid,
// shifts it by -0.9/R, extracts quads with pdmc's dual marching cubes and
// splits each quad into the triangle pair with the larger smallest angle.  Both
// libraries are absent, so this file restates their published steps; the CPU
// oracle/s1_oracle.py defines the same semantics and the results agree bit
// for bit (tests/test_stage1_gpu.py):
//
//   1. normalise: ((p - tris_mean) - tris_min) / tris_max + band) / margin in
//      float32, as preprocess_mesh does with numpy (:60-72);
//   2. unsigned distance (double) from every grid sample ((i + 0.5) / R, ...)
//      within `band` of a triangle to the nearest triangle, else `band`: one
//      warp per triangle walks the samples of its box grown by two voxels and
//      lowers the sample's squared distance with a 64-bit atomic minimum (the
//      bits of a non-negative double order like the value).  Two voxels of the
//      band's three give the same result where the triangles have areas: see kReach;
//   3. sign by flood fill: samples farther than half a voxel from every
//      triangle are free, free samples 6-connected to the grid boundary are
//      outside; the field is +-distance - 0.9/R.  From here on the grid is bits,
//      a word per 32 samples of a row: which samples are free, outside, inside
//      (negative).  Tiles of 8 x 8 rows propagate "outside" in shared memory until
//      they settle, and launches repeat until no word changes (bounded);
//   4. dual marching cubes: a sample is inside where the field is negative.
//      Per cell, the crossed edges pair up on each cube face (an ambiguous face
//      cuts off each outside corner, a rule both cells sharing the face agree
//      on), the pairings split them into cycles, and each cycle (patch) gets
//      one vertex at the mean of its edges' crossing points.  Every crossed
//      grid edge gives one quad through its four cells' patch vertices, wound
//      with the normal towards the outside.  Vertices are numbered by cell and
//      patch, quads by axis and lower sample, through prefix scans over the
//      words' counts; a place within a word is a population count.  Distances
//      (their square roots) are only taken at crossed edges;
//   5. each quad is split into (0,1,3),(1,2,3) or (0,1,2),(0,2,3), whichever
//      has the smaller largest corner cosine (double), first-kind quads first
//      (:95-118); vertices are mapped back to the centred frame in double and
//      rounded to float32.
//
// The output is in the frame centred on tris_mean, as the reference's remesh
// returns it; stage 2 then runs without centring again and adds tris_mean
// back at the end (:130-189).
#include <cstring>
#include <vector>

#include "scan.cuh"
#include "stage1.cuh"

namespace pamo {
namespace s1 {
namespace {

// cube corners c = x + 2 y + 4 z; edges 0-3 along x, 4-7 along y, 8-11 along z
constexpr int kEdgeCorners[12][2] = {{0, 1}, {2, 3}, {4, 5}, {6, 7}, {0, 2}, {1, 3},
                                     {4, 6}, {5, 7}, {0, 4}, {1, 5}, {2, 6}, {3, 7}};
// the faces as corner cycles
constexpr int kFaceCorners[6][4] = {{0, 2, 6, 4}, {1, 3, 7, 5}, {0, 1, 5, 4}, {2, 3, 7, 6}, {0, 1, 3, 2}, {4, 5, 7, 6}};

__constant__ signed char c_patch[256][12];  // patch of each edge per sign case, -1: not crossed
__constant__ unsigned char c_npatch[256];

int edge_of(int a, int b)
{
    for (int i = 0; i < 12; ++i)
        if ((kEdgeCorners[i][0] == a && kEdgeCorners[i][1] == b) || (kEdgeCorners[i][0] == b && kEdgeCorners[i][1] == a))
            return i;
    return -1;
}

// The patch table: for each sign case (bit c set: corner c inside), the crossed
// edges linked by their pairings on the cube faces, split into cycles.
void build_patch_table(signed char (*patch)[12], unsigned char *npatch)
{
    for (int cs = 0; cs < 256; ++cs) {
        bool inside[8], crossed[12];
        for (int c = 0; c < 8; ++c) inside[c] = (cs >> c) & 1;
        for (int e = 0; e < 12; ++e) crossed[e] = inside[kEdgeCorners[e][0]] != inside[kEdgeCorners[e][1]];
        int link[12][2], nl[12] = {0};
        auto join = [&](int a, int b) {
            link[a][nl[a]++] = b;
            link[b][nl[b]++] = a;
        };
        for (int f = 0; f < 6; ++f) {
            int es[4], cr[4], n = 0;
            for (int k = 0; k < 4; ++k) {
                es[k] = edge_of(kFaceCorners[f][k], kFaceCorners[f][(k + 1) % 4]);
                if (crossed[es[k]]) cr[n++] = es[k];
            }
            if (n == 2) {
                join(cr[0], cr[1]);
            } else if (n == 4) {  // cut off each outside corner
                for (int k = 0; k < 4; ++k)
                    if (!inside[kFaceCorners[f][k]]) join(es[(k + 3) % 4], es[k]);
            }
        }
        int pid[12];
        for (int e = 0; e < 12; ++e) pid[e] = -1;
        int np = 0;
        for (int e = 0; e < 12; ++e) {
            if (!crossed[e] || pid[e] >= 0) continue;
            int stack[12], sp = 0;
            stack[sp++] = e;
            pid[e] = np;
            while (sp) {
                const int x = stack[--sp];
                for (int k = 0; k < nl[x]; ++k) {
                    const int y = link[x][k];
                    if (pid[y] < 0) {
                        pid[y] = np;
                        stack[sp++] = y;
                    }
                }
            }
            ++np;
        }
        for (int e = 0; e < 12; ++e) patch[cs][e] = (signed char)pid[e];
        npatch[cs] = (unsigned char)np;
    }
}

__device__ __forceinline__ long long gidx(int x, int y, int z, int R) { return ((long long)z * R + y) * R + x; }

// the corners of cube edge e (the order of kEdgeCorners)
__device__ __forceinline__ void edge_corners(int e, int &a, int &b)
{
    if (e < 4) {
        a = 2 * e;
        b = a + 1;
    } else if (e < 8) {
        const int k = e - 4;
        a = (k & 1) | ((k >> 1) << 2);
        b = a + 2;
    } else {
        a = e - 8;
        b = a + 4;
    }
}

// -------------------------------------------------------------- 1. normalise
// per-axis minimum of the centred corners (ordered ints), then the largest
// coordinate after subtracting it
__global__ void k_s1_min(const float *pts, const int *tris, int m, const float *mean, int *dev)
{
    float lo[3] = {INFINITY, INFINITY, INFINITY};
    PAMO_GRID_STRIDE(f, m)
    {
        for (int c = 0; c < 3; ++c) {
            const int v = tris[3 * f + c];
            for (int k = 0; k < 3; ++k) lo[k] = fminf(lo[k], pts[3 * v + k] - mean[k]);
        }
    }
    for (int k = 0; k < 3; ++k) {
        float x = lo[k];
        for (int o = 16; o > 0; o >>= 1) x = fminf(x, __shfl_down_sync(0xffffffffu, x, o));
        if ((threadIdx.x & 31) == 0) atomicMin(&dev[k], float_to_ordered(x));
    }
}

__global__ void k_s1_max(const float *pts, const int *tris, int m, const float *mean, int *dev)
{
    float lo[3];
    for (int k = 0; k < 3; ++k) lo[k] = ordered_to_float(dev[k]);
    float hi = -INFINITY;
    PAMO_GRID_STRIDE(f, m)
    {
        for (int c = 0; c < 3; ++c) {
            const int v = tris[3 * f + c];
            for (int k = 0; k < 3; ++k) hi = fmaxf(hi, (pts[3 * v + k] - mean[k]) - lo[k]);
        }
    }
    for (int o = 16; o > 0; o >>= 1) hi = fmaxf(hi, __shfl_down_sync(0xffffffffu, hi, o));
    if ((threadIdx.x & 31) == 0) atomicMax(&dev[3], float_to_ordered(hi));
}

struct D3 {
    double x, y, z;
};
__device__ __forceinline__ D3 dsub(D3 a, D3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ double ddot(D3 a, D3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

// Whether point_tri_d2 gives the triangle's distances to 0.03 voxels at every sample
// within the band (all that kReach needs).  Its barycentric terms are differences of
// products of the size |ab| |ac| D^2, D <= L + 3 sqrt(3) / R being a sample's distance
// from a corner and L the longest edge; some 160 roundings of 1.1e-16 of that size,
// over the squared normal and times L, bound the closest point's error (here with a
// factor of two, squared, and D^2 <= 2 (L^2 + 27 / R^2)).  A triangle without an area
// gives NaN on one side of its line, a single point its distance.
__device__ __forceinline__ bool distances_hold(const float *T, int R)
{
    const D3 a = {T[0], T[1], T[2]}, b = {T[3], T[4], T[5]}, c = {T[6], T[7], T[8]};
    const D3 ab = dsub(b, a), ac = dsub(c, a), bc = dsub(c, b);
    const D3 n = {ab.y * ac.z - ab.z * ac.y, ab.z * ac.x - ab.x * ac.z, ab.x * ac.y - ab.y * ac.x};
    const double ab2 = ddot(ab, ab), ac2 = ddot(ac, ac), l2 = fmax(fmax(ab2, ac2), ddot(bc, bc)), nn = ddot(n, n);
    const double k = 4e-14 * R / 0.03, d2 = l2 + 27.0 / ((double)R * R);
    return (nn > 0.0 && 4.0 * k * k * ab2 * ac2 * l2 * d2 * d2 <= nn * nn) || l2 == 0.0;
}

// the triangles in the unit cube; dev[5]: one of them has distances that do not hold
__global__ void k_s1_normalise(const float *pts, const int *tris, int m, const float *mean, int *dev,
                               float band, float margin, int R, float *out)
{
    float lo[3];
    for (int k = 0; k < 3; ++k) lo[k] = ordered_to_float(dev[k]);
    const float mx = ordered_to_float(dev[3]);
    PAMO_GRID_STRIDE(f, m)
    {
        float T[9];
        for (int c = 0; c < 3; ++c) {
            const int v = tris[3 * f + c];
            for (int k = 0; k < 3; ++k) {
                T[3 * c + k] = (((pts[3 * v + k] - mean[k]) - lo[k]) / mx + band) / margin;
                out[9 * f + 3 * c + k] = T[3 * c + k];
            }
        }
        if (!distances_hold(T, R)) dev[5] = 1;
    }
}

// ------------------------------------------------------- 2. unsigned distance

// squared distance from p to triangle abc; the closest point by the Voronoi
// regions of the triangle (Ericson, Real-Time Collision Detection, 5.1.5), with
// the operation order of oracle/s1_oracle.py _point_tri_d2
__device__ double point_tri_d2(D3 p, D3 a, D3 b, D3 c)
{
    const D3 ab = dsub(b, a), ac = dsub(c, a), ap = dsub(p, a);
    const double d1 = ddot(ab, ap), d2 = ddot(ac, ap);
    const D3 bp = dsub(p, b);
    const double d3 = ddot(ab, bp), d4 = ddot(ac, bp);
    const D3 cp = dsub(p, c);
    const double d5 = ddot(ab, cp), d6 = ddot(ac, cp);
    const double vc = d1 * d4 - d3 * d2;
    const double vb = d5 * d2 - d1 * d6;
    const double va = d3 * d6 - d5 * d4;
    D3 q;
    if (d1 <= 0 && d2 <= 0) {
        q = a;
    } else if (d3 >= 0 && d4 <= d3) {
        q = b;
    } else if (vc <= 0 && d1 >= 0 && d3 <= 0) {
        const double v = d1 / (d1 - d3);
        q = {a.x + v * ab.x, a.y + v * ab.y, a.z + v * ab.z};
    } else if (d6 >= 0 && d5 <= d6) {
        q = c;
    } else if (vb <= 0 && d2 >= 0 && d6 <= 0) {
        const double w = d2 / (d2 - d6);
        q = {a.x + w * ac.x, a.y + w * ac.y, a.z + w * ac.z};
    } else if (va <= 0 && (d4 - d3) >= 0 && (d5 - d6) >= 0) {
        const double w = (d4 - d3) / ((d4 - d3) + (d5 - d6));
        const D3 cb = dsub(c, b);
        q = {b.x + w * cb.x, b.y + w * cb.y, b.z + w * cb.z};
    } else {
        const double den = 1.0 / (va + vb + vc);
        const double v = vb * den, w = vc * den;
        q = {a.x + v * ab.x + w * ac.x, a.y + v * ab.y + w * ac.y, a.z + v * ab.z + w * ac.z};
    }
    const D3 d = dsub(p, q);
    return ddot(d, d);
}

// How far from a triangle a sample's distance matters, in voxels.  The distance is
// used where an edge is crossed: between an inside sample A (negative) and a
// neighbour B outside at 0.9 voxels or more.  A is outside within 0.9 voxels, or
// near (within 0.5), or free but not reached -- which no neighbour of an outside
// sample is.  Distances of neighbours differ by at most a voxel, so B's is below
// 1.9, and both ends lie within 2.  Any value of 2 or more in a farther sample
// gives the same bits: free, and not within 0.9.  That neighbours differ by a voxel
// holds for distances, so for computed ones where they are distances: a triangle
// without an area gives none on one side (NaN, dropped by the minimum), and one such
// triangle takes the whole mesh back to the band (distances_hold).  Against 3 voxels a
// small triangle's box has a third of the samples: 2.7 -> 1.6 ms for 500,000 faces
// at R = 256, 8.8 -> 4.9 ms for 2,000,000.
constexpr double kReach = 2.0;

// One warp per triangle over the samples of its box grown by `reach`.  Before
// the full closest-point computation a sample is skipped when a lower bound of
// its distance to the triangle -- the distance to the triangle's bounding box,
// and to its plane -- already reaches the sample's current value (the bounds
// hold in exact arithmetic; the 1e-9 relative margin covers their rounding), so
// the minimum, and therefore the field, is the same as without the test.
// (i + 0.5) / R, the coordinate of sample i; for R a power of two (inv_r > 0)
// the product with 1 / R is that same number and spares the FP64 division
__device__ __forceinline__ double s1_coord(int i, int R, double inv_r)
{
    return inv_r > 0.0 ? (i + 0.5) * inv_r : (i + 0.5) / R;
}

__global__ void __launch_bounds__(256, 3) k_s1_udist(const float *tris, int m, int R, double inv_r, double band,
                                                  const int *dev, unsigned long long *field)
{
    const double reach = dev[5] ? band : kReach / R;
    const int lane = threadIdx.x & 31;
    const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    const double reach2 = reach * reach;
    for (long long t = warp0; t < m; t += nw) {
        const float *T = tris + 9 * t;
        const D3 a = {T[0], T[1], T[2]}, b = {T[3], T[4], T[5]}, c = {T[6], T[7], T[8]};
        int lo[3], n[3];
        const double mn[3] = {fmin(a.x, fmin(b.x, c.x)), fmin(a.y, fmin(b.y, c.y)), fmin(a.z, fmin(b.z, c.z))};
        const double mx[3] = {fmax(a.x, fmax(b.x, c.x)), fmax(a.y, fmax(b.y, c.y)), fmax(a.z, fmax(b.z, c.z))};
        for (int k = 0; k < 3; ++k) {
            // samples (i + 0.5) / R within [mn - reach, mx + reach]
            int l = (int)floor((mn[k] - reach) * R - 0.5), h = (int)ceil((mx[k] + reach) * R - 0.5);
            l = max(l, 0);
            h = min(h, R - 1);
            lo[k] = l;
            n[k] = h >= l ? h - l + 1 : 0;
        }
        // the plane's normal (unnormalised) and 1 / |n|^2
        const D3 ab = dsub(b, a), ac = dsub(c, a);
        const D3 nrm = {ab.y * ac.z - ab.z * ac.y, ab.z * ac.x - ab.x * ac.z, ab.x * ac.y - ab.y * ac.x};
        const double nn = ddot(nrm, nrm);
        const double inv_nn = nn > 0.0 ? 1.0 / nn : 0.0;  // degenerate: no plane bound
        const int nxy = n[0] * n[1];
        const int total = nxy * n[2];
        // the lane's sample (ox, oy, oz) in the box, stepped by 32 without divisions
        int ox = 0, oy = 0, oz = 0;
        if (total > 0) {
            ox = lane % n[0];
            oy = (lane / n[0]) % n[1];
            oz = lane / nxy;
        }
        const int qx = total > 0 ? 32 / n[0] : 0, rx = total > 0 ? 32 % n[0] : 0;
        for (int s = lane; s < total; s += 32) {
            const int ix = lo[0] + ox, iy = lo[1] + oy, iz = lo[2] + oz;
            ox += rx;
            oy += qx;
            if (ox >= n[0]) {
                ox -= n[0];
                ++oy;
            }
            while (oy >= n[1]) {
                oy -= n[1];
                ++oz;
            }
            const D3 p = {s1_coord(ix, R, inv_r), s1_coord(iy, R, inv_r), s1_coord(iz, R, inv_r)};
            const double bx = fmax(fmax(mn[0] - p.x, 0.0), p.x - mx[0]);
            const double by = fmax(fmax(mn[1] - p.y, 0.0), p.y - mx[1]);
            const double bz = fmax(fmax(mn[2] - p.z, 0.0), p.z - mx[2]);
            const double box2 = bx * bx + by * by + bz * bz;
            if (box2 >= reach2 * (1.0 + 1e-9)) continue;  // the value stays reach^2 or more
            unsigned long long *dst = field + gidx(ix, iy, iz, R);
            const double cur = __longlong_as_double((long long)*dst);
            if (box2 > cur * (1.0 + 1e-9)) continue;
            const double hp = ddot(nrm, dsub(p, a));
            if (hp * hp * inv_nn > cur * (1.0 + 1e-9)) continue;
            const double d2 = point_tri_d2(p, a, b, c);
            const unsigned long long bits = (unsigned long long)__double_as_longlong(d2);
            if (bits < *dst) atomicMin(dst, bits);
        }
    }
}

__global__ void k_s1_fill(unsigned long long *a, long long n, unsigned long long v)
{
    PAMO_GRID_STRIDE(i, n) a[i] = v;
}

// ------------------------------------------------------------ the grid as bits
// Word w of row (y, z) holds samples 32 w .. 32 w + 31 of the row.
struct Bits {
    int R, W;  // samples and words per row
    uint32_t *free_, *low, *out, *in;  // free; distance - 0.9/R negative; outside; inside
};

__device__ __forceinline__ long long row_word(const Bits &B, int y, int z) { return ((long long)z * B.R + y) * B.W; }

// the row's samples that exist in word w
__device__ __forceinline__ uint32_t valid_bits(int n, int w)
{
    const int left = n - 32 * w;
    return left >= 32 ? 0xFFFFFFFFu : left <= 0 ? 0u : (1u << left) - 1u;
}

// Free and within-0.9 bits from the squared distances, and the flood's start: the
// free samples on the grid's boundary.  Most samples hold the fill value, whose
// bits are known, so few take a square root.
__global__ void __launch_bounds__(kThreads) k_s1_bits(const unsigned long long *__restrict__ field, Bits B,
                                                      unsigned long long fill)
{
    constexpr int kBatch = 4;  // words a warp has in flight
    const int R = B.R, lane = threadIdx.x & 31;
    const long long words = (long long)R * R * B.W;
    const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long q = (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kBatch; q < words;
         q += warps * kBatch) {
        unsigned long long v[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            const long long row = (q + k) / B.W;
            const int x = (int)((q + k) % B.W) * 32 + lane;
            v[k] = q + k < words && x < R ? field[row * R + x] : fill;
        }
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            if (q + k >= words) break;
            const long long row = (q + k) / B.W;
            const int w = (int)((q + k) % B.W), x = w * 32 + lane;
            bool fr = true, lo = false;
            if (v[k] != fill) {
                const double ud = sqrt(__longlong_as_double((long long)v[k]));
                fr = ud > 0.5 / R;
                lo = ud - 0.9 / R < 0.0;
            }
            const uint32_t f = __ballot_sync(0xffffffffu, fr && x < R), l = __ballot_sync(0xffffffffu, lo && x < R);
            if (lane == 0) {
                const int y = (int)(row % R), z = (int)(row / R);
                uint32_t border = 0;
                if (y == 0 || z == 0 || y == R - 1 || z == R - 1) border = 0xFFFFFFFFu;
                if (w == 0) border |= 1u;
                if (w == (R - 1) >> 5) border |= 1u << ((R - 1) & 31);
                B.free_[q + k] = f;
                B.low[q + k] = l;
                B.out[q + k] = f & border;
            }
        }
    }
}

// ----------------------------------------------------------- 3. flood fill
constexpr int kTile = 8;
constexpr int kMaxWords = 32;  // R <= 1024

// the bits of o spread along the runs of f they lie in
__device__ __forceinline__ uint32_t spread(uint32_t o, uint32_t f)
{
    uint32_t up = f, down = f;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
        o |= (up & (o << k)) | (down & (o >> k));
        up &= up << k;
        down &= down >> k;
    }
    return o;
}

// One block per tile of 8 x 8 whole rows: free samples next to an outside sample
// become outside, repeated in shared memory until the tile settles (each sweep
// but the last adds a bit, so it does); a change is reported in dev[4].  Only
// tiles marked in `dirty_in` (changed, or next to a tile that changed, in the
// previous launch; all tiles in the first) do the work; a tile that changes marks
// itself and its four neighbours in `dirty_out`.  Rows start outside at both
// ends, so a few launches settle the grid.  With a byte per sample in 8^3 tiles a
// launch took 66 us at R = 256; this one takes 6 to 22, 12 on average.
__global__ void __launch_bounds__(kThreads) k_s1_flood(Bits B, int *dev, const uint8_t *dirty_in, uint8_t *dirty_out)
{
    __shared__ uint32_t o[(kTile + 2) * (kTile + 2)][kMaxWords];
    const int R = B.R, W = B.W, tpr = (R + kTile - 1) / kTile;
    if (!dirty_in[blockIdx.x]) return;
    const int by = blockIdx.x % tpr, bz = blockIdx.x / tpr;
    for (int i = threadIdx.x; i < (kTile + 2) * (kTile + 2) * W; i += blockDim.x) {
        const int r = i / W, w = i % W;
        const int y = by * kTile + r % (kTile + 2) - 1, z = bz * kTile + r / (kTile + 2) - 1;
        o[r][w] = y >= 0 && z >= 0 && y < R && z < R ? B.out[row_word(B, y, z) + w] : 0;
    }
    __syncthreads();
    bool any = false;
    for (int sweep = 0; sweep <= 32 * kTile * kTile * W; ++sweep) {
        int changed = 0;
        for (int i = threadIdx.x; i < kTile * kTile * W; i += blockDim.x) {
            const int w = i % W, ty = i / W % kTile, tz = i / W / kTile;
            const int y = by * kTile + ty, z = bz * kTile + tz, r = (tz + 1) * (kTile + 2) + ty + 1;
            if (y >= R || z >= R) continue;
            const uint32_t f = B.free_[row_word(B, y, z) + w], was = o[r][w];
            uint32_t next = o[r - 1][w] | o[r + 1][w] | o[r - kTile - 2][w] | o[r + kTile + 2][w];
            if (w > 0) next |= o[r][w - 1] >> 31;
            if (w + 1 < W) next |= o[r][w + 1] << 31;
            const uint32_t now = spread(was | (next & f), f);
            if (now != was) {
                o[r][w] = now;
                changed = 1;
            }
        }
        changed = __syncthreads_or(changed);
        if (!changed) break;
        any = true;
    }
    if (!any) return;
    for (int i = threadIdx.x; i < kTile * kTile * W; i += blockDim.x) {
        const int w = i % W, ty = i / W % kTile, tz = i / W / kTile;
        const int y = by * kTile + ty, z = bz * kTile + tz;
        if (y < R && z < R) B.out[row_word(B, y, z) + w] = o[(tz + 1) * (kTile + 2) + ty + 1][w];
    }
    if (threadIdx.x == 0) {
        atomicExch(&dev[4], 1);
        dirty_out[blockIdx.x] = 1;
        if (by > 0) dirty_out[blockIdx.x - 1] = 1;
        if (by + 1 < tpr) dirty_out[blockIdx.x + 1] = 1;
        if (bz > 0) dirty_out[blockIdx.x - tpr] = 1;
        if (bz + 1 < tpr) dirty_out[blockIdx.x + tpr] = 1;
    }
}

// inside: the field (outside ? d : -d) - 0.9/R is negative
__global__ void k_s1_inside(Bits B)
{
    PAMO_GRID_STRIDE(i, (long long)B.R * B.R * B.W)
        B.in[i] = (~B.out[i] | B.low[i]) & valid_bits(B.R, (int)(i % B.W));
}

// ------------------------------------------------------- 4. dual marching cubes
__device__ __forceinline__ bool bit_at(const uint32_t *b, const Bits &B, int x, int y, int z)
{
    return b[row_word(B, y, z) + (x >> 5)] >> (x & 31) & 1u;
}

// the field at a sample
__device__ __forceinline__ double fval(const unsigned long long *field, const Bits &B, int x, int y, int z)
{
    const double ud = sqrt(__longlong_as_double((long long)field[gidx(x, y, z, B.R)]));
    return (bit_at(B.out, B, x, y, z) ? ud : -ud) - 0.9 / B.R;
}

__device__ __forceinline__ int cell_case(const Bits &B, int x, int y, int z)
{
    int cs = 0;
    for (int c = 0; c < 8; ++c) cs |= (int)bit_at(B.in, B, x + (c & 1), y + ((c >> 1) & 1), z + ((c >> 2) & 1)) << c;
    return cs;
}

// Word w of row (y, z) of the (R - 1)^3 cells: which cells have at least one, two,
// three, four patches, and the number of patches before the word (first).
struct Cells {
    int C, W;
    uint32_t *has[4];
    int *first;
};

__device__ __forceinline__ long long cell_word(const Cells &K, int x, int y, int z)
{
    return ((long long)z * K.C + y) * K.W + (x >> 5);
}

// the number of the cell's first patch
__device__ __forceinline__ int cell_first(const Cells &K, int x, int y, int z)
{
    const long long i = cell_word(K, x, y, z);
    const uint32_t below = (1u << (x & 31)) - 1u;
    int n = K.first[i];
#pragma unroll
    for (int k = 0; k < 4; ++k) n += __popc(K.has[k][i] & below);
    return n;
}

__global__ void k_s1_cells(Bits B, Cells K)
{
    PAMO_GRID_STRIDE(i, (long long)K.C * K.C * K.W)
    {
        const int w = (int)(i % K.W), y = (int)(i / K.W % K.C), z = (int)(i / ((long long)K.W * K.C));
        uint32_t any = 0, all = 0xFFFFFFFFu;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const long long q = row_word(B, y + (r & 1), z + (r >> 1)) + w;
            const uint32_t a = B.in[q], b = w + 1 < B.W ? B.in[q + 1] : 0u;
            const uint32_t s = (a >> 1) | (b << 31);
            any |= a | s;
            all &= a & s;
        }
        uint32_t has[4] = {0, 0, 0, 0};
        int n = 0;
        for (uint32_t todo = any & ~all & valid_bits(K.C, w); todo; todo &= todo - 1) {
            const int b = __ffs(todo) - 1;
            const int np = c_npatch[cell_case(B, 32 * w + b, y, z)];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (np > k) has[k] |= 1u << b;
            n += np;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) K.has[k][i] = has[k];
        K.first[i] = n;  // counts: scanned in place
    }
}

// The numbered patches and quads as lists, so that the kernels that compute them
// have one of each in every thread: patch k's cell and which of its patches (4 cell
// + patch), quad q's word and bit (32 word + bit).  Warps that looked for set bits
// among their words instead held ten lanes busy and a surface's words fell to few
// of them (k_s1_verts and k_s1_quads 0.75 ms together at R = 256).
__global__ void k_s1_lists(Cells K, const uint32_t *edge_mask, const int *edge_first, long long edge_words,
                           uint32_t *patches, uint32_t *quads)
{
    const long long cwords = (long long)K.C * K.C * K.W;
    PAMO_GRID_STRIDE(i, cwords + edge_words)
    {
        if (i < cwords) {
            int n = K.first[i];
            const uint32_t h0 = K.has[0][i];
            if (!h0) continue;
            const uint32_t h1 = K.has[1][i], h2 = K.has[2][i], h3 = K.has[3][i];
            const uint32_t cell0 = (uint32_t)(i / K.W * K.C + (i % K.W) * 32);
            for (uint32_t todo = h0; todo; todo &= todo - 1) {
                const int b = __ffs(todo) - 1;
                const int np = 1 + (h1 >> b & 1) + (h2 >> b & 1) + (h3 >> b & 1);
                for (int p = 0; p < np; ++p) patches[n++] = 4 * (cell0 + b) + p;
            }
        } else {
            const long long j = i - cwords;
            int n = edge_first[j];
            for (uint32_t todo = edge_mask[j]; todo; todo &= todo - 1)
                quads[n++] = (uint32_t)(32 * j) + (__ffs(todo) - 1);
        }
    }
}

// the patch vertices: the mean of a patch's edges' crossing points (edge order),
// in sample-index coordinates, mapped to the centred frame
__global__ void __launch_bounds__(kThreads) k_s1_verts(const unsigned long long *field, Bits B,
                                                       const uint32_t *patches, int nv, double band, double margin,
                                                       double tmax, const int *dev, float *verts)
{
    const int R = B.R, C = R - 1;
    double lo[3];
    for (int k = 0; k < 3; ++k) lo[k] = (double)ordered_to_float(dev[k]);
    PAMO_GRID_STRIDE(i, nv)
    {
        const uint32_t code = patches[i], cell = code >> 2;
        const int p = (int)(code & 3u);
        const int x = (int)(cell % (uint32_t)C), y = (int)(cell / (uint32_t)C % (uint32_t)C),
                  z = (int)(cell / ((uint32_t)C * (uint32_t)C));
        const int cs = cell_case(B, x, y, z);
        double d[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) d[c] = fval(field, B, x + (c & 1), y + ((c >> 1) & 1), z + ((c >> 2) & 1));
        double sx = 0, sy = 0, sz = 0;
        int cnt = 0;
#pragma unroll
        for (int e = 0; e < 12; ++e) {
            if (c_patch[cs][e] != p) continue;
            int a, b;
            edge_corners(e, a, b);
            const int ax = x + (a & 1), ay = y + ((a >> 1) & 1), az = z + ((a >> 2) & 1);
            const int bx = x + (b & 1), by = y + ((b >> 1) & 1), bz = z + ((b >> 2) & 1);
            const double t = d[a] / (d[a] - d[b]);
            sx += ax + t * (double)(bx - ax);
            sy += ay + t * (double)(by - ay);
            sz += az + t * (double)(bz - az);
            cnt++;
        }
        const double v[3] = {sx / cnt, sy / cnt, sz / cnt};
        for (int k = 0; k < 3; ++k) {
            const double xn = (v[k] + 0.5) / R;
            verts[3LL * i + k] = (float)((xn * margin - band) * tmax + lo[k]);
        }
    }
}

// Crossed grid edges whose four cells exist (every crossed edge, given the grid's
// outer layer is outside), by axis and lower sample: a mask per word of samples
// and its count (scanned in place).
__global__ void k_s1_edges(Bits B, uint32_t *mask, int *first)
{
    const int R = B.R;
    const long long words = (long long)R * R * B.W;
    PAMO_GRID_STRIDE(i, 3 * words)
    {
        const int ax = (int)(i / words);
        const long long g = i % words;
        const int w = (int)(g % B.W), y = (int)(g / B.W % R), z = (int)(g / ((long long)B.W * R));
        // the four cells need the two other coordinates in [1, R - 2]
        const bool room = (ax == 1 ? y + 1 < R : y >= 1 && y <= R - 2) && (ax == 2 ? z + 1 < R : z >= 1 && z <= R - 2);
        uint32_t m = 0;
        if (room) {
            const uint32_t a = B.in[g];
            uint32_t b;
            if (ax == 0) b = (a >> 1) | (w + 1 < B.W ? B.in[g + 1] << 31 : 0u);
            else b = B.in[g + (ax == 1 ? (long long)B.W : (long long)B.W * R)];
            m = (a ^ b) & valid_bits(R - 1, w);  // x <= R - 2
            if (ax != 0 && w == 0) m &= ~1u;
        }
        mask[i] = m;
        first[i] = __popc(m);
    }
}

__device__ __forceinline__ double max_cos(const float *v, int i0, int i1, int i2)
{
    const D3 a = {v[3 * i0], v[3 * i0 + 1], v[3 * i0 + 2]};
    const D3 b = {v[3 * i1], v[3 * i1 + 1], v[3 * i1 + 2]};
    const D3 c = {v[3 * i2], v[3 * i2 + 1], v[3 * i2 + 2]};
    auto cosang = [](D3 p, D3 r, D3 s) {
        D3 u = dsub(r, p), w = dsub(s, p);
        const double nu = fmax(sqrt(u.x * u.x + u.y * u.y + u.z * u.z), 1e-12);
        const double nw = fmax(sqrt(w.x * w.x + w.y * w.y + w.z * w.z), 1e-12);
        u = {u.x / nu, u.y / nu, u.z / nu};
        w = {w.x / nw, w.y / nw, w.z / nw};
        return u.x * w.x + u.y * w.y + u.z * w.z;
    };
    return fmax(fmax(cosang(a, b, c), cosang(b, c, a)), cosang(c, a, b));
}

// one quad per crossed edge, through the patch vertices of its four cells
// (counterclockwise seen from the +axis side when the lower sample is inside),
// and whether it splits the first way
__global__ void __launch_bounds__(kThreads) k_s1_quads(Bits B, Cells K, const uint32_t *list, int nq,
                                                       const float *verts, int4 *quads, int *q_first)
{
    const int R = B.R;
    const uint32_t words = (uint32_t)((long long)R * R * B.W);
    PAMO_GRID_STRIDE(q, nq)
    {
        const uint32_t word = list[q] >> 5;
        const int ax = (int)(word / words);
        const uint32_t g = word % words;
        const int x = (int)(g % B.W * 32 + (list[q] & 31u)), y = (int)(g / B.W % R), z = (int)(g / ((uint32_t)B.W * R));
        // the other two axes in cyclic order (b, c) with b x c = the edge's axis
        const int bax = (ax + 1) % 3, cax = (ax + 2) % 3;
        int vs[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int ob = k == 1 || k == 2 ? -1 : 0, oc = k >= 2 ? -1 : 0;
            const int cx = x + (bax == 0 ? ob : 0) + (cax == 0 ? oc : 0);
            const int cy = y + (bax == 1 ? ob : 0) + (cax == 1 ? oc : 0);
            const int cz = z + (bax == 2 ? ob : 0) + (cax == 2 ? oc : 0);
            // the edge's corners inside this cell
            const int ca = (x - cx) + 2 * (y - cy) + 4 * (z - cz);
            const int e = ax * 4 + (ax == 0 ? (ca >> 1) : (ax == 1 ? ((ca & 1) | ((ca >> 1) & 2)) : (ca & 3)));
            vs[k] = cell_first(K, cx, cy, cz) + c_patch[cell_case(B, cx, cy, cz)][e];
        }
        const bool lower_inside = bit_at(B.in, B, x, y, z);
        const int4 qd = lower_inside ? make_int4(vs[0], vs[1], vs[2], vs[3]) : make_int4(vs[3], vs[2], vs[1], vs[0]);
        quads[q] = qd;
        const double a1 = fmax(max_cos(verts, qd.x, qd.y, qd.w), max_cos(verts, qd.y, qd.z, qd.w));
        const double a2 = fmax(max_cos(verts, qd.x, qd.y, qd.z), max_cos(verts, qd.x, qd.z, qd.w));
        q_first[q] = a1 < a2 ? 1 : 0;
    }
}

__global__ void k_s1_faces(const int4 *quads, const int *flag, const int *pos, int nq, const int *n_first, int *faces)
{
    const int n1 = *n_first;
    PAMO_GRID_STRIDE(q, nq)
    {
        const int4 d = quads[q];
        int *f;
        int t[6];
        if (flag[q]) {
            f = faces + 6LL * pos[q];
            t[0] = d.x; t[1] = d.y; t[2] = d.w; t[3] = d.y; t[4] = d.z; t[5] = d.w;
        } else {
            f = faces + 6LL * (n1 + (q - pos[q]));
            t[0] = d.x; t[1] = d.y; t[2] = d.z; t[3] = d.x; t[4] = d.z; t[5] = d.w;
        }
        for (int k = 0; k < 6; ++k) f[k] = t[k];
    }
}

__global__ void k_s1_dev_init(int *dev)
{
    if (threadIdx.x < 3) dev[threadIdx.x] = 0x7FFFFFFF;  // min (ordered)
    else if (threadIdx.x == 3) dev[3] = (int)0x80000000;
    else if (threadIdx.x < 16) dev[threadIdx.x] = 0;
}

// k_s1_quads numbers a cell's edge from its lower corner: along x by (y, z),
// along y by (x, z), along z by (x, y) -- the order of kEdgeCorners
static_assert(kEdgeCorners[5][0] == 1 && kEdgeCorners[5][1] == 3 && kEdgeCorners[6][0] == 4, "edge numbering");

}  // namespace

#define S1_TRY(expr)                                      \
    do {                                                  \
        cudaError_t _e = (expr);                          \
        if (_e != cudaSuccess) return map_cuda_error(_e); \
    } while (0)

void Stage1::release()
{
    void *p[] = {tris, field, bits, cell_bits, cell_first, edge_bits, edge_first, scan_cells, scan_edges, scan_quads,
                 quads, q_first, q_pos, verts, faces, dev, mean_dev, tile_dirty,
                 patch_list, quad_list};
    for (void *x : p)
        if (x) cudaFree(x);
    if (h_dev) cudaFreeHost(h_dev);
    tris = nullptr;
    field = nullptr;
    bits = cell_bits = edge_bits = patch_list = quad_list = nullptr;
    cell_first = edge_first = scan_cells = scan_edges = scan_quads = nullptr;
    quads = nullptr;
    q_first = q_pos = nullptr;
    verts = nullptr;
    faces = nullptr;
    dev = h_dev = nullptr;
    mean_dev = nullptr;
    tile_dirty = nullptr;
    cap_tris = cap_grid = cap_words = cap_verts = cap_quads = cap_tiles = 0;
}

int Stage1::ensure(long long m, int R_)
{
    const long long n3 = (long long)R_ * R_ * R_;
    const long long tpr = (R_ + kTile - 1) / kTile, nt = tpr * tpr;
    const long long nw = (long long)R_ * R_ * ((R_ + 31) / 32);  // words of the grid; the cells have fewer
    if (m <= cap_tris && n3 <= cap_grid && nt <= cap_tiles && nw <= cap_words && dev) return PAMO_OK;
    const long long ctl = nt > cap_tiles ? nt : cap_tiles, cw = nw > cap_words ? nw : cap_words;
    const long long cm = m > cap_tris ? m : cap_tris, cg = n3 > cap_grid ? n3 : cap_grid;
    void *keep_v = verts, *keep_f = faces, *keep_q = quads, *keep_qf = q_first, *keep_qp = q_pos, *keep_sq = scan_quads;
    void *keep_pl = patch_list, *keep_ql = quad_list;
    const long long kv = cap_verts, kq = cap_quads;
    verts = nullptr;
    faces = nullptr;
    quads = nullptr;
    q_first = q_pos = nullptr;
    scan_quads = nullptr;
    patch_list = quad_list = nullptr;
    release();
    verts = (float *)keep_v;
    faces = (int *)keep_f;
    quads = (int4 *)keep_q;
    q_first = (int *)keep_qf;
    q_pos = (int *)keep_qp;
    scan_quads = (int *)keep_sq;
    patch_list = (uint32_t *)keep_pl;
    quad_list = (uint32_t *)keep_ql;
    cap_verts = kv;
    cap_quads = kq;
#define S1A(ptr, bytes)                                                    \
    if (cudaMalloc((void **)&ptr, (size_t)(bytes)) != cudaSuccess) {       \
        release();                                                         \
        return PAMO_ERR_OOM;                                               \
    }
    S1A(tris, 9 * 4 * (cm + 1));
    S1A(field, 8 * cg);
    S1A(bits, 4 * 4 * cw);
    S1A(tile_dirty, 2 * ctl);
    S1A(cell_bits, 4 * 4 * cw);
    S1A(cell_first, 4 * cw);
    S1A(edge_bits, 3 * 4 * cw);
    S1A(edge_first, 3 * 4 * cw);
    S1A(scan_cells, 4 * scan_scratch_ints(cw));
    S1A(scan_edges, 4 * scan_scratch_ints(3 * cw));
    S1A(dev, 64);
    S1A(mean_dev, 16);
#undef S1A
    if (cudaMallocHost((void **)&h_dev, 64) != cudaSuccess) {
        release();
        return PAMO_ERR_OOM;
    }
    if (scan_scratch_init(scan_cells, scan_scratch_ints(cw)) != cudaSuccess ||
        scan_scratch_init(scan_edges, scan_scratch_ints(3 * cw)) != cudaSuccess) {
        release();
        return PAMO_ERR_OOM;
    }
    cap_tris = cm;
    cap_grid = cg;
    cap_tiles = ctl;
    cap_words = cw;
    return PAMO_OK;
}

int Stage1::ensure_out(long long nv, long long nq)
{
    if (nv > cap_verts || !verts) {
        if (verts) cudaFree(verts);
        if (patch_list) cudaFree(patch_list);
        verts = nullptr;
        patch_list = nullptr;
        cap_verts = 0;
        const long long c = nv + nv / 8 + 64;
        if (cudaMalloc((void **)&verts, (size_t)c * 12) != cudaSuccess ||
            cudaMalloc((void **)&patch_list, (size_t)c * 4) != cudaSuccess)
            return PAMO_ERR_OOM;
        cap_verts = c;
    }
    if (nq > cap_quads || !quads) {
        void *p[] = {quads, q_first, q_pos, faces, scan_quads, quad_list};
        for (void *x : p)
            if (x) cudaFree(x);
        quads = nullptr;
        q_first = q_pos = nullptr;
        faces = nullptr;
        scan_quads = nullptr;
        quad_list = nullptr;
        cap_quads = 0;
        const long long c = nq + nq / 8 + 64;
        if (cudaMalloc((void **)&quads, (size_t)c * 16) != cudaSuccess ||
            cudaMalloc((void **)&q_first, (size_t)c * 4) != cudaSuccess ||
            cudaMalloc((void **)&q_pos, (size_t)c * 4) != cudaSuccess ||
            cudaMalloc((void **)&quad_list, (size_t)c * 4) != cudaSuccess ||
            cudaMalloc((void **)&faces, (size_t)c * 24) != cudaSuccess ||
            cudaMalloc((void **)&scan_quads, (size_t)scan_scratch_ints(c) * 4) != cudaSuccess)
            return PAMO_ERR_OOM;
        if (scan_scratch_init(scan_quads, scan_scratch_ints(c)) != cudaSuccess) return PAMO_ERR_OOM;
        cap_quads = c;
    }
    return PAMO_OK;
}

int remesh(Stage1 &S, const float *d_points, const int *d_tris, int n_pts, int m, const float *mean_dev, int R,
           cudaStream_t s)
{
    (void)n_pts;
    if (R < 4 || R > 1024 || m <= 0) return PAMO_ERR_INVALID_ARG;
    int rc = S.ensure(m, R);
    if (rc) return rc;
    S.R = R;
    static signed char h_patch[256][12];
    static unsigned char h_npatch[256];
    static bool have_table = false;
    if (!have_table) {  // the same table for every device; built once per process
        build_patch_table(h_patch, h_npatch);
        have_table = true;
    }
    S1_TRY(cudaMemcpyToSymbolAsync(c_patch, h_patch, sizeof(h_patch), 0, cudaMemcpyHostToDevice, s));
    S1_TRY(cudaMemcpyToSymbolAsync(c_npatch, h_npatch, sizeof(h_npatch), 0, cudaMemcpyHostToDevice, s));
    const double band = 3.0 / R, margin = band * 2 + 1;
    const long long n3 = (long long)R * R * R;
    // 1. normalise
    if (S.prof) S.prof->begin(PH_S1_PREP, s);
    launch(k_s1_dev_init, 1, 32, 0, s, S.dev);
    launch(k_s1_min, grid_for(m), kThreads, 0, s, d_points, d_tris, m, mean_dev, S.dev);
    launch(k_s1_max, grid_for(m), kThreads, 0, s, d_points, d_tris, m, mean_dev, S.dev);
    launch(k_s1_normalise, grid_for(m), kThreads, 0, s, d_points, d_tris, m, mean_dev, S.dev, (float)band,
           (float)margin, R, S.tris);
    // 2. unsigned distance: squared distances start at band^2 (bits of a double)
    if (S.prof) S.prof->begin(PH_S1_DIST, s);
    const double b2 = band * band;
    unsigned long long fill;
    memcpy(&fill, &b2, 8);
    launch(k_s1_fill, grid_for(n3), kThreads, 0, s, S.field, n3, fill);  // cudaMemset only sets bytes
    const double inv_r = (R & (R - 1)) == 0 ? 1.0 / R : 0.0;
    launch(k_s1_udist, grid_for(32LL * m), 256, 0, s, (const float *)S.tris, m, R, inv_r, band,
           (const int *)S.dev, S.field);
    const int W = (R + 31) / 32, C = R - 1;
    const long long words = (long long)R * R * W;
    const Bits bits{R, W, S.bits, S.bits + words, S.bits + 2 * words, S.bits + 3 * words};
    launch(k_s1_bits, grid_for(8 * words), kThreads, 0, s, (const unsigned long long *)S.field, bits, fill);
    // 3. flood fill from the boundary, until nothing changes
    if (S.prof) S.prof->begin(PH_S1_FLOOD, s);
    const int tpr = (R + kTile - 1) / kTile;
    const int tiles = tpr * tpr;
    // two dirty-tile flag sets used in turn: every tile is dirty at first
    uint8_t *dirty[2] = {S.tile_dirty, S.tile_dirty + tiles};
    S1_TRY(cudaMemsetAsync(dirty[0], 1, (size_t)tiles, s));
    S1_TRY(cudaMemsetAsync(dirty[1], 0, (size_t)tiles, s));
    int cur = 0;
    bool settled = false;
    // A launch that changes anything sets a bit, so n3 + 1 launches settle any grid; a
    // surface takes a few, a path that winds between two tiles one per crossing.
    for (long long round = 0; round <= n3 && !settled; round += 6) {
        for (int k = 0; k < 6; ++k) {
            if (k == 5) S1_TRY(cudaMemsetAsync(S.dev + 4, 0, 4, s));  // settled: nothing changed in the last launch
            launch(k_s1_flood, tiles, kThreads, 0, s, bits, S.dev, (const uint8_t *)dirty[cur], dirty[cur ^ 1]);
            S1_TRY(cudaMemsetAsync(dirty[cur], 0, (size_t)tiles, s));
            cur ^= 1;
        }
        S1_TRY(cudaMemcpyAsync(S.h_dev, S.dev, 64, cudaMemcpyDeviceToHost, s));
        S1_TRY(cudaStreamSynchronize(s));
        if (S.prof) S.prof->collect();
        settled = S.h_dev[4] == 0;
    }
    if (!settled) return PAMO_ERR_DEVICE;  // cannot happen: see above
    launch(k_s1_inside, grid_for(words), kThreads, 0, s, bits);
    // 4. dual marching cubes: patch and quad numbers, then the patch vertices
    if (S.prof) S.prof->begin(PH_S1_DMC, s);
    const long long cwords = (long long)C * C * ((C + 31) / 32);
    const Cells cells{C, (C + 31) / 32,
                      {S.cell_bits, S.cell_bits + cwords, S.cell_bits + 2 * cwords, S.cell_bits + 3 * cwords},
                      S.cell_first};
    launch(k_s1_cells, grid_for(cwords), kThreads, 0, s, bits, cells);
    launch(k_s1_edges, grid_for(3 * words), kThreads, 0, s, bits, S.edge_bits, S.edge_first);
    S1_TRY(scan_jobs(ScanJob{S.cell_first, nullptr, S.cell_first, nullptr, cwords, nullptr, S.scan_cells, S.dev + 8},
                     ScanJob{S.edge_first, nullptr, S.edge_first, nullptr, 3 * words, nullptr, S.scan_edges, S.dev + 9},
                     s, S.dev + 6));
    S1_TRY(cudaMemcpyAsync(S.h_dev, S.dev, 64, cudaMemcpyDeviceToHost, s));
    S1_TRY(cudaStreamSynchronize(s));
    if (S.h_dev[6]) return PAMO_ERR_DEVICE;  // a scan's wait ran out
    const long long nv = S.h_dev[8], nq = S.h_dev[9];
    if (nv <= 0 || nq <= 0 || 2 * nq > 0x7FFFFFFF) return nv <= 0 || nq <= 0 ? PAMO_ERR_INVALID_ARG : PAMO_ERR_CAPACITY;
    if ((rc = S.ensure_out(nv, nq))) return rc;
    float tmax = 0.f;
    {
        // the largest coordinate, an ordered int of a non-negative float: its bits
        const int mx_bits = S.h_dev[3];
        if (mx_bits >= 0) memcpy(&tmax, &mx_bits, 4);
    }
    launch(k_s1_lists, grid_for(cwords + 3 * words), kThreads, 0, s, cells, (const uint32_t *)S.edge_bits,
           (const int *)S.edge_first, 3 * words, S.patch_list, S.quad_list);
    launch(k_s1_verts, grid_for(nv), kThreads, 0, s, (const unsigned long long *)S.field, bits,
           (const uint32_t *)S.patch_list, (int)nv, band, margin, (double)tmax, (const int *)S.dev, S.verts);
    // quads and their split
    launch(k_s1_quads, grid_for(nq), kThreads, 0, s, bits, cells, (const uint32_t *)S.quad_list, (int)nq,
           (const float *)S.verts, S.quads, S.q_first);
    S1_TRY(scan_job(ScanJob{S.q_first, nullptr, S.q_pos, nullptr, nq, nullptr, S.scan_quads, S.dev + 10}, s, S.dev + 6));
    launch(k_s1_faces, grid_for(nq), kThreads, 0, s, (const int4 *)S.quads, (const int *)S.q_first,
           (const int *)S.q_pos, (int)nq, (const int *)(S.dev + 10), S.faces);
    S1_TRY(cudaMemcpyAsync(S.h_dev + 6, S.dev + 6, 4, cudaMemcpyDeviceToHost, s));
    S1_TRY(cudaStreamSynchronize(s));
    if (S.h_dev[6]) return PAMO_ERR_DEVICE;
    if (S.prof) S.prof->end(s);
    S1_TRY(cudaGetLastError());
    S.n_verts = (int)nv;
    S.n_tris = (int)(2 * nq);
    return PAMO_OK;
}

}  // namespace s1
}  // namespace pamo
