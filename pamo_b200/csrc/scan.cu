#include "scan.cuh"

namespace pamo {

namespace {

struct ScanPair {
    ScanJob j[2];
};

__device__ __forceinline__ int scan_value(const ScanJob &J, long long i)
{
    return J.faces ? (J.faces[i].x >= 0) : J.in[i];
}

// Small inputs: one block per job, 16 consecutive items per thread (four vector
// loads and stores where the job's arrays lie on 16-byte boundaries).
constexpr int kSingleThreads = 1024;
constexpr int kSingleItems = 16;

__global__ void __launch_bounds__(kSingleThreads) k_scan_single(const __grid_constant__ ScanPair P)
{
    chain_wait();
    const ScanJob &J = P.j[blockIdx.x];
    const long long n = J.d_n ? (long long)*J.d_n : J.n;
    const long long base = (long long)threadIdx.x * kSingleItems;
    const bool vec = base + kSingleItems <= n && !J.faces &&
                     ((reinterpret_cast<unsigned long long>(J.in) | reinterpret_cast<unsigned long long>(J.out)) & 15) == 0;
    int v[kSingleItems];
    int sum = 0;
    if (vec) {
        const int4 *in4 = reinterpret_cast<const int4 *>(J.in + base);
#pragma unroll
        for (int k = 0; k < kSingleItems / 4; ++k) {
            const int4 x = in4[k];
            v[4 * k] = x.x; v[4 * k + 1] = x.y; v[4 * k + 2] = x.z; v[4 * k + 3] = x.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < kSingleItems; ++k) v[k] = base + k < n ? scan_value(J, base + k) : 0;
    }
#pragma unroll
    for (int k = 0; k < kSingleItems; ++k) sum += v[k];
    int tot;
    int ex = block_excl_scan<kSingleThreads>(sum, tot);
    if (J.list) {
        int at = ex;
#pragma unroll
        for (int k = 0; k < kSingleItems; ++k)
            if (v[k]) J.list[at++] = (int)(base + k);
    }
    if (J.out && vec) {
        int4 *out4 = reinterpret_cast<int4 *>(J.out + base);
#pragma unroll
        for (int k = 0; k < kSingleItems / 4; ++k) {
            int4 x;
            x.x = ex; ex += v[4 * k];
            x.y = ex; ex += v[4 * k + 1];
            x.z = ex; ex += v[4 * k + 2];
            x.w = ex; ex += v[4 * k + 3];
            out4[k] = x;
        }
    } else if (J.out) {
#pragma unroll
        for (int k = 0; k < kSingleItems; ++k) {
            if (base + k < n) J.out[base + k] = ex;
            ex += v[k];
        }
    }
    if (threadIdx.x == 0 && J.d_total) *J.d_total = tot;
}

// Single pass with decoupled look-back (see scan.cuh).  Header: [0] next tile,
// [1] finished blocks, [2] fault.  Status word of a tile: high half the call's
// epoch (30 bits) and a flag (1: the tile's own sum, 2: its inclusive prefix),
// low half the value; a word from an earlier call (another epoch) reads as not
// yet published.
constexpr unsigned kFlagSum = 1, kFlagPrefix = 2;

__device__ __forceinline__ unsigned long long status_word(unsigned epoch, unsigned flag, int value)
{
    return ((unsigned long long)((epoch << 2) | flag) << 32) | (unsigned)value;
}

// spin_limit bounds each wait (polls); absent_tile >= 0 makes that tile never
// publish (only the wait-timeout test passes one: its waiters must give up).
__global__ void __launch_bounds__(kScanThreads) k_scan_lookback(const __grid_constant__ ScanPair P, int blocks0,
                                                                int *fault, unsigned epoch, long long spin_limit,
                                                                long long absent_tile)
{
    chain_wait();
    __shared__ int tile[kScanTile];
    __shared__ long long s_t;
    __shared__ int s_prefix;
    const int which = (int)blockIdx.x >= blocks0 ? 1 : 0;
    const ScanJob &J = P.j[which];
    int *scratch = J.scratch;
    const int job_blocks = which ? (int)gridDim.x - blocks0 : blocks0;
    volatile unsigned long long *status = reinterpret_cast<volatile unsigned long long *>(scratch + kScanHeader);
    const long long n = J.d_n ? (long long)*J.d_n : J.n;
    const long long n_tiles = (n + kScanTile - 1) / kScanTile;
    if (threadIdx.x == 0) s_t = atomicAdd(&scratch[0], 1);
    __syncthreads();
    const long long t = s_t;
    if (t < n_tiles) {
        const long long base = t * kScanTile;
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            long long i = base + (long long)k * kScanThreads + threadIdx.x;
            tile[k * kScanThreads + threadIdx.x] = i < n ? scan_value(J, i) : 0;
        }
        __syncthreads();
        int local[kScanItems];
        int sum = 0;
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            local[k] = sum;
            sum += tile[threadIdx.x * kScanItems + k];
        }
        int agg;
        const int ex = block_excl_scan<kScanThreads>(sum, agg);
        if (threadIdx.x < 32) {
            const int lane = threadIdx.x;
            if (lane == 0 && t != absent_tile) status[t] = status_word(epoch, t == 0 ? kFlagPrefix : kFlagSum, agg);
            int prefix = 0;
            bool timed_out = false;
            for (long long top = t - 1; top >= 0 && !timed_out;) {
                // lane l looks at tile top - l (lane 0 the nearest)
                const long long j = top - lane;
                unsigned flag = kFlagPrefix;
                int val = 0;
                if (j >= 0) {
                    unsigned long long w = status[j];
                    for (long long spins = 0;; ++spins) {
                        const unsigned hi = (unsigned)(w >> 32);
                        if ((hi >> 2) == (epoch & 0x3FFFFFFFu) && (hi & 3u) != 0) {
                            flag = hi & 3u;
                            val = (int)(unsigned)w;
                            break;
                        }
                        if (spins > spin_limit) {  // a tile that started earlier never published
                            timed_out = true;
                            break;
                        }
                        __nanosleep(20);
                        w = status[j];
                    }
                }
                timed_out = __any_sync(0xffffffffu, timed_out);
                // the nearest tile with its prefix ends the look-back (a lane past
                // tile 0 counts as one, with value 0); before it, the tiles' sums
                const unsigned stops = __ballot_sync(0xffffffffu, flag == kFlagPrefix);
                const int stop = stops ? __ffs(stops) - 1 : 31;
                int v = lane <= stop ? val : 0;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                prefix += v;
                if (stops) break;
                top -= 32;
            }
            if (lane == 0) {
                if (timed_out) {
                    atomicExch(&scratch[2], 1);
                    if (fault) atomicExch(fault, 1);
                }
                if (t != absent_tile) status[t] = status_word(epoch, kFlagPrefix, prefix + agg);
                s_prefix = prefix;
                if (t == n_tiles - 1 && J.d_total) *J.d_total = prefix + agg;
            }
        }
        __syncthreads();
        const int off = s_prefix + ex;
        if (J.list) {
#pragma unroll
            for (int k = 0; k < kScanItems; ++k)
                if (tile[threadIdx.x * kScanItems + k])
                    J.list[off + local[k]] = (int)(base + threadIdx.x * kScanItems + k);
        }
        if (J.out) {
#pragma unroll
            for (int k = 0; k < kScanItems; ++k) tile[threadIdx.x * kScanItems + k] = local[k] + off;
            __syncthreads();
#pragma unroll
            for (int k = 0; k < kScanItems; ++k) {
                long long i = base + (long long)k * kScanThreads + threadIdx.x;
                if (i < n) J.out[i] = tile[k * kScanThreads + threadIdx.x];
            }
        }
    } else if (n_tiles == 0 && t == 0 && threadIdx.x == 0 && J.d_total) {
        *J.d_total = 0;
    }
    // the last block to finish leaves the header at zero for the next scan
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&scratch[1], 1) == job_blocks - 1) {
            scratch[0] = 0;
            scratch[1] = 0;
        }
    }
}

constexpr long long kScanSpinLimit = 1LL << 22;  // ~0.1 s of polls: far beyond any real wait

cudaError_t scan_pair(const ScanPair &P, int n_jobs, cudaStream_t s, int *fault, long long spin_limit,
                      long long absent_tile)
{
    static std::atomic<unsigned> epochs{0};
    bool single = true;
    long long tiles[2] = {0, 0};
    for (int k = 0; k < n_jobs; ++k) {
        tiles[k] = (P.j[k].n + kScanTile - 1) / kScanTile;
        single = single && P.j[k].n <= (long long)kSingleThreads * kSingleItems;
    }
    if (single) {
        launch_chained(k_scan_single, n_jobs, kSingleThreads, 0, s, P);
        return cudaGetLastError();
    }
    const unsigned epoch = (epochs.fetch_add(1, std::memory_order_relaxed) + 1) & 0x3FFFFFFFu;
    launch_chained(k_scan_lookback, (unsigned)(tiles[0] + tiles[1]), kScanThreads, 0, s, P, (int)tiles[0], fault, epoch,
           spin_limit, absent_tile);
    return cudaGetLastError();
}

}  // namespace

cudaError_t scan_job(const ScanJob &job, cudaStream_t s, int *fault)
{
    if (job.n <= 0) return job.d_total ? cudaMemsetAsync(job.d_total, 0, sizeof(int), s) : cudaSuccess;
    return scan_pair(ScanPair{{job, ScanJob{}}}, 1, s, fault, kScanSpinLimit, -1);
}

cudaError_t scan_jobs(const ScanJob &a, const ScanJob &b, cudaStream_t s, int *fault)
{
    if (a.n <= 0 || b.n <= 0) {
        const cudaError_t e = scan_job(a, s, fault);
        return e != cudaSuccess ? e : scan_job(b, s, fault);
    }
    return scan_pair(ScanPair{{a, b}}, 2, s, fault, kScanSpinLimit, -1);
}

cudaError_t exclusive_scan(const int *in, int *out, long long n_max, const int *d_n, int *scratch, int *d_total,
                           cudaStream_t s, int *fault)
{
    return scan_job(ScanJob{in, nullptr, out, nullptr, n_max, d_n, scratch, d_total}, s, fault);
}

cudaError_t exclusive_scan_waits(const int *in, int *out, long long n_max, const int *d_n, int *scratch, int *d_total,
                                 cudaStream_t s, int *fault, long long spin_limit, long long absent_tile)
{
    if (n_max <= 0) return d_total ? cudaMemsetAsync(d_total, 0, sizeof(int), s) : cudaSuccess;
    const ScanJob job{in, nullptr, out, nullptr, n_max, d_n, scratch, d_total};
    return scan_pair(ScanPair{{job, ScanJob{}}}, 1, s, fault, spin_limit, absent_tile);
}

}  // namespace pamo
