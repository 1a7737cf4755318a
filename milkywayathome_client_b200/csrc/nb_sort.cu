// LSD radix sort of 64-bit Morton keys with 32-bit body indices, and an int prefix sum.
//
// Replaces the lock-based concurrent insertion of the reference's OpenCL buildTree
// (nbody/kernels/nbody_kernels.cl:898-1159): bodies are ordered by octree path once and
// the tree is derived from the sorted order without locks or spin-waits.
//
// Each of the 8 passes sorts by one 8-bit digit: per-tile digit histograms, a scan of every
// digit's row of the (digit, tile) table (one block a row, its total beside it), and a stable
// scatter that starts each digit after the totals below it: each warp ranks 256 consecutive keys
// with warp match, the tile is put in digit order in shared memory and leaves in runs.  A pass
// reads and writes 12 bytes per key; at a million keys its three launches' latencies bound it.
// The step outside the walk (theta 1), with three more launches a pass for a scan of the whole
// table, a block-wide count of every 256 keys and a key written where it stood -> now: 65,536
// bodies 0.268 -> 0.210 ms, 1,048,576 0.79 -> 0.69 (with the emission's atomics, nb_raise_max).
#include "nb_common.cuh"

namespace {

constexpr int RS_THREADS = 256;
constexpr int RS_ROUNDS = 8;                         // keys per thread per tile
constexpr int RS_TILE = RS_THREADS * RS_ROUNDS;      // 2048 keys per tile
constexpr int RS_WARPS = RS_THREADS / 32;

// digit of item i: 8 bits of its key, or (GROUPED) 8 bits of the group of its index
template <bool GROUPED>
__device__ __forceinline__ unsigned int rs_digit(unsigned long long key, unsigned int idx,
                                                 const int* group, int shift)
{
    if (GROUPED) return ((unsigned) group[idx] >> shift) & 255u;
    return (unsigned) (key >> shift) & 255u;
}

template <bool GROUPED>
__global__ void __launch_bounds__(RS_THREADS)
k_rs_hist(const unsigned long long* __restrict__ keys, const unsigned int* __restrict__ idx,
          const int* __restrict__ group, int n, int shift, unsigned int* __restrict__ hist,
          int nTiles)
{
    __shared__ unsigned int cnt[256];
    cnt[threadIdx.x] = 0;
    __syncthreads();
    const int base = blockIdx.x * RS_TILE;
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; ++r) {
        int i = base + r * RS_THREADS + threadIdx.x;
        if (i < n)
            atomicAdd(&cnt[rs_digit<GROUPED>(GROUPED ? 0ull : keys[i], GROUPED ? idx[i] : 0u,
                                             group, shift)], 1u);
    }
    __syncthreads();
    hist[threadIdx.x * nTiles + blockIdx.x] = cnt[threadIdx.x];
}

template <bool GROUPED>
__global__ void __launch_bounds__(RS_THREADS)
k_rs_scatter(const unsigned long long* __restrict__ keyIn, const unsigned int* __restrict__ idxIn,
             unsigned long long* __restrict__ keyOut, unsigned int* __restrict__ idxOut,
             const int* __restrict__ group, int n, int shift,
             const unsigned int* __restrict__ hist, const unsigned int* __restrict__ totals, int nTiles)
{
    __shared__ unsigned int part[2][RS_WARPS];
    __shared__ unsigned int wHist[RS_WARPS][256];  // per-warp counts, then each warp's start
    __shared__ unsigned int toGlobal[256];         // of each digit: global less tile position
    __shared__ unsigned long long sKey[RS_TILE];   // the tile's keys and indices in digit order
    __shared__ unsigned int sIdx[RS_TILE];
    __shared__ unsigned char sDigit[RS_TILE];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    unsigned int* const mine = wHist[warp];
#pragma unroll
    for (int q = 0; q < 256 / 32; ++q) mine[32 * q + lane] = 0;
    const unsigned int total = totals[t], before = hist[t * nTiles + blockIdx.x];
    __syncwarp();
    // a warp ranks its own run of consecutive keys, 32 at a time, with no word from the others
    const int base = blockIdx.x * RS_TILE + warp * 32 * RS_ROUNDS + lane;
    unsigned long long key[RS_ROUNDS];
    unsigned int idx[RS_ROUNDS], digit[RS_ROUNDS], rank[RS_ROUNDS];
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; ++r) {
        const int i = base + 32 * r;
        const bool valid = i < n;
        key[r] = valid ? keyIn[i] : 0ull;
        idx[r] = valid ? idxIn[i] : 0u;
        digit[r] = valid ? rs_digit<GROUPED>(key[r], idx[r], group, shift) : 256u;
    }
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; ++r) {
        const unsigned int peers = __match_any_sync(NB_FULL_MASK, digit[r]);
        const unsigned int below = __popc(peers & ((1u << lane) - 1u));
        const bool valid = digit[r] < 256u;
        rank[r] = below + (valid ? mine[digit[r]] : 0u);
        __syncwarp();
        if (valid && below == 0) mine[digit[r]] += __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // exclusive sums over the digits (a digit a thread) of all keys' and of this tile's counts
    unsigned int count = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) count += wHist[w][t];
    unsigned int all = total, here = count;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int u = __shfl_up_sync(NB_FULL_MASK, all, o);
        const unsigned int v = __shfl_up_sync(NB_FULL_MASK, here, o);
        if (lane >= o) { all += u; here += v; }
    }
    if (lane == 31) { part[0][warp] = all; part[1][warp] = here; }
    __syncthreads();
    for (int w = 0; w < warp; ++w) { all += part[0][w]; here += part[1][w]; }
    unsigned int off = here - count;
    toGlobal[t] = all - total + before - off;
    // warp counts to each warp's start in the tile, in warp order (keeps the sort stable)
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) {
        const unsigned int c = wHist[w][t];
        wHist[w][t] = off;
        off += c;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; ++r)
        if (digit[r] < 256u) {
            const unsigned int at = mine[digit[r]] + rank[r];
            sKey[at] = key[r];
            sIdx[at] = idx[r];
            sDigit[at] = (unsigned char) digit[r];
        }
    __syncthreads();
    // the tile leaves in digit order: neighbouring threads write neighbouring keys, runs of ~8
    const int tileKeys = min(RS_TILE, n - (int) blockIdx.x * RS_TILE);
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; ++r) {
        const int at = r * RS_THREADS + t;
        if (at < tileKeys) {
            const unsigned int pos = toGlobal[sDigit[at]] + at;
            keyOut[pos] = sKey[at];
            idxOut[pos] = sIdx[at];
        }
    }
}

// ---- int inclusive scan (three phases) ----
constexpr int PS_THREADS = 1024;
constexpr int PS_ITEMS = 4;
constexpr int PS_TILE = PS_THREADS * PS_ITEMS;

__device__ __forceinline__ int block_inclusive_scan(int v, int* sh)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int u = __shfl_up_sync(NB_FULL_MASK, v, o);
        if (lane >= o) v += u;
    }
    if (lane == 31) sh[warp] = v;
    __syncthreads();
    if (warp == 0) {
        int w = lane < (blockDim.x >> 5) ? sh[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int u = __shfl_up_sync(NB_FULL_MASK, w, o);
            if (lane >= o) w += u;
        }
        sh[lane] = w;
    }
    __syncthreads();
    int r = v + (warp > 0 ? sh[warp - 1] : 0);
    __syncthreads();
    return r;
}

// Row d of the table to its exclusive prefix, its total to totals[d].
__global__ void __launch_bounds__(PS_THREADS)
k_rs_rows(unsigned int* __restrict__ hist, int nTiles, unsigned int* __restrict__ totals)
{
    __shared__ int sh[32];
    __shared__ int last;
    unsigned int* row = hist + (size_t) blockIdx.x * nTiles;
    int carry = 0;
    for (int base = 0; base < nTiles; base += blockDim.x) {
        const int i = base + threadIdx.x;
        const int v = i < nTiles ? (int) row[i] : 0;
        const int incl = block_inclusive_scan(v, sh);
        if (i < nTiles) row[i] = (unsigned int) (incl - v + carry);
        if (threadIdx.x == blockDim.x - 1) last = incl;
        __syncthreads();
        carry += last;
        __syncthreads();
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = (unsigned int) carry;
}

__global__ void __launch_bounds__(PS_THREADS)
k_ps_tile(int* __restrict__ data, int n, int* __restrict__ tileSums)
{
    __shared__ int sh[32];
    const int base = blockIdx.x * PS_TILE + threadIdx.x * PS_ITEMS;
    int v[PS_ITEMS];
    int s = 0;
#pragma unroll
    for (int k = 0; k < PS_ITEMS; ++k) {
        const int x = base + k < n ? data[base + k] : 0;
        s += x;
        v[k] = s;
    }
    int incl = block_inclusive_scan(s, sh);
    int excl = incl - s;
#pragma unroll
    for (int k = 0; k < PS_ITEMS; ++k)
        if (base + k < n) data[base + k] = v[k] + excl;
    if (threadIdx.x == blockDim.x - 1) tileSums[blockIdx.x] = incl;
}

__global__ void __launch_bounds__(PS_THREADS)
k_ps_top(int* __restrict__ tileSums, int nTiles)
{
    __shared__ int sh[32];
    int carry = 0;
    for (int base = 0; base < nTiles; base += PS_THREADS) {
        int i = base + threadIdx.x;
        int v = i < nTiles ? tileSums[i] : 0;
        int incl = block_inclusive_scan(v, sh);
        if (i < nTiles) tileSums[i] = incl - v + carry;   // exclusive
        int total = __shfl_sync(NB_FULL_MASK, incl, 31);
        __shared__ int last;
        if (threadIdx.x == PS_THREADS - 1) last = incl;
        __syncthreads();
        carry += last;
        __syncthreads();
        (void) total;
    }
}

__global__ void __launch_bounds__(PS_THREADS)
k_ps_apply(int* __restrict__ data, int n, const int* __restrict__ tileSums)
{
    const int off = tileSums[blockIdx.x];
    const int base = blockIdx.x * PS_TILE + threadIdx.x * PS_ITEMS;
#pragma unroll
    for (int k = 0; k < PS_ITEMS; ++k)
        if (base + k < n) data[base + k] += off;
}

}  // namespace

static void rs_passes(NbSortBuffers& b, int n, const int* group, cudaStream_t s)
{
    if (n <= 0) return;
    const int nTiles = (n + RS_TILE - 1) / RS_TILE;
    unsigned long long* kin = b.keyA; unsigned long long* kout = b.keyB;
    unsigned int* iin = b.idxA; unsigned int* iout = b.idxB;
    const int passes = group ? 10 : 8;
    const int rowThreads = nTiles > 512 ? 1024 : nTiles > 128 ? 512 : 128;
    for (int pass = 0; pass < passes; ++pass) {
        const bool grouped = pass >= 8;
        const int shift = grouped ? (pass - 8) * 8 : pass * 8;
        if (grouped)
            k_rs_hist<true><<<nTiles, RS_THREADS, 0, s>>>(kin, iin, group, n, shift, b.hist, nTiles);
        else
            k_rs_hist<false><<<nTiles, RS_THREADS, 0, s>>>(kin, iin, nullptr, n, shift, b.hist, nTiles);
        k_rs_rows<<<256, rowThreads, 0, s>>>(b.hist, nTiles, b.totals);
        if (grouped)
            k_rs_scatter<true><<<nTiles, RS_THREADS, 0, s>>>(kin, iin, kout, iout, group, n, shift,
                                                             b.hist, b.totals, nTiles);
        else
            k_rs_scatter<false><<<nTiles, RS_THREADS, 0, s>>>(kin, iin, kout, iout, nullptr, n,
                                                              shift, b.hist, b.totals, nTiles);
        nb_count_launch(3);
        unsigned long long* tk = kin; kin = kout; kout = tk;
        unsigned int* ti = iin; iin = iout; iout = ti;
    }
    // an even number of passes: the result is back in keyA / idxA.
}

void nb_radix_sort(NbSortBuffers& b, int n, cudaStream_t s) { rs_passes(b, n, nullptr, s); }

void nb_radix_sort_grouped(NbSortBuffers& b, int n, const int* group, cudaStream_t s)
{
    rs_passes(b, n, group, s);
}

int nb_scan_tmp_ints(int n) { return (n + PS_TILE - 1) / PS_TILE + 1; }

void nb_inclusive_scan(int* data, int n, int* tmp, cudaStream_t s)
{
    if (n <= 0) return;
    const int nTiles = (n + PS_TILE - 1) / PS_TILE;
    k_ps_tile<<<nTiles, PS_THREADS, 0, s>>>(data, n, tmp);
    k_ps_top<<<1, PS_THREADS, 0, s>>>(tmp, nTiles);
    k_ps_apply<<<nTiles, PS_THREADS, 0, s>>>(data, n, tmp);
    nb_count_launch(3);
}
