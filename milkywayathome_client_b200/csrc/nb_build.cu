// The whole octree build of a small system in one launch: one cluster of eight blocks.
//
// The phases are those of nb_tree.cu (nb_tree_phase.cuh), one hardware cluster barrier apart
// instead of one launch: drift and bounding box, root size and keys, the eight passes of a
// stable radix sort, grid coordinates, equal-key runs, parting depths and their prefix sum, node
// emission, links.  What bounds the launched sequence at these sizes is not work but launches,
// 49 of them at some 4 us each in a replayed graph; here a phase costs its own L2 round trips and
// a barrier (well under a microsecond).  The cluster holds 8,192 threads, four bodies a thread at
// the most, so the whole GPU's launched phases win above CLUSTER_MAX_BODIES.
// A step without its walk, launched -> here: 1,024 bodies 0.164 -> 0.112 ms, 5,000 0.221 -> 0.131,
// 12,000 0.239 -> 0.172, 20,000 0.244 -> 0.209, 32,768 0.258 -> 0.257: the line is there.
// Compiled with -fmad=false like nb_tree.cu.
#include "nb_common.cuh"
#include "nb_tree_phase.cuh"
#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace {

constexpr int CB_CTAS = 8;
constexpr int CB_THREADS = 1024;
constexpr int CB_WARPS = CB_THREADS / 32;
constexpr int CB_ITEMS = 4;                                   // a thread's keys in the sort
constexpr int CLUSTER_MAX_BODIES = CB_CTAS * CB_THREADS * CB_ITEMS;

struct CbShared {
    unsigned hist[2][256];              // this block's digit counts, read by the whole cluster
    unsigned run[256];                  // next position of each digit
    unsigned wHist[CB_WARPS][256];      // per warp counts, then positions
    unsigned part[CB_WARPS];
    double wmax[CB_WARPS];
    int total;                          // this block's owned cells, read by the whole cluster
};

// Inclusive sum over the block (every thread calls it).
__device__ __forceinline__ unsigned cb_scan(unsigned v, unsigned* part)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned u = __shfl_up_sync(NB_FULL_MASK, v, o);
        if (lane >= o) v += u;
    }
    if (lane == 31) part[warp] = v;
    __syncthreads();
    unsigned before = 0;
    for (int w = 0; w < warp; ++w) before += part[w];
    __syncthreads();
    return v + before;
}

__global__ void __cluster_dims__(CB_CTAS, 1, 1) __launch_bounds__(CB_THREADS, 1)
k_build_cluster(NbTreeBuffers b, int n, int criterion, double theta, int drift, double dt, double sx,
                double sy, double sz)
{
    __shared__ CbShared S;
    const cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int) cluster.block_rank();
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int tid = rank * CB_THREADS + t;
    constexpr int STRIDE = CB_CTAS * CB_THREADS;
    NbScalars* const sc = b.sc;
    const double rsize0 = sc->rsize;

    // ---- drift, bounding box ----
    double top = 0.0;
    for (int i = tid; i < n; i += STRIDE) top = fmax(top, nb_phase_drift(b, i, drift, dt, sx, sy, sz));
    for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(NB_FULL_MASK, top, o));
    if (lane == 0) S.wmax[warp] = top;
    __syncthreads();
    if (warp == 0) {
        top = S.wmax[lane];
        for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(NB_FULL_MASK, top, o));
        // non-negative doubles order like their bit patterns
        if (lane == 0) atomicMax(&sc->xyzmaxBits, (unsigned long long) __double_as_longlong(top));
    }
    cluster.sync();

    // ---- root size and keys: item r of thread t in this block's run of consecutive bodies ----
    const double rsize = nb_phase_root_size(rsize0, __longlong_as_double((long long) __ldcg(&sc->xyzmaxBits)));
    double scale = 0.0;
    int depthEps = 0;
    if (isfinite(rsize)) nb_phase_grid_constants(rsize, scale, depthEps);
    if (tid == 0) {
        sc->rsize = rsize;
        sc->gridScale = scale;
        sc->depthEps = depthEps;
        if (!isfinite(rsize)) nb_raise(sc, NBODY_TREE_STRUCTURE_ERROR);
    }
    if (!isfinite(rsize)) return;                     // every thread alike
    const int per = (n + CB_CTAS - 1) / CB_CTAS;
    const int lo = rank * per, hi = min(n, lo + per);
    unsigned long long key[CB_ITEMS];
    unsigned idx[CB_ITEMS];
    unsigned massive = 0;
#pragma unroll
    for (int r = 0; r < CB_ITEMS; ++r) {
        const int i = lo + r * CB_THREADS + t;
        key[r] = 0ull;
        idx[r] = (unsigned) i;
        if (i < hi) massive += nb_phase_key(b, i, scale, key[r]);
    }
    massive = __reduce_add_sync(NB_FULL_MASK, massive);
    if (lane == 0 && massive) atomicAdd(&sc->nTree, (int) massive);

    // ---- stable radix sort, 8 passes of 8 bits ----
    unsigned long long *kin = b.sort.keyA, *kout = b.sort.keyB;
    unsigned *iin = b.sort.idxA, *iout = b.sort.idxB;
    for (int pass = 0; pass < 8; ++pass) {
        const int shift = 8 * pass;
        unsigned* hist = S.hist[pass & 1];
        if (t < 256) hist[t] = 0;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < CB_ITEMS; ++r) {
            const int i = lo + r * CB_THREADS + t;
            if (i >= hi) continue;
            if (pass > 0) { key[r] = kin[i]; idx[r] = iin[i]; }
            atomicAdd(&hist[(unsigned) (key[r] >> shift) & 255u], 1u);
        }
        cluster.sync();
        unsigned below = 0, total = 0;
        if (t < 256) {
#pragma unroll
            for (int q = 0; q < CB_CTAS; ++q) {
                const unsigned v = *cluster.map_shared_rank(&hist[t], q);
                total += v;
                if (q < rank) below += v;
            }
        }
        const unsigned upTo = cb_scan(total, S.part);
        if (t < 256) S.run[t] = upTo - total + below;
#pragma unroll
        for (int r = 0; r < CB_ITEMS; ++r) {
            if (lo + r * CB_THREADS >= hi) break;     // the whole block
            __syncthreads();                          // wHist of the round before is done with
#pragma unroll
            for (int q = 0; q < 256 * CB_WARPS / CB_THREADS; ++q)
                (&S.wHist[0][0])[q * CB_THREADS + t] = 0;
            __syncthreads();
            const bool valid = lo + r * CB_THREADS + t < hi;
            const unsigned d = valid ? (unsigned) (key[r] >> shift) & 255u : 256u;
            const unsigned peers = __match_any_sync(NB_FULL_MASK, d);
            const unsigned rankInWarp = __popc(peers & ((1u << lane) - 1u));
            if (valid && rankInWarp == 0) S.wHist[warp][d] = __popc(peers);
            __syncthreads();
            if (t < 256) {          // warp counts to positions, in warp order (keeps it stable)
                unsigned off = S.run[t];
#pragma unroll
                for (int q = 0; q < CB_WARPS; ++q) {
                    const unsigned c = S.wHist[q][t];
                    S.wHist[q][t] = off;
                    off += c;
                }
                S.run[t] = off;
            }
            __syncthreads();
            if (valid) {
                const unsigned at = S.wHist[warp][d] + rankInWarp;
                kout[at] = key[r];
                iout[at] = idx[r];
            }
        }
        cluster.sync();
        unsigned long long* tk = kin; kin = kout; kout = tk;
        unsigned* ti = iin; iin = iout; iout = ti;
    }

    // ---- sorted grid coordinates, equal-key runs, parting depths ----
    const int m = __ldcg(&sc->nTree);
    for (int i = tid; i < m; i += STRIDE) nb_phase_gather(b, i, scale);
    cluster.sync();
    for (int i = tid; i + 1 < m; i += STRIDE) nb_phase_fix_run(b, i, m);
    cluster.sync();
    bool bad = false;
    int cum[CB_ITEMS];
    unsigned carry = 0;
#pragma unroll
    for (int r = 0; r < CB_ITEMS; ++r) {              // block-local inclusive sums of owned cells
        cum[r] = 0;
        if (lo + r * CB_THREADS >= hi) break;         // the whole block
        const int i = lo + r * CB_THREADS + t;
        const unsigned owned = i < hi ? (unsigned) nb_phase_delta(b, i, m, depthEps, bad) : 0u;
        const unsigned s = cb_scan(owned, S.part);
        cum[r] = (int) (carry + s);
        if (t == CB_THREADS - 1) S.total = (int) (carry + s);
        __syncthreads();
        carry = (unsigned) S.total;
        __syncthreads();
    }
    if (t == 0) S.total = (int) carry;
    if (bad) nb_raise(sc, NBODY_TREE_STRUCTURE_ERROR);
    cluster.sync();
    int before = 0;
    for (int q = 0; q < rank; ++q) before += *cluster.map_shared_rank(&S.total, q);
#pragma unroll
    for (int r = 0; r < CB_ITEMS; ++r) {
        const int i = lo + r * CB_THREADS + t;
        if (i < hi) b.cum[i] = before + cum[r];
    }
    cluster.sync();
    if (nb_failed(sc)) return;                        // raised before the barrier: every thread alike

    // ---- nodes ----
    const int cells = m <= 1 ? 1 : __ldcg(&b.cum[m - 2]);
    if (tid == 0) {
        sc->nCells = cells;
        sc->nNodes = m + cells;
        sc->neededNodes = m + cells;
    }
    if (m + cells > sc->capNodes) {
        if (tid == 0) nb_raise(sc, NBODY_CELL_OVERFLOW_ERROR);
        return;
    }
    int maxLev = 0;
    for (int i = tid; i < m; i += STRIDE) maxLev = max(maxLev, nb_phase_emit_body(b, i, m));
    maxLev = __reduce_max_sync(NB_FULL_MASK, maxLev);
    if (lane == 0 && maxLev) atomicMax(&sc->maxDepth, maxLev);
    const int bounds = m <= 1 ? 1 : m - 1;            // the root-only tree uses one slot
    for (int a = tid; a < bounds; a += STRIDE) nb_phase_emit_cells(b, a, m, rsize, criterion, theta);
    cluster.sync();
    for (int c = tid; c < m + cells; c += STRIDE) nb_phase_link(b, c);
}

}  // namespace

bool nb_build_in_cluster(int n) { return n >= 1 && n <= CLUSTER_MAX_BODIES; }

// Everything of nb_build_tree but the moments.  The scalars' counters must be zero.
void nb_launch_build_cluster(const NbTreeBuffers& b, int n, int criterion, double theta, int drift,
                             double dt, const double* shift, cudaStream_t s)
{
    const double sx = shift ? shift[0] : 0.0, sy = shift ? shift[1] : 0.0;
    const double sz = shift ? shift[2] : 0.0;
    k_build_cluster<<<CB_CTAS, CB_THREADS, 0, s>>>(b, n, criterion, theta, drift, dt, sx, sy, sz);
    nb_count_launch();
}
