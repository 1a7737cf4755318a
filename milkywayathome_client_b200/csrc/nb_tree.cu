// Octree build on the GPU, bit-exact with the reference CPU tree (nbMakeTree,
// nbody/src/nbody_tree.c:429-460).  Compiled with -fmad=false: every floating-point
// expression below is evaluated with the reference's operation order and no FMA
// contraction, so cell centres, centres of mass, rcrit2 and quadrupole moments carry the
// same bits as the CPU's.
//
// The CPU builds its tree by top-down insertion (nbLoadBody, :242-282) from a root centred
// at the origin whose size is doubled until it covers the bodies (expandBox, :156-176).
// The resulting octree is unique: a cell exists at depth D for every octree path prefix
// that at least two massive bodies share (chains of single-child cells included), plus
// the root.  Here the same octree is derived from bodies sorted by octree path:
//   1. bounding box (max |x|,|y|,|z|) and the root size doubling of expandBox;
//   2. integer grid coordinates floor(x*2^62/rsize) + 2^61: bit (61-d) is the child
//      octant bit at depth d, i.e. exactly the CPU's `mid <= pos` test (:42-49);
//   3. sort by the top 21 levels (63-bit Morton key, radix sort) and order the rare runs
//      of equal keys by the full 62-level path;
//   4. delta_i = depth at which sorted bodies i and i+1 part; boundary i "owns" the cells
//      at depths (delta_{i-1}, delta_i], so a prefix sum of owned counts gives every
//      node its position in the walk (preorder) order of threadTree (:127-150) directly;
//   5. each cell finds the last body of its range (galloping search on the sorted grid
//      coordinates), which gives Next(); parents and child counts follow from Next();
//   6. centres of mass, rcrit2 (findRCrit, :308-343) and quadrupoles (hackQuad, :70-121)
//      bottom-up: the last child to finish (atomic arrival counter) computes its parent,
//      reading the children in octant order as hackCofM does (:386-424).  No thread ever
//      waits on another.
// Steps 1 to 5 are one launch a phase here, over the whole GPU; small systems take them in one
// launch (nb_build.cu).
#include "nb_common.cuh"
#include "nb_tree_phase.cuh"

// ---------------------------------------------------------------------------------
// 1. bounding box (optionally fused with the first half of the leapfrog step)
// ---------------------------------------------------------------------------------
__global__ void k_drift_bbox(NbTreeBuffers b, int n, int drift, double dt, double sx, double sy,
                             double sz, NbScalars* __restrict__ sc)
{
    double m = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        m = fmax(m, nb_phase_drift(b, i, drift, dt, sx, sy, sz));
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(NB_FULL_MASK, m, o));
    __shared__ double wm[32];
    if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < (blockDim.x >> 5) ? wm[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(NB_FULL_MASK, m, o));
        // non-negative doubles order like their bit patterns
        if (threadIdx.x == 0) atomicMax(&sc->xyzmaxBits, (unsigned long long) __double_as_longlong(m));
    }
}

// expandBox's doubling and the grid constants derived from rsize.
__global__ void k_root_size(NbScalars* sc)
{
    if (nb_failed(sc)) return;
    const double rsize = nb_phase_root_size(sc->rsize, __longlong_as_double((long long) sc->xyzmaxBits));
    sc->rsize = rsize;
    if (!isfinite(rsize)) { nb_raise(sc, NBODY_TREE_STRUCTURE_ERROR); return; }
    nb_phase_grid_constants(rsize, sc->gridScale, sc->depthEps);
}

// ---------------------------------------------------------------------------------
// 2. keys
// ---------------------------------------------------------------------------------
__global__ void k_keys(NbTreeBuffers b, int n, NbScalars* __restrict__ sc)
{
    if (nb_failed(sc)) return;
    const double scale = sc->gridScale;
    int cnt = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        unsigned long long k;
        cnt += nb_phase_key(b, i, scale, k);
        b.sort.keyA[i] = k;
        b.sort.idxA[i] = (unsigned) i;
    }
    // one atomic a block: they all go to one word, a few ns each
    __shared__ int blockCount;
    if (threadIdx.x == 0) blockCount = 0;
    __syncthreads();
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(NB_FULL_MASK, cnt, o);
    if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(&blockCount, cnt);
    __syncthreads();
    if (threadIdx.x == 0 && blockCount) atomicAdd(&sc->nTree, blockCount);
}

// Grid coordinates of the sorted bodies.
__global__ void k_gather_grid(NbTreeBuffers b, NbScalars* __restrict__ sc)
{
    if (nb_failed(sc)) return;
    const int m = sc->nTree;
    const double scale = sc->gridScale;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x)
        nb_phase_gather(b, i, scale);
}

__global__ void k_fix_runs(NbTreeBuffers b, NbScalars* __restrict__ sc)
{
    if (nb_failed(sc)) return;
    const int m = sc->nTree;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i + 1 < m; i += gridDim.x * blockDim.x)
        nb_phase_fix_run(b, i, m);
}

// ---------------------------------------------------------------------------------
// 4. parting depths and owned-cell counts
// ---------------------------------------------------------------------------------
// delta[i] for boundary i in [0, m-2]; cum[i] = cells owned by boundary i.
__global__ void k_delta(NbTreeBuffers b, int n, NbScalars* __restrict__ sc)
{
    if (nb_failed(sc)) return;
    const int m = sc->nTree;
    const int depthEps = sc->depthEps;
    bool bad = false;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i + 1 < n; i += gridDim.x * blockDim.x)
        b.cum[i] = nb_phase_delta(b, i, m, depthEps, bad);
    if (bad) nb_raise(sc, NBODY_TREE_STRUCTURE_ERROR);
}

// Total node count; checks the capacity.
__global__ void k_count_nodes(const int* __restrict__ cum, NbScalars* __restrict__ sc)
{
    if (nb_failed(sc)) return;
    const int m = sc->nTree;
    const int cells = m <= 1 ? 1 : cum[m - 2];
    sc->nCells = cells;
    sc->nNodes = m + cells;
    sc->neededNodes = m + cells;
    sc->maxDepth = 0;
    if (m + cells > sc->capNodes) nb_raise(sc, NBODY_CELL_OVERFLOW_ERROR);
}

// ---------------------------------------------------------------------------------
// 5. node emission in walk order
// ---------------------------------------------------------------------------------
__global__ void k_emit_bodies(NbTreeBuffers b, NbScalars* __restrict__ sc)
{
    if (nb_failed(sc)) return;
    const int m = sc->nTree;
    int maxLev = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x)
        maxLev = max(maxLev, nb_phase_emit_body(b, i, m));
    for (int o = 16; o > 0; o >>= 1) maxLev = max(maxLev, __shfl_xor_sync(NB_FULL_MASK, maxLev, o));
    nb_raise_max(&sc->maxDepth, maxLev);
}

__global__ void k_emit_cells(NbTreeBuffers b, int criterion, double theta, NbScalars* __restrict__ sc)
{
    if (nb_failed(sc)) return;
    const int m = sc->nTree;
    const double rsize = sc->rsize;
    const int nb = m <= 1 ? 1 : m - 1;        // boundaries (the root-only tree uses one slot)
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < nb; a += gridDim.x * blockDim.x)
        nb_phase_emit_cells(b, a, m, rsize, criterion, theta);
}

// Parent pointers and child lists from Next().
__global__ void k_link_children(NbTreeBuffers b, NbScalars* __restrict__ sc)
{
    if (nb_failed(sc)) return;
    const int nNodes = sc->nNodes;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < nNodes; c += gridDim.x * blockDim.x)
        nb_phase_link(b, c);
}

// ---------------------------------------------------------------------------------
// 6. moments, bottom-up
// ---------------------------------------------------------------------------------
// One thread per cell, from the cells without child cells up (nb_bottom_up).
__global__ void __launch_bounds__(128, 4)
k_moments(double4* nodePM, double* nodeCrit, const int2* nodeLink, const int* nodeDepth,
          const int2* nodeRange, double* nodeQuad, const int* __restrict__ parent, int* pending,
          const int* __restrict__ cellNode, const int4* kids, int criterion, double theta,
          int useQuad, NbScalars* sc)
{
    if (nb_failed(sc)) return;
    const int nCells = sc->nCells;
    const double rsize = sc->rsize;
    int structErr = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nCells; i += gridDim.x * blockDim.x)
        nb_bottom_up(i, cellNode, parent, pending, [&](int c) {
            structErr |= nb_cell_moments(c, nodePM, nodeCrit, nodeLink, nodeDepth, nodeRange,
                                         nodeQuad, kids, rsize, criterion, theta, useQuad);
        });
    if (structErr) nb_raise(sc, NBODY_TREE_STRUCTURE_ERROR);
}

// Eight lanes per cell (nb_moments_up).
__global__ void __launch_bounds__(NB_MOM_WARPS * 32)
k_moments_team(double4* nodePM, double* nodeCrit, const int2* nodeLink, const int* nodeDepth,
          const int2* nodeRange, double* nodeQuad, const int* parent, int* pending,
          const int* cellNode, const int4* kids, int criterion, double theta, int useQuad,
          NbScalars* sc)
{
    if (__any_sync(0xffffffffu, nb_failed(sc))) return;     // the lanes of a warp alike
    const double rsize = sc->rsize;
    bool structErr = false;
    nb_moments_up(sc->nCells, nodePM, nodeCrit, nodeLink, nodeDepth, nodeRange, nodeQuad, parent,
                  pending, cellNode, kids, criterion, theta, useQuad, [&](int) { return rsize; },
                  [&](int) { structErr = true; });
    if (structErr) nb_raise(sc, NBODY_TREE_STRUCTURE_ERROR);
}

// ---------------------------------------------------------------------------------
// host driver
// ---------------------------------------------------------------------------------


static inline int nb_grid_for(int n, int threads, int cap)
{
    int g = (n + threads - 1) / threads;
    if (g < 1) g = 1;
    return g < cap ? g : cap;
}

// Steps 1 to 5, a launch a phase.
static void nb_launch_build_phases(NbTreeBuffers& b, int n, int capNodes, int criterion, double theta,
                                   int drift, double dt, int numSMs, cudaStream_t s,
                                   const double* shift)
{
    const double sx = shift ? shift[0] : 0.0, sy = shift ? shift[1] : 0.0;
    const double sz = shift ? shift[2] : 0.0;
    const int T = 256;
    const int gCap = numSMs * 8;
    k_drift_bbox<<<nb_grid_for(n, T, gCap), T, 0, s>>>(b, n, drift, dt, sx, sy, sz, b.sc);
    k_root_size<<<1, 1, 0, s>>>(b.sc);
    k_keys<<<nb_grid_for(n, T, gCap), T, 0, s>>>(b, n, b.sc);
    nb_count_launch(3);
    nb_radix_sort(b.sort, n, s);
    const int g = nb_grid_for(n, T, 1 << 20);
    k_gather_grid<<<g, T, 0, s>>>(b, b.sc);
    k_fix_runs<<<g, T, 0, s>>>(b, b.sc);
    k_delta<<<g, T, 0, s>>>(b, n, b.sc);
    nb_count_launch(3);
    // cum = inclusive prefix sum of owned-cell counts over boundaries [0, n-2] (the kernels
    // only read the first m-1 entries; entries past m-2 hold stale counts and are unused)
    if (n > 1) nb_inclusive_scan(b.cum, n - 1, b.scanTmp, s);
    k_count_nodes<<<1, 1, 0, s>>>(b.cum, b.sc);
    k_emit_bodies<<<g, T, 0, s>>>(b, b.sc);
    k_emit_cells<<<g, T, 0, s>>>(b, criterion, theta, b.sc);
    k_link_children<<<nb_grid_for(capNodes, T, 1 << 20), T, 0, s>>>(b, b.sc);
    nb_count_launch(4);
}

// Kernel sequence of nbMakeTree.  drift != 0 fuses advancePosVel into the bounding box.  The
// scalars come with zero counters.
void nb_build_tree(NbTreeBuffers& b, int n, int capNodes, int criterion, double theta, int useQuad,
                   int drift, double dt, int numSMs, cudaStream_t s, const double* shift)
{
    if (nb_build_in_cluster(n)) nb_launch_build_cluster(b, n, criterion, theta, drift, dt, shift, s);
    else nb_launch_build_phases(b, n, capNodes, criterion, theta, drift, dt, numSMs, s, shift);
    // a cell parts at least two bodies (or is the root), but chains of single-child cells make
    // more of them than bodies now and then: the loop takes any number
    if (nb_moments_team(n))
        k_moments_team<<<nb_grid_for(n, NB_MOM_WARPS * 4, 1 << 20), NB_MOM_WARPS * 32, 0, s>>>(
            b.nodePM, b.nodeCrit, b.nodeLink, b.nodeDepth, b.nodeRange, b.nodeQuad, b.parent,
            b.pending, b.cellNode, b.walkKids, criterion, theta, useQuad, b.sc);
    else
        k_moments<<<nb_grid_for(n, 128, 1 << 20), 128, 0, s>>>(
            b.nodePM, b.nodeCrit, b.nodeLink, b.nodeDepth, b.nodeRange, b.nodeQuad, b.parent,
            b.pending, b.cellNode, b.walkKids, criterion, theta, useQuad, b.sc);
    nb_count_launch();
}

void nb_launch_drift_only(NbTreeBuffers& b, int n, double dt, int numSMs, cudaStream_t s,
                          const double* shift)
{
    const int T = 256;
    const double sx = shift ? shift[0] : 0.0, sy = shift ? shift[1] : 0.0;
    const double sz = shift ? shift[2] : 0.0;
    k_drift_bbox<<<nb_grid_for(n, T, numSMs * 8), T, 0, s>>>(b, n, 1, dt, sx, sy, sz, b.sc);
    nb_count_launch();
}
