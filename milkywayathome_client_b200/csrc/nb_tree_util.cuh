// Device helpers of the octree build shared by the single-tree build (nb_tree.cu) and the
// batched forest build (nb_batch.cu).  Included only by translation units compiled with
// -fmad=false: the floating-point expressions keep the reference's rounding.  Bare line
// citations (:N) refer to nbody/src/nbody_tree.c.
#pragma once
#include "nb_common.cuh"

// max into a word that every warp updates (v the warp's own maximum): most warps see that it is
// there already and leave out the atomic, of which one a warp, all to one word, took most of the
// node emission of a million bodies (91 -> 45 us).
__device__ __forceinline__ void nb_raise_max(int* word, int v)
{
    if ((threadIdx.x & 31) == 0 && v > *(volatile const int*) word) atomicMax(word, v);
}

__device__ __forceinline__ long long nb_grid(double x, double scale)
{
    // CPU: a NaN coordinate fails every `mid <= pos`, i.e. it always takes the lower child.
    if (isnan(x)) return 0;
    double f = floor(x * scale);
    long long k = (long long) f + (1ll << (NB_GRID_LEVELS - 1));
    if (k < 0) k = 0;
    if (k > (1ll << NB_GRID_LEVELS) - 1) k = (1ll << NB_GRID_LEVELS) - 1;
    return k;
}

__device__ __forceinline__ unsigned long long nb_spread21(unsigned long long v)
{
    v &= 0x1fffffull;
    v = (v | (v << 32)) & 0x1f00000000ffffull;
    v = (v | (v << 16)) & 0x1f0000ff0000ffull;
    v = (v | (v << 8)) & 0x100f00f00f00f00full;
    v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
    v = (v | (v << 2)) & 0x1249249249249249ull;
    return v;
}

// x is the most significant bit of each octant triplet: the child index of nbSubIndex
// is 4*[x] + 2*[y] + [z] (:36-52), so key order is the CPU's child order at every level.
__device__ __forceinline__ unsigned long long nb_morton63(long long kx, long long ky, long long kz)
{
    const int sh = NB_GRID_LEVELS - NB_KEY_LEVELS;
    return (nb_spread21((unsigned long long) kx >> sh) << 2) |
           (nb_spread21((unsigned long long) ky >> sh) << 1) |
            nb_spread21((unsigned long long) kz >> sh);
}

// Morton order of two full 62-level paths: the first differing level decides, and within
// it x outranks y outranks z (child index 4x+2y+z).
__device__ __forceinline__ bool nb_path_less(long long ax, long long ay, long long az,
                                             long long bx, long long by, long long bz)
{
    const unsigned long long dx = (unsigned long long) (ax ^ bx);
    const unsigned long long dy = (unsigned long long) (ay ^ by);
    const unsigned long long dz = (unsigned long long) (az ^ bz);
    const int hx = dx ? 63 - __clzll(dx) : -1;
    const int hy = dy ? 63 - __clzll(dy) : -1;
    const int hz = dz ? 63 - __clzll(dz) : -1;
    if (hx < 0 && hy < 0 && hz < 0) return false;
    if (hx >= hy && hx >= hz) return ax < bx;
    if (hy >= hz) return ay < by;
    return az < bz;
}

__device__ __forceinline__ int nb_part_depth(long long ax, long long ay, long long az,
                                             long long bx, long long by, long long bz)
{
    unsigned long long d = (unsigned long long) ((ax ^ bx) | (ay ^ by) | (az ^ bz));
    if (d == 0) return NB_GRID_LEVELS;            // same point on the grid
    return (NB_GRID_LEVELS - 1) - (63 - __clzll(d));
}

// Last sorted body sharing the depth-D path prefix of body a (bodies of one cell are
// contiguous in path order): galloping then binary search, every probe a dependent load, so one
// 8-byte key decides it down to the key's depth (the three grid coordinates below it): the
// emission of 1,048,576 bodies' cells went from 114 to 66 us.
template <typename Same>
__device__ __forceinline__ int nb_gallop(int a, int m, Same same)
{
    int lo = a, step = 1;
    while (lo + step < m && same(lo + step)) {
        lo += step;
        step <<= 1;
    }
    int hi = min(lo + step, m);          // first index known (or assumed) outside
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (same(mid)) lo = mid;
        else hi = mid;
    }
    return lo;
}

__device__ inline int nb_range_end(const unsigned long long* key, const long long* gx,
                                   const long long* gy, const long long* gz, int a, int D, int m)
{
    if (D == 0) return m - 1;
    if (D <= NB_KEY_LEVELS) {
        const int s = 3 * (NB_KEY_LEVELS - D);
        const unsigned long long want = key[a] >> s;
        return nb_gallop(a, m, [&](int i) { return key[i] >> s == want; });
    }
    const int s = NB_GRID_LEVELS - D;
    const long long ax = gx[a] >> s, ay = gy[a] >> s, az = gz[a] >> s;
    return nb_gallop(a, m, [&](int i) {
        return (gx[i] >> s) == ax && (gy[i] >> s) == ay && (gz[i] >> s) == az;
    });
}

// findRCrit (:308-343) from the cell's geometric centre, CoM and size.
__device__ __forceinline__ double nb_find_rcrit2(int criterion, double theta, double rsize,
                                                 double cx, double cy, double cz,
                                                 double mx, double my, double mz, double psize)
{
    if (theta == 0.0) {
        const double rc = 2.0 * rsize;
        return rc * rc;
    }
    switch (criterion) {
    case NBCUDA_TREECODE: {
        const double dx = mx - cx, dy = my - cy, dz = mz - cz;
        const double rc = psize / theta + sqrt(dx * dx + dy * dy + dz * dz);
        return rc * rc;
    }
    case NBCUDA_SW93: {
        double dmin, b, bmax2;
        dmin = mx - (cx - 0.5 * psize); b = fmax(dmin, psize - dmin); bmax2 = b * b;
        dmin = my - (cy - 0.5 * psize); b = fmax(dmin, psize - dmin); bmax2 += b * b;
        dmin = mz - (cz - 0.5 * psize); b = fmax(dmin, psize - dmin); bmax2 += b * b;
        return bmax2 / (theta * theta);
    }
    case NBCUDA_BH86: {
        const double rc = psize / theta;
        return rc * rc;
    }
    default:
        return 0.0;
    }
}

// L2 loads (bypass L1: cells computed by other blocks in this kernel must not be read
// from a stale L1 line)
__device__ __forceinline__ double4 nb_ld_pm(const double4* p)
{
    const double2* q = reinterpret_cast<const double2*>(p);
    const double2 a = __ldcg(q), b = __ldcg(q + 1);
    return make_double4(a.x, a.y, b.x, b.y);
}

// A cell's children in octant order, from its slot's two int4 (-1 past the last).  L2 loads: a list is
// read once, and the records it leads to are L2 loads anyway.
__device__ __forceinline__ void nb_load_kids(const int4* kids, int slot, int (&k)[8])
{
    const int4 a = __ldcg(kids + 2 * (size_t) slot), b = __ldcg(kids + 2 * (size_t) slot + 1);
    k[0] = a.x; k[1] = a.y; k[2] = a.z; k[3] = a.w;
    k[4] = b.x; k[5] = b.y; k[6] = b.z; k[7] = b.w;
}

// Parent links and child list of cell c: children are c + 1, then Next() up to Next(c).  The list
// is stored densely by slot, the cell's number among the cells: its node number less the sorted
// bodies before it (the first body of its range).  pending: the child cells its moments wait for;
// cellNode: the slot's node, complemented where there are any.
__device__ __forceinline__ void nb_link_cell(int c, int2 link, int slot, const int2* nodeLink,
                                             int* parent, int* pending, int* cellNode, int4* kids)
{
    int ch[8] = {-1, -1, -1, -1, -1, -1, -1, -1};
    int k = c + 1, cells = 0;
#pragma unroll
    for (int m = 0; m < 8; ++m)
        if (k < link.x) {
            const int2 l = nodeLink[k];
            ch[m] = k;
            if (l.y < 0) { parent[k] = c; ++cells; }
            k = l.x;
        }
    kids[2 * (size_t) slot] = make_int4(ch[0], ch[1], ch[2], ch[3]);
    kids[2 * (size_t) slot + 1] = make_int4(ch[4], ch[5], ch[6], ch[7]);
    pending[c] = cells;
    cellNode[slot] = cells ? ~c : c;
}

// Moments of cell c whose children are complete: hackCofM (:394-424), findRCrit, the structure
// check (:345-380) and hackQuad (:70-121), children added in octant order.  Returns whether the
// centre of mass left the cell.  A cell is one thread's work and its parent waits for it, so the
// pass is a chain of L2 latencies, tree level by tree level: the child list lets every child's
// records be fetched at once (a few round trips a cell where following Next() took up to 16).
__device__ __forceinline__ bool nb_cell_moments(int c, double4* nodePM, double* nodeCrit,
                                                const int2* nodeLink, const int* nodeDepth,
                                                const int2* nodeRange, double* nodeQuad,
                                                const int4* kids, double rsize, int criterion,
                                                double theta, int useQuad)
{
    const double4 geo = nb_ld_pm(&nodePM[c]);
    const int D = __ldcg(&nodeDepth[c]);
    int k[8];
    nb_load_kids(kids, c - __ldcg(&nodeRange[c].x), k);
    double4 q[8];
    bool cell[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        q[m] = make_double4(0.0, 0.0, 0.0, 0.0);
        cell[m] = false;
        if (k[m] >= 0) {
            q[m] = nb_ld_pm(&nodePM[k[m]]);
            cell[m] = __ldcg(&nodeLink[k[m]].y) < 0;
        }
    }
    double M = 0.0, cmx = 0.0, cmy = 0.0, cmz = 0.0;
#pragma unroll
    for (int m = 0; m < 8; ++m)
        if (k[m] >= 0) {
            M = M + q[m].w;
            cmx = cmx + q[m].w * q[m].x;
            cmy = cmy + q[m].w * q[m].y;
            cmz = cmz + q[m].w * q[m].z;
        }
    if (M > 0.0) { cmx = cmx / M; cmy = cmy / M; cmz = cmz / M; }
    else { cmx = geo.x; cmy = geo.y; cmz = geo.z; }
    const double psize = ldexp(rsize, -D);      // rsize halved D times: exact
    const double h = 0.5 * psize;
    const bool outside = cmx < geo.x - h || cmx > geo.x + h || cmy < geo.y - h ||
                         cmy > geo.y + h || cmz < geo.z - h || cmz > geo.z + h;
    nodeCrit[c] = nb_find_rcrit2(criterion, theta, rsize, geo.x, geo.y, geo.z, cmx, cmy, cmz, psize);
    double2* Q = reinterpret_cast<double2*>(nodeQuad + 6 * (size_t) c);
    double qxx = 0.0, qxy = 0.0, qxz = 0.0, qyy = 0.0, qyz = 0.0, qzz = 0.0;
    if (useQuad) {                              // else the record reads as zero
#pragma unroll
        for (int half = 0; half < 8; half += 2) {
            double2 A[2], B[2], C[2];
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                A[m] = B[m] = C[m] = make_double2(0.0, 0.0);
                if (cell[half + m]) {
                    const double2* kq = reinterpret_cast<const double2*>(nodeQuad + 6 * (size_t) k[half + m]);
                    A[m] = __ldcg(kq); B[m] = __ldcg(kq + 1); C[m] = __ldcg(kq + 2);
                }
            }
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                if (k[half + m] < 0) continue;
                const double4 p = q[half + m];
                const double dx = p.x - cmx, dy = p.y - cmy, dz = p.z - cmz;
                const double drsq = dz * dz + (dy * dy + dx * dx);
                const double mq = p.w;
                double txx = mq * (3.0 * (dx * dx) - drsq);
                double txy = mq * (3.0 * (dx * dy));
                double txz = mq * (3.0 * (dx * dz));
                double tyy = mq * (3.0 * (dy * dy) - drsq);
                double tyz = mq * (3.0 * (dy * dz));
                double tzz = mq * (3.0 * (dz * dz) - drsq);
                if (cell[half + m]) {
                    txx = txx + A[m].x; txy = txy + A[m].y; txz = txz + B[m].x;
                    tyy = tyy + B[m].y; tyz = tyz + C[m].x; tzz = tzz + C[m].y;
                }
                qxx = qxx + txx; qxy = qxy + txy; qxz = qxz + txz;
                qyy = qyy + tyy; qyz = qyz + tyz; qzz = qzz + tzz;
            }
        }
    }
    Q[0] = make_double2(qxx, qxy); Q[1] = make_double2(qxz, qyy); Q[2] = make_double2(qyz, qzz);
    nodePM[c] = make_double4(cmx, cmy, cmz, M);
    return outside;
}

// The cells that wait for no other cell start; each goes on to its parent when it was the last
// child cell the parent waited for (no thread ever waits).  visit(c) computes cell c.
// (Started from the bodies, every body's arrival was an atomic of its own: with that and the Next()
// chains the pass took 420 us at 1,048,576 bodies and 149 at 20,000; now 270 and 80.)
template <typename Visit>
__device__ __forceinline__ void nb_bottom_up(int slot, const int* cellNode, const int* parent,
                                             int* pending, Visit visit)
{
    int c = cellNode[slot];
    if (c < 0) return;                  // (not by `pending`, which falls while the cells run)
    for (;;) {
        visit(c);
        c = parent[c];
        if (c < 0) return;
        __threadfence();
        if (atomicSub(&pending[c], 1) != 1) return;
        __threadfence();
    }
}

// The same pass (nb_bottom_up over nb_cell_moments, the same operations in the same order) with
// eight lanes a cell, where a chip that is not full waits for the chain of levels: each lane fetches
// a child and computes its terms, and lane q adds quantity q of all eight through shared memory;
// what is known of the parent (its children, centre and depth) is fetched meanwhile.  The four
// cells of a warp go in step.  rsizeOf(first body) gives the root size of a start's tree,
// outsideOf(first body) hears that a centre of mass left its cell.
// The step outside the walk, a thread a cell -> eight lanes: 256 bodies 0.099 -> 0.075 ms, 1,024
// 0.112 -> 0.093, 5,000 0.131 -> 0.108, 20,000 0.209 -> 0.184, 65,536 0.217 -> 0.202, 100,000
// 0.230 -> 0.226; 262,144 0.306 -> 0.338, 1,048,576 0.689 -> 0.956, where issue slots are short and
// most teams of a warp idle while one climbs: hence the line.
constexpr int NB_MOM_WARPS = 4;
constexpr int NB_MOM_TEAM_MAX = 100000;
static inline bool nb_moments_team(int n) { return n <= NB_MOM_TEAM_MAX; }

template <typename RsizeOf, typename OutsideOf>
__device__ __forceinline__ void nb_moments_up(int nCells, double4* nodePM, double* nodeCrit,
                                              const int2* __restrict__ nodeLink,
                                              const int* __restrict__ nodeDepth,
                                              const int2* __restrict__ nodeRange, double* nodeQuad,
                                              const int* __restrict__ parent, int* pending,
                                              const int* __restrict__ cellNode,
                                              const int4* __restrict__ kids, int criterion,
                                              double theta, int useQuad, RsizeOf rsizeOf,
                                              OutsideOf outsideOf)
{
    const unsigned FULL = 0xffffffffu;
    __shared__ __align__(16) double terms[NB_MOM_WARPS][4][6 * 8 + 8];  // + 8: teams in other banks
    const int warp = threadIdx.x >> 5, team = (threadIdx.x & 31) >> 3, sub = threadIdx.x & 7;
    double* const T = terms[warp][team];
    const int* const kid8 = reinterpret_cast<const int*>(kids);
    for (int base = (blockIdx.x * NB_MOM_WARPS + warp) * 4; base < nCells;
         base += gridDim.x * NB_MOM_WARPS * 4) {
        const int slot = base + team;
        int c = slot < nCells ? cellNode[slot] : -1;    // complemented (< 0): waits for others
        const int first = c - slot;                     // the cell's first body, as nb_link_cell
        int kid = -1, D = 0;
        bool kidCell = false;                           // a start has no child cells
        double4 geo = make_double4(0.0, 0.0, 0.0, 0.0);
        double rsize = 1.0;
        if (c >= 0) {
            kid = kid8[8 * (size_t) slot + sub];
            D = nodeDepth[c];
            geo = nb_ld_pm(&nodePM[c]);
            rsize = rsizeOf(first);
        }
        while (__any_sync(FULL, c >= 0)) {
            double4 q = make_double4(0.0, 0.0, 0.0, 0.0);
            double2 A = make_double2(0.0, 0.0), B = A, C = A;
            if (kid >= 0) q = nb_ld_pm(&nodePM[kid]);
            if (kidCell && useQuad) {
                const double2* kq = reinterpret_cast<const double2*>(nodeQuad + 6 * (size_t) kid);
                A = __ldcg(kq); B = __ldcg(kq + 1); C = __ldcg(kq + 2);
            }
            const int p = c >= 0 ? parent[c] : -1;
            T[sub] = q.w;                               // zeros past the last child: an ordered sum
            T[8 + sub] = q.w * q.x;                     // from +0 is never -0, so they change nothing
            T[16 + sub] = q.w * q.y;
            T[24 + sub] = q.w * q.z;
            int pFirst = 0, pD = 0;
            double4 pGeo = geo;
            if (p >= 0) {                               // (p's centre of mass waits for this cell)
                pFirst = nodeRange[p].x;
                pD = nodeDepth[p];
                pGeo = nb_ld_pm(&nodePM[p]);
            }
            __syncwarp();
            double s = 0.0;
            const int row = sub & 3;
#pragma unroll
            for (int m = 0; m < 8; m += 2) {
                const double2 t = *reinterpret_cast<const double2*>(&T[8 * row + m]);
                s = s + t.x;
                s = s + t.y;
            }
            const double M = __shfl_sync(FULL, s, 0, 8);
            const double com = M > 0.0 ? s / M : row == 1 ? geo.x : row == 2 ? geo.y : geo.z;
            const double cmx = __shfl_sync(FULL, com, 1, 8);
            const double cmy = __shfl_sync(FULL, com, 2, 8);
            const double cmz = __shfl_sync(FULL, com, 3, 8);
            const int pKid = p >= 0 ? kid8[8 * (size_t) (p - pFirst) + sub] : -1;
            double quad = 0.0;                          // of lanes 0 to 5
            if (useQuad) {                              // else the record reads as zero
                const double dx = q.x - cmx, dy = q.y - cmy, dz = q.z - cmz;
                const double drsq = dz * dz + (dy * dy + dx * dx);
                const double mq = q.w;
                double txx = mq * (3.0 * (dx * dx) - drsq);
                double txy = mq * (3.0 * (dx * dy));
                double txz = mq * (3.0 * (dx * dz));
                double tyy = mq * (3.0 * (dy * dy) - drsq);
                double tyz = mq * (3.0 * (dy * dz));
                double tzz = mq * (3.0 * (dz * dz) - drsq);
                if (kidCell) {
                    txx = txx + A.x; txy = txy + A.y; txz = txz + B.x;
                    tyy = tyy + B.y; tyz = tyz + C.x; tzz = tzz + C.y;
                }
                if (kid < 0) txx = txy = txz = tyy = tyz = tzz = 0.0;
                __syncwarp();                           // the sums above have been read
                T[sub] = txx; T[8 + sub] = txy; T[16 + sub] = txz;
                T[24 + sub] = tyy; T[32 + sub] = tyz; T[40 + sub] = tzz;
                __syncwarp();
                const int qrow = sub < 6 ? sub : 5;
#pragma unroll
                for (int m = 0; m < 8; m += 2) {
                    const double2 t = *reinterpret_cast<const double2*>(&T[8 * qrow + m]);
                    quad = quad + t.x;
                    quad = quad + t.y;
                }
            }
            const bool pKidCell = pKid >= 0 && nodeLink[pKid].y < 0;
            if (c >= 0) {
                const double psize = ldexp(rsize, -D);  // rsize halved D times: exact
                const double h = 0.5 * psize;
                const double crit = nb_find_rcrit2(criterion, theta, rsize, geo.x, geo.y, geo.z,
                                                   cmx, cmy, cmz, psize);
                if (sub < 6) nodeQuad[6 * (size_t) c + sub] = quad;
                if (sub == 0) {
                    nodeCrit[c] = crit;
                    nodePM[c] = make_double4(cmx, cmy, cmz, M);
                    if (cmx < geo.x - h || cmx > geo.x + h || cmy < geo.y - h ||
                        cmy > geo.y + h || cmz < geo.z - h || cmz > geo.z + h)
                        outsideOf(first);
                }
            }
            __threadfence();                            // the cell, before its arrival
            __syncwarp();                               // (and T is read before the next cell's terms)
            int left = 0;
            if (sub == 0 && p >= 0) left = atomicSub(&pending[p], 1);
            left = __shfl_sync(FULL, left, 0, 8);
            __threadfence();
            const bool up = left == 1;
            c = up ? p : -1;
            kid = up ? pKid : -1;
            kidCell = up && pKidCell;
            D = pD;
            geo = pGeo;
        }
    }
}
