// The phases of the single-tree build, one body, boundary or cell per call: shared by the
// kernels of nb_tree.cu, which run a phase over all of them per launch, and the one-cluster build
// of nb_build.cu, which runs every phase in one launch.  Plain pointers (no __restrict__): in the
// latter a phase reads what other blocks wrote in the one before.  Bare line citations (:N)
// refer to nbody/src/nbody_tree.c.
#pragma once
#include "nb_tree_util.cuh"
#include <cfloat>

// advancePosVel (nbody/src/nbody_plain.c:268-284): v += (a + acc_i) * dtHalf; x += v * dt, acc_i
// the Milky Way's reflex acceleration of LMC runs (0 otherwise); then the body's share of
// expandBox's max |x - root| with root = 0.
__device__ __forceinline__ double nb_phase_drift(const NbTreeBuffers& b, int i, int drift, double dt,
                                                 double sx, double sy, double sz)
{
    double x = b.px[i], y = b.py[i], z = b.pz[i];
    if (drift) {
        const double dtHalf = 0.5 * dt;
        double vvx = b.vx[i], vvy = b.vy[i], vvz = b.vz[i];
        vvx = vvx + dtHalf * (b.ax[i] + sx);
        vvy = vvy + dtHalf * (b.ay[i] + sy);
        vvz = vvz + dtHalf * (b.az[i] + sz);
        x = x + dt * vvx;
        y = y + dt * vvy;
        z = z + dt * vvz;
        b.vx[i] = vvx; b.vy[i] = vvy; b.vz[i] = vvz;
        b.px[i] = x; b.py[i] = y; b.pz[i] = z;
    }
    double m = fmax(0.0, fabs(x - 0.0));
    m = fmax(m, fabs(y - 0.0));
    return fmax(m, fabs(z - 0.0));
}

// expandBox's doubling loop (:172-175).
__device__ __forceinline__ double nb_phase_root_size(double rsize, double xyzmax)
{
    while (rsize < 2.0 * xyzmax) rsize *= 2.0;
    return rsize;
}

// The grid constants of a finite root size.
__device__ __forceinline__ void nb_phase_grid_constants(double rsize, double& scale, int& depthEps)
{
    scale = ldexp(1.0, NB_GRID_LEVELS - ilogb(rsize));
    int d = 0;
    double q = rsize;
    while (!(q <= DBL_EPSILON)) { q *= 0.5; ++d; }   // nbLoadBody: qsize <= REAL_EPSILON
    depthEps = d;
}

// The body's sort key; returns whether the tree holds the body (test particles do not, :440).
__device__ __forceinline__ bool nb_phase_key(const NbTreeBuffers& b, int i, double scale,
                                             unsigned long long& key)
{
    key = NB_MASSLESS_KEY;
    if (b.mass[i] == 0.0) return false;
    key = nb_morton63(nb_grid(b.px[i], scale), nb_grid(b.py[i], scale), nb_grid(b.pz[i], scale));
    return true;
}

// Grid coordinates of sorted body i.
__device__ __forceinline__ void nb_phase_gather(const NbTreeBuffers& b, int i, double scale)
{
    const unsigned j = b.sort.idxA[i];
    b.gx[i] = nb_grid(b.px[j], scale);
    b.gy[i] = nb_grid(b.py[j], scale);
    b.gz[i] = nb_grid(b.pz[j], scale);
}

// A run of bodies whose 21-level keys are equal, starting at i, is put in full-path order
// (insertion sort; such runs hold only close pairs in practice).
__device__ __forceinline__ void nb_phase_fix_run(const NbTreeBuffers& b, int i, int m)
{
    const unsigned long long* key = b.sort.keyA;
    unsigned* idx = b.sort.idxA;
    if (key[i + 1] != key[i] || (i > 0 && key[i - 1] == key[i])) return;
    int end = i + 2;
    while (end < m && key[end] == key[i]) ++end;
    for (int a = i + 1; a < end; ++a) {
        const long long x = b.gx[a], y = b.gy[a], z = b.gz[a];
        const unsigned id = idx[a];
        int c = a - 1;
        while (c >= i && nb_path_less(x, y, z, b.gx[c], b.gy[c], b.gz[c])) {
            b.gx[c + 1] = b.gx[c]; b.gy[c + 1] = b.gy[c]; b.gz[c + 1] = b.gz[c]; idx[c + 1] = idx[c];
            --c;
        }
        b.gx[c + 1] = x; b.gy[c + 1] = y; b.gz[c + 1] = z; idx[c + 1] = id;
    }
}

// The parting depth at boundary i (written) and the cells the boundary owns (returned).
// nbLoadBody raises a structure error when it must descend through a cell whose size is <=
// REAL_EPSILON (:256-264): that happens iff some pair parts at a depth beyond depthEps.
__device__ __forceinline__ int nb_phase_delta(const NbTreeBuffers& b, int i, int m, int depthEps,
                                              bool& bad)
{
    if (i + 1 >= m) return 0;                        // keep the scanned tail finite
    int d = nb_part_depth(b.gx[i], b.gy[i], b.gz[i], b.gx[i + 1], b.gy[i + 1], b.gz[i + 1]);
    if (d >= depthEps + 1 || d >= NB_GRID_LEVELS) { bad = true; d = min(d, NB_GRID_LEVELS - 1); }
    b.delta[i] = d;
    int prev = -1;
    if (i > 0) {
        prev = nb_part_depth(b.gx[i - 1], b.gy[i - 1], b.gz[i - 1], b.gx[i], b.gy[i], b.gz[i]);
        prev = min(prev, NB_GRID_LEVELS - 1);
    }
    return d > prev ? d - prev : 0;
}

__device__ __forceinline__ int nb_delta_or(const int* delta, int i, int m)
{
    return (i < 0 || i > m - 2) ? -1 : delta[i];
}

// Number of cells owned by boundaries 0..i (inclusive prefix, clamped to the last boundary).
__device__ __forceinline__ int nb_cells_before_body(const int* cum, int i, int m)
{
    if (m <= 1) return 1;                              // root only
    if (i < 0) return 0;
    return cum[min(i, m - 2)];
}

// The node of sorted body i; returns the level of its parent.
__device__ __forceinline__ int nb_phase_emit_body(const NbTreeBuffers& b, int i, int m)
{
    const unsigned j = b.sort.idxA[i];
    const int p = i + nb_cells_before_body(b.cum, i, m);
    b.nodePM[p] = make_double4(b.px[j], b.py[j], b.pz[j], b.mass[j]);
    b.nodeCrit[p] = 0.0;
    b.nodeLink[p] = make_int2(p + 1, (int) j);
    b.nodeRange[p] = make_int2(i, i);
    const int lev = max(0, max(nb_delta_or(b.delta, i - 1, m), nb_delta_or(b.delta, i, m)));
    b.nodeDepth[p] = lev + 1;
    b.bodyNode[i] = p;
    return lev;
}

// Cells owned by boundary a: depths (delta_{a-1}, delta_a].  Writes the geometric centre
// (nbInitMidpoint/calcOffset, :226-239: c += 0.25 * (+-size) level by level from the
// origin) into nodePM.xyz until the moment pass replaces it by the centre of mass.
__device__ __forceinline__ void nb_phase_emit_cells(const NbTreeBuffers& b, int a, int m,
                                                    double rsize, int criterion, double theta)
{
    int dPrev, dHere;
    if (m <= 1) { dPrev = -1; dHere = 0; }
    else { dPrev = nb_delta_or(b.delta, a - 1, m); dHere = b.delta[a]; }
    if (dHere <= dPrev) return;
    const int cellsBefore = a > 0 ? b.cum[a - 1] : 0;
    // centre of the depth-(dPrev+1) cell on body a's path
    double cx = 0.0, cy = 0.0, cz = 0.0, size = rsize;
    const long long bx = m >= 1 ? b.gx[a] : 0, by = m >= 1 ? b.gy[a] : 0, bz = m >= 1 ? b.gz[a] : 0;
    for (int d = 0; d <= dPrev; ++d) {
        const int sh = NB_GRID_LEVELS - 1 - d;
        cx = cx + 0.25 * (((bx >> sh) & 1) ? size : -size);
        cy = cy + 0.25 * (((by >> sh) & 1) ? size : -size);
        cz = cz + 0.25 * (((bz >> sh) & 1) ? size : -size);
        size *= 0.5;
    }
    for (int D = dPrev + 1; D <= dHere; ++D) {
        const int p = a + cellsBefore + (D - dPrev - 1);
        int next, last;
        if (m <= 1) { next = m + 1; last = m - 1; }
        else {
            last = nb_range_end(b.sort.keyA, b.gx, b.gy, b.gz, a, D, m);
            next = last + nb_cells_before_body(b.cum, last, m) + 1;
        }
        b.nodeRange[p] = make_int2(a, last);
        b.nodePM[p] = make_double4(cx, cy, cz, 0.0);
        b.nodeCrit[p] = 0.0;
        b.nodeLink[p] = make_int2(next, -1);
        b.nodeDepth[p] = D;
        if (m == 0) {
            // empty tree: hackCofM of a massless root keeps the geometric centre
            b.nodeCrit[p] = nb_find_rcrit2(criterion, theta, rsize, cx, cy, cz, cx, cy, cz, rsize);
            for (int k = 0; k < 6; ++k) b.nodeQuad[6 * (size_t) p + k] = 0.0;
        }
        // step to the child on body a's path
        const int sh = NB_GRID_LEVELS - 1 - D;
        if (sh >= 0) {
            cx = cx + 0.25 * (((bx >> sh) & 1) ? size : -size);
            cy = cy + 0.25 * (((by >> sh) & 1) ? size : -size);
            cz = cz + 0.25 * (((bz >> sh) & 1) ? size : -size);
        }
        size *= 0.5;
    }
}

// Parent and child list of node c if it is a cell.
__device__ __forceinline__ void nb_phase_link(const NbTreeBuffers& b, int c)
{
    if (c == 0) b.parent[0] = -1;
    const int2 l = b.nodeLink[c];
    if (l.y >= 0) return;              // body
    nb_link_cell(c, l, c - b.nodeRange[c].x, b.nodeLink, b.parent, b.pending, b.cellNode, b.walkKids);
}
