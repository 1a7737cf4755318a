// Force evaluation: FP64 Barnes-Hut walk, FP64 direct summation and the external Milky Way
// potential.  Compiled with -fmad=false so every expression keeps the reference's rounding
// (the reference CPU build uses SSE2 without FMA, milkyway/include/milkyway_math_double.h:128).
//
// Walk (nbGravity, nbody/src/nbody_grav.c:42-124): the reference's stackless walk of every body.
// At node q the body accepts (interacts, then jumps to Next(q)) if q is a body or |dr|^2 >=
// rcrit2(q), otherwise it opens q (goes to More(q) = q + 1 in walk order).  Two kernels: the team
// walk (k_walk_fp64_team) gives four bodies a warp and evaluates eight nodes at once for each, for
// systems too small to fill the GPU with one lane a body; the walk with a lane a body
// (k_walk_fp64_lanes), where each lane takes its own body's path, or the warp the union of its
// bodies' paths.  Either way each body gets exactly the nodes of its own CPU walk, and sums the
// same terms in the CPU's order.  A monopole interaction is 18 flops
// + sqrt + 2 divisions, a quadrupole cell adds 38 flops + 2 divisions.
#include "nb_common.cuh"
#include "nb_potential.cuh"
#include "nb_rdiv.cuh"

constexpr int WALK_THREADS = 128;

// FOREST: the nodes hold one tree per dwarf (batched dwarfs); each lane walks its own
// dwarf's tree, [rootNode, rootEnd), with that dwarf's softening and time step.
// The walk reads one packed record per node (k_pack_walk): 96 bytes, three double4 --
// {CoM, mass}, {rcrit2, Next and, as one 64-bit word with it, the body index or the complement of
// the cell's slot, Qxx, Qxy}, {Qxz, Qyy, Qyz, Qzz} -- so a visit touches one record instead of four
// arrays.  (128-byte records that also held the children were measured: the per-lane walk of 1M
// bodies went from 28.9 to 37.6 ms.)
__global__ void k_pack_walk(const double4* __restrict__ nodePM, const double* __restrict__ nodeCrit,
                            const int2* __restrict__ nodeLink, const int2* __restrict__ nodeRange,
                            const double* __restrict__ nodeQuad, double4* __restrict__ rec,
                            const NbScalars* __restrict__ sc)
{
    if (nb_failed(sc)) return;
    const int nNodes = sc->nNodes;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nNodes; k += gridDim.x * blockDim.x) {
        const int2 l = nodeLink[k];
        const bool body = l.y >= 0;
        const int who = body ? l.y : nodeRange ? ~(k - nodeRange[k].x) : -1;
        const long long word = (long long) (unsigned) l.x | ((long long) who << 32);
        const double* Q = nodeQuad + 6 * (size_t) k;
        double4* r = rec + 3 * (size_t) k;
        r[0] = nodePM[k];
        r[1] = make_double4(nodeCrit[k], __longlong_as_double(word), body ? 0.0 : Q[0],
                            body ? 0.0 : Q[1]);
        r[2] = body ? make_double4(0.0, 0.0, 0.0, 0.0) : make_double4(Q[2], Q[3], Q[4], Q[5]);
    }
}

// The radial factors of one interaction at s = |dr|^2 + eps^2: mor3 = (m / sqrt(s)) / s, and for
// a cell with quadrupole dr5inv = 1 / ((s s) sqrt(s)) and phiQ = 2.5 (dr5inv drQdr) / s, each
// operation rounded as the reference's, with one reciprocal estimate for the root and all four
// divisions (nb_rdiv.cuh).  2^-100 <= s < 2^100 and a mass and a numerator of phiQ between 2^-700
// and 2^700 keep every intermediate and every residual normal; the operators take the rest, and
// the divisors next to an all-ones significand.
// ALWAYS: the quadrupole's factors are formed whether or not this lane's node is a cell (no branch).
// Returns whether the operands are in those ranges (a mass of +-0, for which mor3 comes out as a
// zero all the same, is not: only the direct sum meets one, and asks nb_mor3_shared again).
template <bool ALWAYS>
__device__ __forceinline__ bool nb_radial_shared(double s, double m, bool cell, double drQdr,
                                                 double& mor3, double& dr5inv, double& phiQ)
{
    double y;
    const double drab = nb_sqrt_recip(s, nb_rsqrt_estimate(s), y);
    const double z = nb_recip_step(s, y * y);
    mor3 = nb_quot(nb_quot(m, drab, y), s, z);
    bool ok = nb_pos_exp_in<-100, 100>(s) && nb_exp_in<-700, 700>(m) && !nb_near_ones(s);
    if (ALWAYS || cell) {
        const double t = (s * s) * drab;
        dr5inv = nb_recip_step(t, nb_recip_step(t, (z * z) * y));
        const double a = 2.5 * (dr5inv * drQdr);
        phiQ = nb_quot(a, s, z);
        ok = ok && (!cell || (nb_exp_in<-700, 700>(a) && !nb_near_ones(t)));
    }
    return ok;
}

// Whether nb_radial_shared's mor3 stands.
__device__ __forceinline__ bool nb_mor3_shared(double s, double m)
{
    return nb_pos_exp_in<-100, 100>(s) && !nb_near_ones(s) && (nb_exp_in<-700, 700>(m) || nb_is_zero(m));
}

// The operators' forms.
__device__ __forceinline__ void nb_radial_general(double s, double m, bool cell, double drQdr,
                                                  double& mor3, double& dr5inv, double& phiQ)
{
    const double root = sqrt(s);
    mor3 = (m / root) / s;
    if (cell) {
        dr5inv = 1.0 / ((s * s) * root);
        phiQ = 2.5 * (dr5inv * drQdr) / s;
    }
}

template <bool ALWAYS>
__device__ __forceinline__ void nb_radial(double s, double m, bool need, bool cell, double drQdr,
                                          double& mor3, double& dr5inv, double& phiQ)
{
    const bool ok = nb_radial_shared<ALWAYS>(s, m, cell, drQdr, mor3, dr5inv, phiQ);
    if (need && !ok) nb_radial_general(s, m, cell, drQdr, mor3, dr5inv, phiQ);
}

// The team walk: a warp walks for TEAM_BODIES consecutive bodies, TEAM_LANES lanes each (lane =
// TEAM_BODIES * p + b: lane p of body b's team).  The warp walks the union of its bodies' paths
// depth first, a cell's children tested at once (lane p tests child p for body b, one ballot
// gives every child's bodies), and lists the nodes that some body takes in walk order: a node
// taken by a body is closed to it with all below (`cover`), a child that some body opens is
// walked into before its later siblings.  Every TEAM_LANES listed nodes are evaluated at once, one
// lane per (node, body); the terms go through shared memory to one lane per (body, component),
// which adds them in list order while the next eight are evaluated -- every body sums its CPU
// walk's terms in the CPU's order, and only the additions are serial.
// What bounds it: latency (about 2.8 cycles a warp instruction wait on a dependent result) and,
// at its upper end, issue slots: four bodies share ~200 instructions per eight nodes and ~150 per
// opened cell, against ~190 a node for 32 bodies in the per-lane walk, which carries the
// root-and-divisions chain of every node in its serial part on an eighth of the warps.  Five
// resident blocks (96 registers): six to eight (80 to 64) were 3 to 20 % slower.
// Walk times, per lane with the early load -> team, ms, on the two-component dwarf: with quadrupoles
// 5,000 bodies (theta 1) 0.338 -> 0.159, 12,000 0.391 -> 0.213, 20,000 0.422 -> 0.349 (theta 0.5:
// 1.457 -> 1.183), 25,000 0.430 -> 0.440 (0.7: 0.783 -> 0.774, 0.5: 1.537 -> 1.407), 32,768 0.461 ->
// 0.542; without them, when the additions are most of a node's work, 5,000 0.190 -> 0.156, 12,000
// 0.217 -> 0.211 (0.7: 0.362 -> 0.367, 0.5: 0.684 -> 0.713), 16,384 0.218 -> 0.306, 32,768 0.254 ->
// 0.529.  Hence the automatic choice's two lines.  Small opening angles take few cells and many
// bodies, whose work is mostly the additions again.  With quadrupoles, union -> team: 12,000 bodies,
// theta 0.05 6.09 -> 5.65, 0 7.09 -> 11.8; 14,000, 0.1 7.08 -> 6.39; 16,384, 0.1 8.02 -> 8.72, 0.05 8.35 ->
// 12.4; 20,000, 0.15 8.79 -> 8.49, 0.1 9.84 -> 11.6; 24,000, 0.2 8.23 -> 7.85, 0.15 10.2 -> 11.3; 32,768, 0.2
// 11.0 -> 10.2, 0.15 13.5 -> 16.0.  So form 0 is the team walk up to the smaller line, and up to
// TEAM_MAX_BODIES where theta >= min(TEAM_THETA, (bodies - 9,000) / 85,000).
constexpr int TEAM_BODIES = 4;
constexpr int TEAM_MAX_BODIES = 32768;
constexpr int TEAM_AUTO_QUAD = 24576, TEAM_AUTO_MONO = 12288;
constexpr double TEAM_THETA = 0.2;
// with quadrupoles and up to the smaller line it is the fastest form down to this angle (10,000 bodies at
// 0.05: early load 5.64, team 4.43; 12,000: 6.81, 5.65; at 0: 5.53, 11.8)
constexpr double TEAM_SMALL_THETA = 0.04;
constexpr int TEAM_LANES = 32 / TEAM_BODIES;                // 8: a cell's children
constexpr unsigned TEAM_ALL = (1u << TEAM_BODIES) - 1u;     // every body of the warp
constexpr unsigned TEAM_FIRST = 0x11111111u;                // the lanes with b = 0
constexpr int TEAM_RING = 16;         // at most 7 listed before a cell's up to 8
struct NbTeam {
    double term[3][3 * 32 + 4];         // component: three terms of every lane (padded)
    int2 ring[TEAM_RING];               // listed: {node, cells complemented; bodies that take it}
    // the cells with children still to list: {cell's slot, the bodies of its eight children in
    // four bits each, next child | cover << 8 | open children << 16 | children that are bodies << 24}
    int4 frame[NB_GRID_LEVELS + 2];
};

template <bool COUNT, bool FOREST>
__global__ void __launch_bounds__(WALK_THREADS, 5)
k_walk_fp64_team(const double4* __restrict__ rec, const int* __restrict__ kids,
            const unsigned int* __restrict__ order, const double* __restrict__ px,
            const double* __restrict__ py, const double* __restrict__ pz,
            double* __restrict__ ax, double* __restrict__ ay, double* __restrict__ az,
            NbWalkParams wp, NbScalars* __restrict__ sc, NbForest forest)
{
    __shared__ NbTeam teams[WALK_THREADS / 32];
    if (nb_failed(sc)) return;
    NbTeam& T = teams[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int b = lane % TEAM_BODIES, p = lane / TEAM_BODIES;
    const int i = (int) ((blockIdx.x * (unsigned) blockDim.x + threadIdx.x) >> 5) * TEAM_BODIES + b;
    if (i - b >= wp.n) return;                      // the whole warp
    const bool valid = i < wp.n;
    const unsigned j = valid ? order[i] : 0xffffffffu;
    const double x0 = valid ? px[j] : 0.0, y0 = valid ? py[j] : 0.0, z0 = valid ? pz[j] : 0.0;
    double eps2 = wp.eps2;
    const bool useQuad = wp.useQuad != 0;
    int root = 0;
    if (FOREST && valid) {
        const NbDwarfDev& dw = forest.dwarfs[forest.bodyDwarf[i]];
        eps2 = dw.eps2;
        root = dw.rootNode;
    }
    double acc = 0.0;                   // lanes 0..11: component p of body b
    bool metSelf = false;
    unsigned long long cVisit = 0, cBB = 0, cBC = 0, cSteps = 0;

    // the current cell's children, child p in lanes 4 p ..: node, the bodies that take it
    int kid = -1, kidSlot = 0, cellSlot = 0;
    unsigned use = 0;
    unsigned todo = __ballot_sync(NB_FULL_MASK, valid) & TEAM_ALL;   // bodies whose tree is to come
    unsigned open = 0, leaf = 0;        // bit 4 p: some body opens child p; child p is a body
    unsigned cover = 0;                 // bodies that took an ancestor of these children
    int pos = TEAM_LANES;               // the next child to list
    int level = 0, head = 0, tail = 0;

    // the opening test (nbody/src/nbody_grav.c:55-62) of the children in `kid`
    auto test = [&]() {
        const double4* r = rec + 3 * (size_t) max(kid, 0);
        const double4 nd = nb_ld32(r);
        const double2 r1 = __ldg(reinterpret_cast<const double2*>(r + 1));
        const int bodyIndex = __double2hiint(r1.y);
        const double dx = nd.x - x0, dy = nd.y - y0, dz = nd.z - z0;
        const double drSq = dz * dz + (dy * dy + dx * dx);
        const bool mine = kid >= 0 && !((cover >> b) & 1u);     // this body still walks here
        const bool body = kid >= 0 && bodyIndex >= 0;
        kidSlot = ~bodyIndex;
        const bool self = mine && body && (unsigned) bodyIndex == j;
        const bool take = mine && (body ? !self : drSq >= r1.x);
        metSelf |= self;
        use = (__ballot_sync(NB_FULL_MASK, take) >> (TEAM_BODIES * p)) & TEAM_ALL;
        leaf = __ballot_sync(NB_FULL_MASK, body) & TEAM_FIRST;
        open = __ballot_sync(NB_FULL_MASK, kid >= 0 && !body && (cover | use) != TEAM_ALL) & TEAM_FIRST;
        pos = 0;
        if (COUNT) {
            cVisit += __popc(__ballot_sync(NB_FULL_MASK, mine));
            cBB += __popc(__ballot_sync(NB_FULL_MASK, take && body));
            cBC += __popc(__ballot_sync(NB_FULL_MASK, take && !body));
            ++cSteps;
        }
    };
    // adds the last batch's terms in list order (every lane, for the arithmetic to overlap the
    // next batch's; a zero term of either sign leaves the sum, which never is -0, as it is)
    const double* const sums = T.term[min(p, 2)] + b;
    auto add_terms = [&]() {
#pragma unroll
        for (int e = 0; e < TEAM_LANES; ++e) {
            acc = acc + sums[TEAM_BODIES * e];
            acc = acc + sums[32 + TEAM_BODIES * e];
            acc = acc - sums[64 + TEAM_BODIES * e];
        }
    };
    // the terms of up to TEAM_LANES listed nodes (nbody/src/nbody_grav.c:64-100)
    auto evaluate = [&]() {
        if (COUNT) ++cSteps;
        const int2 entry = T.ring[(tail + p) % TEAM_RING];
        const bool take = tail + p < head && (((unsigned) entry.y >> b) & 1u);
        const int node = take ? (entry.x < 0 ? ~entry.x : entry.x) : 0;
        const bool cell = entry.x < 0 && useQuad && take;
        const double4* r = rec + 3 * (size_t) node;
        const double4 nd = nb_ld32(r);
        const double2 r1 = __ldg(reinterpret_cast<const double2*>(r + 1) + 1);
        const double4 r2 = nb_ld32(r + 2);
        add_terms();
        const double dx = nd.x - x0, dy = nd.y - y0, dz = nd.z - z0;
        const double s = (dz * dz + (dy * dy + dx * dx)) + eps2;
        const double qxx = r1.x, qxy = r1.y, qxz = r2.x, qyy = r2.y, qyz = r2.z, qzz = r2.w;
        const double qdx = qxx * dx + qxy * dy + qxz * dz;
        const double qdy = qxy * dx + qyy * dy + qyz * dz;
        const double qdz = qxz * dx + qyz * dy + qzz * dz;
        const double drQdr = qdx * dx + qdy * dy + qdz * dz;
        double mor3, dr5inv, phiQ;
        nb_radial<true>(s, nd.w, take, cell, drQdr, mor3, dr5inv, phiQ);
        __syncwarp();
        T.term[0][lane] = take ? mor3 * dx : 0.0;
        T.term[1][lane] = take ? mor3 * dy : 0.0;
        T.term[2][lane] = take ? mor3 * dz : 0.0;
        T.term[0][32 + lane] = cell ? phiQ * dx : 0.0;
        T.term[1][32 + lane] = cell ? phiQ * dy : 0.0;
        T.term[2][32 + lane] = cell ? phiQ * dz : 0.0;
        T.term[0][64 + lane] = cell ? dr5inv * qdx : 0.0;
        T.term[1][64 + lane] = cell ? dr5inv * qdy : 0.0;
        T.term[2][64 + lane] = cell ? dr5inv * qdz : 0.0;
        __syncwarp();
        tail += TEAM_LANES;
    };

#pragma unroll
    for (int k = 0; k < 3; ++k)
        T.term[0][32 * k + lane] = T.term[1][32 * k + lane] = T.term[2][32 * k + lane] = 0.0;
    __syncwarp();
    for (;;) {
        if (pos >= TEAM_LANES) {                    // this cell's children are done
            if (level > 0) {
                --level;
                __syncwarp();
                const int4 f = T.frame[level];
                cellSlot = f.x;
                kid = __ldg(kids + 8 * (size_t) cellSlot + p);
                // the upper half of the record's link word
                kidSlot = ~__ldg(reinterpret_cast<const int*>(rec + 3 * (size_t) max(kid, 0) + 1) + 3);
                use = ((unsigned) f.y >> (4 * p)) & TEAM_ALL;
                pos = f.z & 255;
                cover = ((unsigned) f.z >> 8) & 255u;
                open = (unsigned) f.w & TEAM_FIRST;
                leaf = ((unsigned) f.w >> 1) & TEAM_FIRST;
            } else if (todo) {                      // the next root (one tree per dwarf)
                const int r = __shfl_sync(NB_FULL_MASK, root, __ffs(todo) - 1);
                const unsigned group = __ballot_sync(NB_FULL_MASK, valid && root == r) & TEAM_ALL;
                todo &= ~group;
                cover = TEAM_ALL & ~group;
                kid = p == 0 ? r : -1;
                test();
            } else {
                break;
            }
        }
        // list the children up to the next one that some body opens
        const unsigned om = open & (~0u << (TEAM_BODIES * pos));
        const int stop = om ? (__ffs(om) - 1) / TEAM_BODIES : TEAM_LANES - 1;
        const unsigned taken = __ballot_sync(NB_FULL_MASK, b == 0 && use != 0u);
        const unsigned adds = taken & (~0u << (TEAM_BODIES * pos)) &
                              (~0u >> (TEAM_BODIES * (TEAM_LANES - 1 - stop)));
        if ((adds >> lane) & 1u)
            T.ring[(head + __popc(adds & ((1u << lane) - 1u))) % TEAM_RING] =
                make_int2((leaf >> lane) & 1u ? kid : ~kid, (int) use);
        head += __popc(adds);
        pos = stop + 1;
        if (om) {                                   // walk into it
            const int c = __shfl_sync(NB_FULL_MASK, kidSlot, TEAM_BODIES * stop);
            const unsigned u = __shfl_sync(NB_FULL_MASK, use, TEAM_BODIES * stop);
            const int next = __ldg(kids + 8 * (size_t) c + p);
            if (pos < TEAM_LANES && ((taken | open) >> (TEAM_BODIES * pos)) != 0u) {
                const unsigned uses = __reduce_or_sync(NB_FULL_MASK, use << (4 * p));
                if (lane == 0)
                    T.frame[level] = make_int4(cellSlot, (int) uses, pos | (int) (cover << 8),
                                               (int) (open | leaf << 1));
                ++level;
            }
            cover |= u;
            cellSlot = c;
            kid = next;
            test();
        }
        if (head - tail >= TEAM_LANES) {
            __syncwarp();
            evaluate();
        }
    }
    __syncwarp();
    if (tail < head) evaluate();
    add_terms();
    if (COUNT && lane == 0) {           // every lane counted the warp's numbers alike
        atomicAdd(&sc->nWarpSteps, cSteps);
        atomicAdd(&sc->nVisit, cVisit);
        atomicAdd(&sc->nBodyBody, cBB);
        atomicAdd(&sc->nBodyCell, cBC);
    }
    // the team's lanes met the children between them
    metSelf = (__ballot_sync(NB_FULL_MASK, metSelf) & (TEAM_FIRST << b)) != 0u;
    if (!valid) return;
    // a body that never meets itself is tree incest (nbody/src/nbody_grav.c:111-118)
    if (p == 0 && !metSelf) {
        atomicOr(&sc->incest, 1);
        if (FOREST)
            atomicOr(&forest.dwarfs[forest.bodyDwarf[i]].status, NBODY_TREE_INCEST_NONFATAL);
    }
    // self-gravity only; k_body_epilogue adds the external potential and kicks (kept out of
    // this kernel so that its registers serve the walk)
    if (p < 3) (p == 0 ? ax : p == 1 ? ay : az)[j] = acc;
}

// The walk with a lane a body.  LANES_OWN: each iteration every lane
// that has not finished takes the next node of its own walk (a per-lane gather of the node
// record, one 32-byte load per sector), so a lane is idle only when its walk is over.  Each lane
// meets exactly its CPU walk's nodes in the CPU's order and sums the same terms in the same
// order.  Bodies consecutive in path order have walks of similar length, so the warp runs about
// as many iterations as its longest walk (0.96 of the lane slots do work on the 131k-body dwarf
// at theta 0.5).  Bound by the L1 data pipe (88 % busy: a 32-byte load is at least eight
// wavefronts a warp, more with distinct records) and the FP64 pipe (59 %).  Sharing one
// reciprocal among the root and the divisions (nb_radial) took the 1,048,576-body dwarf from 28.9
// to 28.1 ms at theta 0.5 and from 7.05 to 6.54 ms at theta 1.
// LANES_EARLY: the next node's record is loaded as soon as the opening test has chosen it, before
// this node's terms are computed, so its latency overlaps the FP64 arithmetic (79 registers
// against 63: it pays where few warps are resident, up to some 80,000 bodies).
// LANES_UNION: the warp takes the smallest of its lanes' next nodes, the lanes that are at it do it:
// one broadcast load a node, but an iteration for every node that any lane visits (FP64 pipe 68 %
// busy, L1 data pipe 37 %).  The smaller the
// opening angle, the more of a walk its neighbours share: walks of 1,048,576 bodies, own -> union:
// theta 0.7 12.4 -> 13.6 ms, 0.5 28.1 -> 28.2, 0.4 49.4 -> 44.2, 0.3 107 -> 84.5, 0.2 302 -> 210; 50,000
// bodies, early -> union: 0.5 1.89 -> 2.70, 0.25 9.64 -> 9.98, 0.2 15.2 -> 13.6, 0.1 34.2 -> 22.3.
enum { LANES_OWN, LANES_EARLY, LANES_UNION };
template <bool COUNT, bool FOREST, int PATH>
__global__ void __launch_bounds__(WALK_THREADS)
k_walk_fp64_lanes(const double4* __restrict__ rec,
                  const unsigned int* __restrict__ order, const double* __restrict__ px,
                  const double* __restrict__ py, const double* __restrict__ pz,
                  double* __restrict__ ax, double* __restrict__ ay, double* __restrict__ az,
                  NbWalkParams wp, NbScalars* __restrict__ sc, NbForest forest)
{
    if (nb_failed(sc)) return;
    const int end = sc->nNodes;
    const int lane = threadIdx.x & 31;
    const int i = (int) ((blockIdx.x * (unsigned) blockDim.x + threadIdx.x) >> 5) * 32 + lane;
    const bool valid = i < wp.n;
    const unsigned j = valid ? order[i] : 0u;
    const double x0 = valid ? px[j] : 0.0, y0 = valid ? py[j] : 0.0, z0 = valid ? pz[j] : 0.0;
    double eps2 = wp.eps2;
    const bool useQuad = wp.useQuad != 0;
    int myEnd = end;
    int ptr = 0;
    NbDwarfDev* dw = nullptr;
    if (FOREST && valid) {
        dw = &forest.dwarfs[forest.bodyDwarf[i]];
        eps2 = dw->eps2;
        ptr = dw->rootNode;
        myEnd = dw->rootEnd;
    }
    if (!valid) ptr = myEnd;
    double accx = 0.0, accy = 0.0, accz = 0.0;
    bool metSelf = false;
    unsigned long long cVisit = 0, cBB = 0, cBC = 0, cSteps = 0;
    constexpr bool PREFETCH = PATH == LANES_EARLY;
    double4 nd = make_double4(0.0, 0.0, 0.0, 0.0), r1 = nd;
    if (PREFETCH && ptr < myEnd) {
        nd = nb_ld32(rec + 3 * (size_t) ptr);
        r1 = nb_ld32(rec + 3 * (size_t) ptr + 1);
    }
    for (;;) {
        // every lane takes part in the vote of every iteration (a finished lane idles in the
        // loop), and the warp leaves the loop together when all its walks are over
        int q = ptr;
        bool active;
        if (PATH == LANES_UNION) {
            if (FOREST && ptr >= myEnd) ptr = end;      // this lane's tree is done
            q = __reduce_min_sync(NB_FULL_MASK, ptr);
            if (q >= end) break;
            active = ptr == q;
        } else {
            active = ptr < myEnd;
            if (!__any_sync(NB_FULL_MASK, active)) break;
        }
        if (COUNT) ++cSteps;
        if (!active) continue;
        if (!PREFETCH) {
            nd = nb_ld32(rec + 3 * (size_t) q);
            r1 = nb_ld32(rec + 3 * (size_t) q + 1);
        }
        const long long word = __double_as_longlong(r1.y);
        const int2 link = make_int2((int) (unsigned) (word & 0xffffffffll), (int) (word >> 32));
        const double dx = nd.x - x0, dy = nd.y - y0, dz = nd.z - z0;
        double drSq = dz * dz + (dy * dy + dx * dx);
        const bool isBody = link.y >= 0;
        if (COUNT) ++cVisit;
        const bool accept = isBody || drSq >= r1.x;
        ptr = accept ? link.x : q + 1;
        double4 ndNext = nd, r1Next = r1;
        if (PREFETCH && ptr < myEnd) {
            ndNext = nb_ld32(rec + 3 * (size_t) ptr);
            r1Next = nb_ld32(rec + 3 * (size_t) ptr + 1);
        }
        if (accept && isBody && (unsigned) link.y == j) metSelf = true;
        else if (accept) {
            if (COUNT) { if (isBody) ++cBB; else ++cBC; }
            drSq = drSq + eps2;
            const bool quad = useQuad && !isBody;
            double qdx, qdy, qdz, drQdr = 0.0, mor3, dr5inv, phiQ;
            if (quad) {
                const double4 r2 = nb_ld32(rec + 3 * (size_t) q + 2);
                const double qxx = r1.z, qxy = r1.w, qxz = r2.x, qyy = r2.y, qyz = r2.z, qzz = r2.w;
                qdx = qxx * dx + qxy * dy + qxz * dz;
                qdy = qxy * dx + qyy * dy + qyz * dz;
                qdz = qxz * dx + qyz * dy + qzz * dz;
                drQdr = qdx * dx + qdy * dy + qdz * dz;
            }
            nb_radial<false>(drSq, nd.w, true, quad, drQdr, mor3, dr5inv, phiQ);
            accx = accx + mor3 * dx;
            accy = accy + mor3 * dy;
            accz = accz + mor3 * dz;
            if (quad) {
                accx = accx + phiQ * dx;
                accy = accy + phiQ * dy;
                accz = accz + phiQ * dz;
                accx = accx - dr5inv * qdx;
                accy = accy - dr5inv * qdy;
                accz = accz - dr5inv * qdz;
            }
        }
        if (PREFETCH) { nd = ndNext; r1 = r1Next; }
    }
    if (COUNT) {
        // every lane counted the warp's iterations alike
        for (int o = 16; o > 0; o >>= 1) {
            cVisit += __shfl_xor_sync(NB_FULL_MASK, cVisit, o);
            cBB += __shfl_xor_sync(NB_FULL_MASK, cBB, o);
            cBC += __shfl_xor_sync(NB_FULL_MASK, cBC, o);
        }
        if (lane == 0) {
            atomicAdd(&sc->nWarpSteps, cSteps);
            atomicAdd(&sc->nVisit, cVisit);
            atomicAdd(&sc->nBodyBody, cBB);
            atomicAdd(&sc->nBodyCell, cBC);
        }
    }
    if (!valid) return;
    // a body that never meets itself is tree incest (nbody/src/nbody_grav.c:111-118)
    if (!metSelf) {
        atomicOr(&sc->incest, 1);
        if (FOREST) atomicOr(&dw->status, NBODY_TREE_INCEST_NONFATAL);
    }
    ax[j] = accx; ay[j] = accy; az[j] = accz;
}

// nbMapForceBody's epilogue for every body after a tree walk: a = self-gravity (as the walk
// stored it) + nbExtAcceleration + the zero LMC term, then the optional kick (nb_finish_body).
// FOREST: each body with its dwarf's time step and the bar's time of its dwarf.
// CAUSTIC: the potential's halo is the caustic one (its code compiled in only then).
template <bool FOREST, bool CAUSTIC>
__global__ void k_body_epilogue(const double* __restrict__ px, const double* __restrict__ py,
                                const double* __restrict__ pz, double* __restrict__ ax,
                                double* __restrict__ ay, double* __restrict__ az,
                                double* __restrict__ vx, double* __restrict__ vy,
                                double* __restrict__ vz, NbWalkParams wp, NbPot pot,
                                const NbScalars* __restrict__ sc, NbForest forest)
{
    if (nb_failed(sc)) return;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < wp.n; j += gridDim.x * blockDim.x) {
        NbWalkParams w = wp;
        NbPot p = pot;
        if (FOREST) {
            const int dj = forest.bodyDwarf[j];
            NbDwarfDev& d = forest.dwarfs[dj];
            w.dtHalf = 0.5 * d.dt;
            p.time = d.time;
            // LMC runs: this dwarf's LMC and its reflex acceleration acc_i1 (selects, not
            // branches: a conditional update of the copies costs the kernel ~70 registers)
            const bool lmc = forest.lmcShift != nullptr;
            p.lmc = lmc ? d.lmc : p.lmc;
            const double* sh = lmc && w.kick
                ? forest.lmcShift + 3 * ((size_t) dj * forest.nShift + sc->step + 1) : w.shift;
            const double s0 = sh[0], s1 = sh[1], s2 = sh[2];
            w.shift[0] = s0; w.shift[1] = s1; w.shift[2] = s2;
        }
        nb_finish_body<CAUSTIC>(p, w, (unsigned) j, px[j], py[j], pz[j], ax[j], ay[j], az[j], ax, ay, az,
                       vx, vy, vz);
    }
}

void nb_launch_body_epilogue(const double* px, const double* py, const double* pz, double* ax,
                             double* ay, double* az, double* vx, double* vy, double* vz,
                             const NbWalkParams& wp, const NbPot& pot, const NbScalars* sc,
                             int numSMs, cudaStream_t s, const NbForest* forest)
{
    if (wp.n <= 0) return;
    const int g = numSMs > 0 ? min((wp.n + 255) / 256, numSMs * 8) : (wp.n + 255) / 256;
    const NbForest f = forest ? *forest : NbForest{nullptr, nullptr, 0, nullptr, 0};
    const bool caustic = pot.enabled && pot.haloType == NBCUDA_CAUSTIC_HALO;
#define NB_EPI_ARGS px, py, pz, ax, ay, az, vx, vy, vz, wp, pot, sc, f
    if (forest) {
        if (caustic) k_body_epilogue<true, true><<<g, 256, 0, s>>>(NB_EPI_ARGS);
        else k_body_epilogue<true, false><<<g, 256, 0, s>>>(NB_EPI_ARGS);
    } else {
        if (caustic) k_body_epilogue<false, true><<<g, 256, 0, s>>>(NB_EPI_ARGS);
        else k_body_epilogue<false, false><<<g, 256, 0, s>>>(NB_EPI_ARGS);
    }
#undef NB_EPI_ARGS
    nb_count_launch();
}

// nbGravity_Exact (nbody/src/nbody_grav.c:205-227): direct sum over all bodies in input order
// (the self term contributes 0 * dr).  H lanes share a body: each forms the terms of every H-th
// group of EXACT_UNROLL sources, EXACT_UNROLL independent root-and-division chains at once with
// the next group's loads behind them, and the terms are added one after another in input order
// (lane by lane through shuffles).  Bound by the FP64 pipe, 31 operations a pair, once enough
// warps are resident; a warp alone on its scheduler, the usual case here, waits for its own
// chains (116 cycles a source where the pipe takes 62).  A thread a body in blocks of 256, one
// chain at a time, took 2.24 ms at 10,007 bodies and 0.23 at 1,000; now 0.59 and 0.041.  H = 1 / 2 /
// 4 in ms: 4,000 bodies 0.244 / 0.175 / 0.135, 7,000 0.420 / 0.304 / 0.357, 10,007 0.593 / 0.693 /
// 0.779, 20,000 2.03 / 2.11 / 2.50 (4.46 before), 30,000 3.03 / 4.08 / 5.20.  With every eighth body a
// test particle 20,000 take 2.46 (6.40 with the operators for every group that holds one).
constexpr int EXACT_TILE = 256;
constexpr int EXACT_UNROLL = 8;
template <int H>
__global__ void __launch_bounds__(32)
k_direct_fp64(const double* __restrict__ px, const double* __restrict__ py,
              const double* __restrict__ pz, const double* __restrict__ mass,
              double* __restrict__ ax, double* __restrict__ ay, double* __restrict__ az,
              NbWalkParams wp)
{
    constexpr int U = EXACT_UNROLL;
    const int n = wp.n;
    const int lane = threadIdx.x & 31;
    const int h = lane % H;
    const int i = blockIdx.x * (32 / H) + lane / H;
    const bool valid = i < n;
    const double x0 = valid ? px[i] : 0.0, y0 = valid ? py[i] : 0.0, z0 = valid ? pz[i] : 0.0;
    const double eps2 = wp.eps2;
    double acc[3] = {0.0, 0.0, 0.0};
    double x[U], y[U], z[U], m[U];
    auto fetch = [&](int k0) {
        if (k0 + U <= n) {
#pragma unroll
            for (int u = 0; u < U; u += 4) {            // k0 is a multiple of 8: 32-byte aligned
                const double4 a = nb_ld32(reinterpret_cast<const double4*>(px + k0 + u));
                const double4 b = nb_ld32(reinterpret_cast<const double4*>(py + k0 + u));
                const double4 c = nb_ld32(reinterpret_cast<const double4*>(pz + k0 + u));
                const double4 d = nb_ld32(reinterpret_cast<const double4*>(mass + k0 + u));
                x[u] = a.x; x[u + 1] = a.y; x[u + 2] = a.z; x[u + 3] = a.w;
                y[u] = b.x; y[u + 1] = b.y; y[u + 2] = b.z; y[u + 3] = b.w;
                z[u] = c.x; z[u + 1] = c.y; z[u + 2] = c.z; z[u + 3] = c.w;
                m[u] = d.x; m[u + 1] = d.y; m[u + 2] = d.z; m[u + 3] = d.w;
            }
        } else {                                        // past the end: the last body, taken as none
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int k = min(k0 + u, n - 1);
                x[u] = px[k]; y[u] = py[k]; z[u] = pz[k]; m[u] = mass[k];
            }
        }
    };
    fetch(U * h);
    for (int base = 0; base < n; base += U * H) {
        const int k0 = base + U * h;
        // one test for all: a branch a source would keep the chains from overlapping
        double t[U][3], r2[U], mm[U], mor3[U], dr5inv, phiQ;
        bool ok = true;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            t[u][0] = x[u] - x0; t[u][1] = y[u] - y0; t[u][2] = z[u] - z0;
            r2[u] = (t[u][2] * t[u][2] + (t[u][1] * t[u][1] + t[u][0] * t[u][0])) + eps2;
            mm[u] = m[u];
        }
        fetch(k0 + U * H);                              // the next sources, behind this arithmetic
#pragma unroll
        for (int u = 0; u < U; ++u)
            ok &= nb_radial_shared<false>(r2[u], mm[u], false, 0.0, mor3[u], dr5inv, phiQ);
        if (!ok) {                                      // test particles among the sources, or worse
            ok = true;
#pragma unroll
            for (int u = 0; u < U; ++u) ok &= nb_mor3_shared(r2[u], mm[u]);
            if (!ok)
#pragma unroll
                for (int u = 0; u < U; ++u)
                    nb_radial_general(r2[u], mm[u], false, 0.0, mor3[u], dr5inv, phiQ);
        }
        // the sum never is -0, so a zero term leaves it as it is
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int c = 0; c < 3; ++c) t[u][c] = k0 + u < n ? mor3[u] * t[u][c] : 0.0;
#pragma unroll
        for (int q = 0; q < H; ++q)
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    acc[c] = acc[c] + (H == 1 ? t[u][c]
                                              : __shfl_sync(NB_FULL_MASK, t[u][c], lane - h + q));
    }
    // self-gravity only; k_body_epilogue adds the external potential and kicks
    if (valid && h == 0) { ax[i] = acc[0]; ay[i] = acc[1]; az[i] = acc[2]; }
}

// Direct FP64 sums (nbGravity_Exact arithmetic) for a sample of target bodies: the accuracy
// oracle of the walk forms.  Self-gravity only.
__global__ void __launch_bounds__(EXACT_TILE)
k_direct_sample(const double* __restrict__ px, const double* __restrict__ py,
                const double* __restrict__ pz, const double* __restrict__ mass, int n,
                const int* __restrict__ targets, int count, double eps2, double* __restrict__ out)
{
    __shared__ double4 tile[EXACT_TILE];
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = t < count;
    const int i = valid ? targets[t] : 0;
    const double x0 = px[i], y0 = py[i], z0 = pz[i];
    double accx = 0.0, accy = 0.0, accz = 0.0;
    for (int base = 0; base < n; base += EXACT_TILE) {
        const int k = base + threadIdx.x;
        __syncthreads();
        tile[threadIdx.x] = k < n ? make_double4(px[k], py[k], pz[k], mass[k]) : make_double4(0, 0, 0, 0);
        __syncthreads();
        const int lim = min(EXACT_TILE, n - base);
        for (int s = 0; s < lim; ++s) {
            const double4 b = tile[s];
            const double dx = b.x - x0, dy = b.y - y0, dz = b.z - z0;
            const double drSq = (dz * dz + (dy * dy + dx * dx)) + eps2;
            const double drab = sqrt(drSq);
            const double phii = b.w / drab;
            const double mor3 = phii / drSq;
            accx = accx + mor3 * dx;
            accy = accy + mor3 * dy;
            accz = accz + mor3 * dz;
        }
    }
    if (valid) { out[3 * t] = accx; out[3 * t + 1] = accy; out[3 * t + 2] = accz; }
}

// Total energy of the current state, FP64 direct summation (the energy-drift oracle of the
// walk forms; O(N^2)): out[0] += sum m v^2 / 2, out[1] += -sum_{i<j} m_i m_j / sqrt(r^2 + eps^2)
// (the softened pair potential whose gradient the walk's forces are), out[2] += sum m Phi_ext.
__global__ void __launch_bounds__(EXACT_TILE)
k_energy(const double* __restrict__ px, const double* __restrict__ py,
         const double* __restrict__ pz, const double* __restrict__ vx,
         const double* __restrict__ vy, const double* __restrict__ vz,
         const double* __restrict__ mass, int n, double eps2, NbPot pot, double* __restrict__ out)
{
    __shared__ double4 tile[EXACT_TILE];
    __shared__ double red[3][EXACT_TILE / 32];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < n;
    const double x0 = valid ? px[i] : 0.0, y0 = valid ? py[i] : 0.0, z0 = valid ? pz[i] : 0.0;
    double phi = 0.0;
    for (int base = 0; base < n; base += EXACT_TILE) {
        const int k = base + threadIdx.x;
        __syncthreads();
        tile[threadIdx.x] = k < n ? make_double4(px[k], py[k], pz[k], mass[k]) : make_double4(0, 0, 0, 0);
        __syncthreads();
        const int lim = min(EXACT_TILE, n - base);
        for (int s = 0; s < lim; ++s) {
            const double4 b = tile[s];
            const double dx = b.x - x0, dy = b.y - y0, dz = b.z - z0;
            const double drSq = (dz * dz + (dy * dy + dx * dx)) + eps2;
            phi += base + s == i ? 0.0 : b.w / sqrt(drSq);
        }
    }
    double e[3] = {0.0, 0.0, 0.0};
    if (valid) {
        const double m = mass[i];
        e[0] = 0.5 * m * (vx[i] * vx[i] + vy[i] * vy[i] + vz[i] * vz[i]);
        e[1] = -0.5 * m * phi;
        e[2] = pot.enabled ? m * nb_ext_potential(pot, x0, y0, z0) : 0.0;
    }
    for (int c = 0; c < 3; ++c) {
        double v = e[c];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(NB_FULL_MASK, v, o);
        if ((threadIdx.x & 31) == 0) red[c][threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double v = 0.0;
        for (int w = 0; w < EXACT_TILE / 32; ++w) v += red[threadIdx.x][w];
        atomicAdd(out + threadIdx.x, v);
    }
}

void nb_launch_energy(const double* px, const double* py, const double* pz, const double* vx,
                      const double* vy, const double* vz, const double* mass, int n, double eps2,
                      const NbPot& pot, double* out, cudaStream_t s)
{
    cudaMemsetAsync(out, 0, 3 * sizeof(double), s);
    if (n <= 0) return;
    k_energy<<<(n + EXACT_TILE - 1) / EXACT_TILE, EXACT_TILE, 0, s>>>(px, py, pz, vx, vy, vz, mass,
                                                                     n, eps2, pot, out);
    nb_count_launch();
}

// FMA throughput probe: independent FMA chains per thread (the denominator of the walk's
// pipe roofline).  fp64 selects DFMA or FFMA.
template <typename T>
__global__ void k_fma_probe(T* out, int iters, T seed)
{
    T a0 = seed + (T) threadIdx.x, a1 = a0 + (T) 1, a2 = a0 + (T) 2, a3 = a0 + (T) 3;
    T a4 = a0 + (T) 4, a5 = a0 + (T) 5, a6 = a0 + (T) 6, a7 = a0 + (T) 7;
    const T m = (T) 0.999999, c = (T) 1e-7;
    for (int k = 0; k < iters; ++k) {
        a0 = fma(a0, m, c); a1 = fma(a1, m, c); a2 = fma(a2, m, c); a3 = fma(a3, m, c);
        a4 = fma(a4, m, c); a5 = fma(a5, m, c); a6 = fma(a6, m, c); a7 = fma(a7, m, c);
    }
    const T s = ((a0 + a1) + (a2 + a3)) + ((a4 + a5) + (a6 + a7));
    if (s == (T) -1) out[0] = s;   // keeps the chains live
}

__global__ void k_ext_only(const double* __restrict__ pos, double* __restrict__ acc, int n, NbPot pot)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double ex, ey, ez;
        nb_ext_accel(pot, pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], ex, ey, ez);
        acc[3 * i] = ex; acc[3 * i + 1] = ey; acc[3 * i + 2] = ez;
    }
}

// ---- host launchers ----

void nb_launch_pack_walk(const NbTreeBuffers& b, int capNodes, bool slots, cudaStream_t s)
{
    k_pack_walk<<<min((capNodes + 255) / 256, 4096), 256, 0, s>>>(
        b.nodePM, b.nodeCrit, b.nodeLink, slots ? b.nodeRange : nullptr, b.nodeQuad, b.walkRec, b.sc);
    nb_count_launch();
}

// Form 0's kernel, and where it is the team walk and the fastest form without timing.
int nb_walk_shared(int n, double theta)
{
    const double least = fmin(TEAM_THETA, (n - 9000) / 85000.0);
    return n <= TEAM_AUTO_MONO || (n <= TEAM_MAX_BODIES && theta >= least) ? NB_WALK_TEAM
                                                                          : NB_WALK_UNION;
}
bool nb_walk_team_auto(int n, int useQuad, double theta)
{
    if (useQuad && n <= TEAM_AUTO_MONO) return theta >= TEAM_SMALL_THETA;
    return n <= (useQuad ? TEAM_AUTO_QUAD : TEAM_AUTO_MONO) && theta >= TEAM_THETA;
}

// A batch's kernel.  Its bodies in all fill the chip, but a body meets only those of its dwarf, of
// which a small dwarf's walk takes most whatever the angle.  Measured: steps of batches of 40,000 to
// 3,000,000 bodies in dwarfs of 200 to 100,000.
//   * The team walk at sizes that leave the chip idle, as for single systems, but not where nearly
//     every body is met: between its lines it needs bodies-a-dwarf x theta^2 >= 300 (20,000 bodies
//     in all, early load -> team: 100 dwarfs, theta 1 0.310 -> 0.332 ms; 20, 1 0.440 -> 0.436, 0.5 0.687 ->
//     0.705; 10, 0.5 0.926 -> 0.895, 0.2 1.39 -> 1.70; 2, 0.2 5.19 -> 4.76, 0.05 6.37 -> 8.76).
//   * The union where walks share most of their nodes: theta^5 x bodies-a-dwarf <= 440 with a full
//     chip (own path -> union: 20 dwarfs of 10,000, theta 0.6 3.14 -> 3.24, 0.5 4.36 -> 4.01, 0.3 10.2 ->
//     7.20; 100 of 2,000, 0.85 1.34 -> 1.37, 0.7 1.66 -> 1.59, 0.5 2.44 -> 2.02), 990 from 524,288 bodies in
//     all (1,000 of 1,000: 1.0 3.39 -> 3.58, 0.85 3.89 -> 3.86, 0.5 6.17 -> 5.06; 100 of 10,000: 0.7 8.72 ->
//     8.96, 0.6 11.6 -> 11.4; 16 of 64,000: 0.5 22.6 -> 22.2, 0.4 37.1 -> 32.8), less below 131,072,
//     where the longer walk's latency shows (early load -> union: 40 of 1,000, 0.7 0.596 -> 0.613, 0.5
//     0.746 -> 0.709; 1 of 40,000, 0.3 5.8 -> 7.1), and less without quadrupoles (own path -> union: 20
//     of 10,000, 0.5 2.84 -> 2.87, 0.4 4.22 -> 3.77; 100 of 10,000, 0.7 5.70 -> 6.30, 0.5 10.6 -> 10.3).
//     Not where a walk is nearly all bodies (early load -> union: 50 dwarfs of 1,000, 0.1 0.907 -> 1.18)
//     nor for the smallest dwarfs (80 of 500: 0.3 0.557 -> 0.594; 200 of 200: 0.5 0.361 -> 0.430).
//   * Else own paths, with the early load while few warps are resident (own -> early, theta 0.7: 65,536
//     bodies 1.04 -> 0.97, 80,000 1.11 -> 1.04, 96,758 1.19 -> 1.20, 131,072 1.33 -> 1.57).
constexpr int EARLY_MAX_BODIES = 81920;
constexpr int UNION_FULL_BODIES = 131072, UNION_MANY_BODIES = 524288;
int nb_walk_batch(int n, int dwarfs, int useQuad, double theta)
{
    const double mean = (double) n / dwarfs, cells = mean * (theta * theta);
    if (n <= TEAM_AUTO_MONO && theta >= 0.02) return NB_WALK_TEAM;
    if (useQuad && n <= TEAM_AUTO_QUAD && cells >= 300.0) return NB_WALK_TEAM;
    const double full = n < UNION_FULL_BODIES ? (double) n / UNION_FULL_BODIES : 1.0;
    const double shared = (theta * theta) * (theta * cells);
    const bool many = n >= UNION_MANY_BODIES;
    const double limit = useQuad ? (many ? 990.0 : 440.0 * (full * full))
                                 : (many ? 1040.0 : full >= 0.75 ? 104.0 * (full * full) : -1.0);
    if (mean >= 600.0 && cells * full >= 8.0 && shared <= limit && (useQuad || theta <= 0.5))
        return NB_WALK_UNION;
    return n <= EARLY_MAX_BODIES ? NB_WALK_EARLY : NB_WALK_LANES;
}

void nb_launch_walk_fp64(const NbTreeBuffers& b, int capNodes, const NbWalkParams& wp,
                         const NbPot& pot, bool count, cudaStream_t s, const NbForest* forest,
                         int kernel)
{
    const int warps = (wp.n + 31) / 32;
    const int blocks = (warps * 32 + WALK_THREADS - 1) / WALK_THREADS;
    if (blocks <= 0) return;
    nb_launch_pack_walk(b, capNodes, true, s);
    const NbForest f = forest ? *forest : NbForest{nullptr, nullptr, 0};
    const int perTeamBlock = TEAM_BODIES * WALK_THREADS / 32;
    const int teamBlocks = (wp.n + perTeamBlock - 1) / perTeamBlock;
#define NB_LANES_ARGS b.walkRec, b.sort.idxA, b.px, b.py, b.pz, b.ax, b.ay, b.az, wp, b.sc, f
#define NB_TEAM_ARGS                                                                          \
    b.walkRec, (const int*) b.walkKids, b.sort.idxA, b.px, b.py, b.pz, b.ax, b.ay, b.az, wp, b.sc, f
#define NB_TEAM(COUNT, FOREST) k_walk_fp64_team<COUNT, FOREST><<<teamBlocks, WALK_THREADS, 0, s>>>(NB_TEAM_ARGS)
#define NB_LANES(COUNT, FOREST, PATH)                                                         \
    k_walk_fp64_lanes<COUNT, FOREST, PATH><<<blocks, WALK_THREADS, 0, s>>>(NB_LANES_ARGS)
#define NB_WALK(COUNT, FOREST)                                                                \
    do {                                                                                      \
        if (kernel == NB_WALK_TEAM) NB_TEAM(COUNT, FOREST);                                   \
        else if (kernel == NB_WALK_EARLY) NB_LANES(COUNT, FOREST, LANES_EARLY);               \
        else if (kernel == NB_WALK_UNION) NB_LANES(COUNT, FOREST, LANES_UNION);               \
        else NB_LANES(COUNT, FOREST, LANES_OWN);                                              \
    } while (0)
    if (forest) NB_WALK(false, true);               // a batch does not count
    else if (count) NB_WALK(true, false);
    else NB_WALK(false, false);
#undef NB_WALK
#undef NB_LANES
#undef NB_TEAM
#undef NB_LANES_ARGS
#undef NB_TEAM_ARGS
    nb_count_launch();
    nb_launch_body_epilogue(b.px, b.py, b.pz, b.ax, b.ay, b.az, b.vx, b.vy, b.vz, wp, pot, b.sc, 0, s,
                            forest);
}

void nb_launch_direct_fp64(const double* px, const double* py, const double* pz,
                           const double* mass, double* ax, double* ay, double* az, double* vx,
                           double* vy, double* vz, const NbWalkParams& wp, const NbPot& pot,
                           NbScalars* sc, int numSMs, cudaStream_t s)
{
    if (wp.n <= 0) return;
    // the most lanes a body that leave one warp a scheduler (4 an SM): past that the warps take
    // turns, and sharing a body only adds the shuffles
    const int slots = 32 * 4 * numSMs;
    const int H = 4ll * wp.n <= slots ? 4 : 2ll * wp.n <= slots ? 2 : 1;
    const int blocks = (wp.n + 32 / H - 1) / (32 / H);
    if (H == 4) k_direct_fp64<4><<<blocks, 32, 0, s>>>(px, py, pz, mass, ax, ay, az, wp);
    else if (H == 2) k_direct_fp64<2><<<blocks, 32, 0, s>>>(px, py, pz, mass, ax, ay, az, wp);
    else k_direct_fp64<1><<<blocks, 32, 0, s>>>(px, py, pz, mass, ax, ay, az, wp);
    nb_count_launch();
    nb_launch_body_epilogue(px, py, pz, ax, ay, az, vx, vy, vz, wp, pot, sc, numSMs, s, nullptr);
}

void nb_launch_ext_only(const double* dpos, double* dacc, int n, const NbPot& pot, cudaStream_t s)
{
    if (n <= 0) return;
    k_ext_only<<<(n + 255) / 256, 256, 0, s>>>(dpos, dacc, n, pot);
    nb_count_launch();
}

void nb_launch_direct_sample(const double* px, const double* py, const double* pz,
                             const double* mass, int n, const int* targets, int count,
                             double eps2, double* out, cudaStream_t s)
{
    if (count <= 0) return;
    k_direct_sample<<<(count + EXACT_TILE - 1) / EXACT_TILE, EXACT_TILE, 0, s>>>(
        px, py, pz, mass, n, targets, count, eps2, out);
    nb_count_launch();
}

// Returns the achieved FMA rate in TFLOP/s (2 flops per FMA) over blocks x 256 threads.
double nb_fma_probe(int fp64, int numSMs, cudaStream_t s)
{
    const int threads = 256, blocks = numSMs * 8, iters = 1 << 14;
    void* out = nullptr;
    cudaMalloc(&out, 16);
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    double best = 0.0;
    for (int rep = 0; rep < 3; ++rep) {
        cudaEventRecord(e0, s);
        if (fp64) k_fma_probe<double><<<blocks, threads, 0, s>>>((double*) out, iters, 1.0);
        else k_fma_probe<float><<<blocks, threads, 0, s>>>((float*) out, iters, 1.0f);
        cudaEventRecord(e1, s);
        cudaEventSynchronize(e1);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        const double flops = 2.0 * 8.0 * (double) iters * threads * (double) blocks;
        if (ms > 0.f) best = fmax(best, flops / (ms * 1e-3) / 1e12);
    }
    nb_count_launch(3);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(out);
    return best;
}
