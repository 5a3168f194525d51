// Device-side Sibson (natural-neighbour) query: one cooperative group of G
// lanes per query.
//
// Per query (natinterp3d's getWeightsSingleQueryIF, natural_insertionfree.c:591-738):
//   1. locate   seed tet = the tet whose centroid is nearest to the query, as
//               natinterp3d's k-d tree returns it (delaunay.c:392-395), found in
//               a uniform grid of centroids (an octree where the grid is too
//               coarse); then
//               natinterp3d's visibility walk (delaunay.c:398-405), the four
//               face tests of a step on 4 lanes
//   2. cavity   the connected set of tets whose circumsphere strictly contains
//               the query (inspherefast > 0, natural_insertionfree.c:502-530),
//               found breadth-first with all lanes testing in parallel; a
//               single-lane integer replay then recovers natinterp3d's LIFO
//               visiting order, which fixes the column order and the
//               floating-point summation order of every weight
//   3. boundary faces and natural neighbours in first-seen order (:559-584)
//   4. signed Voronoi-subcell volumes: +cavity-tet terms (:642-676) and
//      -virtual-tet terms (:681-719), added to each neighbour's sum in
//      natinterp3d's accumulation order: the split rows (split_row_body) store
//      a neighbour's terms next to each other and one lane adds them, the fused
//      and large rows fold a term per lane
//   5. normalisation (:721-737)
// Tet circumcentres and face circumcentres are read from the per-mesh cache
// (computed with the same formulas and argument orders); a face shared by two
// cavity tets uses the circumcentre computed from the tet natinterp3d visits
// first, as natinterp3d's face cache does (:233-253).
//
// Predicates.  natinterp3d evaluates orient3dfast / inspherefast and uses their
// signs as they come (predicates.c:1687, 3301); that is the default here
// (PRED_FAST).  Two more modes per mesh: PRED_AUDIT keeps those signs and
// counts every evaluation whose fast value the static error bound cannot
// certify ("uncertain"), and those whose decision the exact sign would change
// ("flipped"); PRED_EXACT decides by the exact sign.  The row routine comes in
// three variants: PM_PLAIN (fast signs only), PM_FILTER (fast kernel of the
// non-default modes: certified signs only, the row is handed to the
// large-row kernel at the first uncertain evaluation that matters) and
// PM_RESOLVE (large-row kernel: uncertain evaluations are resolved exactly,
// one lane at a time, in a per-group global scratch, and counted).
#pragma once
#include <limits.h>
#include <stddef.h>
#include <stdint.h>

#include <type_traits>

#include "nif_exact.h"
#include "nif_geometry.cuh"

namespace nif {

// per-row status codes (stored as int8)
constexpr int ST_OK = 0;
constexpr int ST_WALK = 1;       // walk step limit
constexpr int ST_CAPACITY = 2;   // per-query capacity of this kernel exceeded
constexpr int ST_UNCERTAIN = 4;  // a predicate needs exact evaluation (PM_FILTER only)

// predicate modes of a mesh (MeshView::pmode)
constexpr int PRED_FAST = 0;
constexpr int PRED_AUDIT = 1;
constexpr int PRED_EXACT = 2;

// row-routine variants
constexpr int PM_PLAIN = 0;
constexpr int PM_FILTER = 1;
constexpr int PM_RESOLVE = 2;

constexpr int WALK_LIMIT = 1 << 16;
constexpr int SEED_STEP_LIMIT = 1 << 16;  // node and leaf visits of one nearest-centroid search
constexpr int OCT_BITS = 20;              // centroid code: cell bits per axis
constexpr int OCT_KMAX = 10;              // octree node levels below the root (6 code bits each)
constexpr int OCT_SPLIT = 128;            // a node with more centroids than this has children

struct __align__(32) d4 {
    double x, y, z, w;
};

// Resident mesh (device pointers) and its parameters, passed by value.
struct MeshView {
    const d4 *__restrict__ vtx;        // [nv] x, y, z, 0
    const int4 *__restrict__ tv;       // [nt] vertex ids
    const int4 *__restrict__ tn;       // [nt] neighbour tets (-1 = none)
    const uint32_t *__restrict__ tinfo;// [nt] bit0: orient3dfast(p0..p3) > 0; bit1: that sign is
                                       // uncertain; bit2: exact orient3d(p0..p3) > 0;
                                       // bits 8+2j: mirror slot of face j
    const d4 *__restrict__ tcc;        // [nt] tet circumcentre; w: see sphere_side
    const d4 *__restrict__ fcc;        // [nt*4] circumcentre of the face opposite p[i]
    const d4 *__restrict__ corner;     // [nt*16] corner terms (corner_term), or null
    // Tet centroids, (p0 + p1 + p2 + p3) / 4 per axis as natinterp3d's
    // constructor computes them for its k-d tree (delaunay.c:151-157), sorted
    // by a 60-bit Morton code of their cell in a 2^20 grid per axis over the
    // bounding box of all vertices: x, y, z and the tet id (as a double).
    // An octree over that order: node k spans the centroids of one octree
    // cell, two octree levels (64 sub-cells, one 6-bit code digit) per node
    // level.  onode[2 k] = float box lo (w: first child node, or first
    // centroid of a leaf, as int bits); onode[2 k + 1] = box hi (w: number of
    // children, or minus the centroid count of a leaf); omask[k] = the
    // digits of the children present.  Boxes are rounded outwards.
    const d4 *__restrict__ cs;
    const float4 *__restrict__ onode;
    const unsigned long long *__restrict__ omask;
    double olo[3], osc[3];             // cell of x: floor((x - olo) * osc), clamped
    double oext;                       // largest extent of the code space
    int n;                             // data vertices (ids >= n are super-simplex vertices)
    int nv, nt;
    int pmode;                         // PRED_*
    int small;                         // some tet is flat_sized
    // Uniform grid over the data bounding box, gdim cells per axis (cell of x
    // along axis a: floor((x - glo) * ginv), clamped), about two centroids a
    // cell: the centroids of cell k are gitems[gstart[k] .. gstart[k + 1]),
    // x, y, z and the tet id (as a double), in no particular order.  The
    // seed search reads it first; query bucketing normalises by the same box.
    const int *__restrict__ gstart;
    const d4 *__restrict__ gitems;
    int gdim[3];
    double glo[3], ginv[3];
    double gh[3];                      // cell size, 1 / ginv
    double gext;                       // largest extent of the grid (margins)
};

__device__ __forceinline__ int comp(const int4 &v, int i) {
    return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w));
}

// getFaceVerticies3 (delaunay.c:444-467): face f = (p[a], p[b], p[c]) lies
// opposite p[3-f] and is shared with neighbour s[f].
__device__ __forceinline__ int face_vslot(int f, int j) {
    constexpr unsigned bits = (0u | 1u << 2 | 2u << 4) | ((3u | 1u << 2 | 0u << 4) << 6) |
                              ((0u | 2u << 2 | 3u << 4) << 12) | ((3u | 2u << 2 | 1u << 4) << 18);
    return (bits >> (6 * f + 2 * j)) & 3;
}

__device__ __forceinline__ dv3 vload(const MeshView &M, int vid) {
    const d4 v = M.vtx[vid];
    return dv3{v.x, v.y, v.z};
}

__device__ __forceinline__ void prefetch_l2(const void *p) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

__device__ __forceinline__ dv3 cload(const d4 *p) {
    const d4 v = *p;
    return dv3{v.x, v.y, v.z};
}

// Squared distance between a tet centroid and q as natinterp3d's k-d tree
// evaluates it: dist_sq = 0; dist_sq += SQ(node->pos[i] - pos[i]) for
// i = 0, 1, 2 (kdtree.c:411-414; 0 + a == a exactly).
__device__ __forceinline__ double kd_dist2(const d4 &c, const dv3 &q) {
    const double dx = fsub(c.x, q.x), dy = fsub(c.y, q.y), dz = fsub(c.z, q.z);
    return fadd(fadd(fmul(dx, dx), fmul(dy, dy)), fmul(dz, dz));
}

// A lower bound of kd_dist2 over every centroid inside the box [lo, hi]:
// per axis the rounded distance to the nearer face (0 inside), squared and
// summed in the same order.  Rounding is monotonic, so no centroid in the
// box evaluates below it.
__device__ __forceinline__ double box_dist2(const float4 &lo, const float4 &hi, const dv3 &q) {
    auto axis = [](double x, float l, float h) {
        return x < (double)l ? fsub((double)l, x) : (x > (double)h ? fsub(x, (double)h) : 0.0);
    };
    const double ax = axis(q.x, lo.x, hi.x), ay = axis(q.y, lo.y, hi.y), az = axis(q.z, lo.z, hi.z);
    return fadd(fadd(fmul(ax, ax), fmul(ay, ay)), fmul(az, az));
}

// Lane helpers for a group of G consecutive lanes of a warp.
template <int G>
struct Grp {
    unsigned mask;  // warp-lane mask of the group
    int lane;       // lane within the group
    int base;       // first warp lane of the group
    __device__ __forceinline__ Grp() {
        const int wl = threadIdx.x & 31;
        lane = wl % G;
        base = wl - lane;
        mask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << base);
    }
    __device__ __forceinline__ unsigned local(unsigned m) const {
        return (G == 32) ? m : ((m >> base) & ((1u << G) - 1u));
    }
    __device__ __forceinline__ unsigned ballot(bool p) const { return local(__ballot_sync(mask, p)); }
    __device__ __forceinline__ bool any(bool p) const { return __any_sync(mask, p); }
    __device__ __forceinline__ unsigned lt() const { return (1u << lane) - 1u; }
    __device__ __forceinline__ void sync() const { __syncwarp(mask); }
    __device__ __forceinline__ unsigned match(int v) const { return local(__match_any_sync(mask, v)); }
    __device__ __forceinline__ int shfl(int v, int src) const { return __shfl_sync(mask, v, src, G); }
    __device__ __forceinline__ double shfl(double v, int src) const {
        return __shfl_sync(mask, v, src, G);
    }
    __device__ __forceinline__ int shfl_xor(int v, int off) const {
        return __shfl_xor_sync(mask, v, off, G);
    }
    __device__ __forceinline__ double shfl_xor_d(double v, int off) const {
        return __shfl_xor_sync(mask, v, off, G);
    }
};

__device__ __forceinline__ unsigned long long spread3_64(unsigned v) {  // 20 bits -> every third bit
    unsigned long long x = v & 0xfffffu;
    x = (x | x << 32) & 0x1f00000000ffffull;
    x = (x | x << 16) & 0x1f0000ff0000ffull;
    x = (x | x << 8) & 0x100f00f00f00f00full;
    x = (x | x << 4) & 0x10c30c30c30c30c3ull;
    x = (x | x << 2) & 0x1249249249249249ull;
    return x;
}

// cell coordinates (clamped) and 60-bit Morton code of a point in the
// centroid code space
__device__ __forceinline__ unsigned long long oct_code(const MeshView &M, const dv3 &p, int ix[3]) {
    const double c[3] = {p.x, p.y, p.z};
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const double f = (c[a] - M.olo[a]) * M.osc[a];
        ix[a] = f > 0.0 ? (f < (double)((1 << OCT_BITS) - 1) ? (int)f : (1 << OCT_BITS) - 1) : 0;
    }
    return spread3_64(ix[0]) | (spread3_64(ix[1]) << 1) | (spread3_64(ix[2]) << 2);
}

// True when every point within sqrt(best) of q lies inside q's octree cell
// at octree level 2 m (margins absorb the rounding of the cell bounds and of
// the centroids' own cell assignment).
__device__ __forceinline__ bool ball_in_cell(const MeshView &M, const dv3 &q, double best,
                                             const int ix[3], int m) {
    if (!(best < INFINITY)) return false;
    const double r = sqrt(best) * (1.0 + 1e-9) + 1e-9 * M.oext;
    const double c[3] = {q.x, q.y, q.z};
    const int sh = OCT_BITS - 2 * m;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const double w = (double)(1 << sh) / M.osc[a];
        const double lo = M.olo[a] + (double)(ix[a] >> sh) * w;
        if (!(c[a] - r > lo && c[a] + r < lo + w)) return false;
    }
    return true;
}

// The tet whose centroid is nearest to q under kd_dist2, ties to the lowest
// tet id: the seed natinterp3d's k-d tree returns (kd_nearest3_data,
// kdtree.c:543-564).  Its pruning never skips a strictly nearer centroid, so
// it returns a minimiser of the same rounded distance; among exactly equal
// distances its visiting order decides, here the lowest id.
// Bottom-up over the octree, one lane per child (two per lane for 64):
//   1. descend along q's own code to the deepest node holding q's cell;
//   2. search that node's subtree;
//   3. walk back up: stop as soon as the ball of radius sqrt(best) around q
//      lies inside the cell just searched (octree cells are disjoint, so no
//      other centroid can be nearer); otherwise search the parent's other
//      children.
// A subtree search is depth-first, entering a child while its box bound is
// <= best (an equal distance may still lose to a lower id).  stk: 64 ints of
// group scratch (the descent path and the search frames); every lane keeps
// the same control state and lane 0 stores it.  Bounded by SEED_STEP_LIMIT
// visits (then the best centroid so far, a valid seed for the walk).
template <int G>
__device__ int nearest_centroid(const MeshView &M, const dv3 q, const Grp<G> &g, int *stk) {
    static_assert(G == 32, "two children of a 64-wide node per lane");
    int *path = stk;        // [OCT_KMAX + 1]
    int *frm = stk + 16;    // 3 ints a frame: node, pending children (lo, hi word)
    int ix[3];
    const unsigned long long code = oct_code(M, q, ix);
    int node = 0, depth = 0;
    if (g.lane == 0) path[0] = 0;
    for (; depth < OCT_KMAX; depth++) {
        const int nch = __float_as_int(M.onode[2 * node + 1].w);
        if (nch <= 0) break;
        const unsigned long long mask = M.omask[node];
        const int dg = (int)((code >> (6 * (OCT_KMAX - 1 - depth))) & 63ull);
        if (!((mask >> dg) & 1ull)) break;
        node = __float_as_int(M.onode[2 * node].w) + __popcll(mask & ((1ull << dg) - 1ull));
        if (g.lane == 0) path[depth + 1] = node;
    }
    g.sync();
    double best = INFINITY;
    int bid = INT_MAX;
    int steps = 0;
    // centroids [a, a + n) of a leaf
    auto leaf_pass = [&](int a, int n) {
        for (int k0 = a; k0 < a + n; k0 += G) {
            const int k = k0 + g.lane;
            double d = INFINITY;
            int id = INT_MAX;
            if (k < a + n) {
                const d4 e = M.cs[k];
                d = kd_dist2(e, q);
                id = (int)e.w;
            }
            const bool better = d < best || (d == best && id < bid);
            if (g.any(better)) {
                double bd = better ? d : best;
                int bi = better ? id : bid;
#pragma unroll
                for (int off = G / 2; off > 0; off >>= 1) {
                    const double od = g.shfl_xor_d(bd, off);
                    const int oi = g.shfl_xor(bi, off);
                    if (od < bd || (od == bd && oi < bi)) {
                        bd = od;
                        bi = oi;
                    }
                }
                best = bd;
                bid = bi;
            }
        }
    };
    // every centroid under node r, except under its child `skip`
    auto subtree = [&](int r, int skip) {
        {
            const float4 lo = M.onode[2 * r], hi = M.onode[2 * r + 1];
            if (__float_as_int(hi.w) <= 0) {
                ++steps;
                leaf_pass(__float_as_int(lo.w), -__float_as_int(hi.w));
                return;
            }
        }
        int sp = 1;
        if (g.lane == 0) frm[0] = r;
        bool fresh = true;
        unsigned long long pend = 0;
        while (sp > 0 && steps < SEED_STEP_LIMIT) {
            ++steps;
            g.sync();
            const int nd = frm[3 * (sp - 1)];
            if (!fresh)
                pend = (unsigned long long)(unsigned)frm[3 * (sp - 1) + 1] |
                       ((unsigned long long)(unsigned)frm[3 * (sp - 1) + 2] << 32);
            const int first = __float_as_int(M.onode[2 * nd].w);
            const int nch = __float_as_int(M.onode[2 * nd + 1].w);
            // box bounds of the children lane and lane + 32
            double d0 = INFINITY, d1 = INFINITY;
            const int c0 = first + g.lane, c1 = first + 32 + g.lane;
            if (g.lane < nch && c0 != skip) d0 = box_dist2(M.onode[2 * c0], M.onode[2 * c0 + 1], q);
            if (32 + g.lane < nch && c1 != skip) d1 = box_dist2(M.onode[2 * c1], M.onode[2 * c1 + 1], q);
            auto within = [&]() {
                return (unsigned long long)g.ballot(d0 <= best) |
                       ((unsigned long long)g.ballot(d1 <= best) << 32);
            };
            pend = fresh ? within() : (pend & within());
            fresh = false;
            bool pushed = false;
            while (pend && steps < SEED_STEP_LIMIT) {
                const int c = __ffsll((long long)pend) - 1;
                pend &= pend - 1ull;
                const int ch = first + c;
                const float4 clo = M.onode[2 * ch], chi = M.onode[2 * ch + 1];
                ++steps;
                if (__float_as_int(chi.w) <= 0) {
                    leaf_pass(__float_as_int(clo.w), -__float_as_int(chi.w));
                    pend &= within();  // the same children, against the improved best
                } else {
                    if (g.lane == 0) {
                        frm[3 * (sp - 1) + 1] = (int)(unsigned)pend;
                        frm[3 * (sp - 1) + 2] = (int)(unsigned)(pend >> 32);
                        frm[3 * sp] = ch;
                    }
                    ++sp;
                    fresh = true;
                    pushed = true;
                    break;
                }
            }
            if (!pushed) --sp;
        }
        g.sync();
    };
    subtree(node, -1);
    for (int l = depth - 1; l >= 0; l--) {
        if (ball_in_cell(M, q, best, ix, l + 1)) break;
        subtree(path[l], path[l + 1]);
    }
    return bid == INT_MAX ? 0 : bid;
}

constexpr int GRID_DENSE = 256;  // centroids in a search block beyond which the octree searches
constexpr int GRID_RMAX = 3;     // largest block radius (cells) the grid search widens to

// The nearest tet centroid to q (same distance and ties as nearest_centroid)
// from the uniform grid: the centroids of the cells within Chebyshev radius
// r of q's cell, one lane per cell, r = 1 first; done once the best distance
// is below the distance from q to the searched block's open sides (sides on
// the grid's boundary are closed: centroids beyond them are clamped into the
// boundary cells, which have been searched).  Returns -1 where the block
// holds more than GRID_DENSE centroids or r would exceed GRID_RMAX: the
// octree search takes over there (clustered data, far-away queries).
template <int G>
__device__ int grid_nearest(const MeshView &M, const dv3 q) {
    static_assert(G == 32, "one lane per cell of a 3x3x3 block");
    const double c[3] = {q.x, q.y, q.z};
    double f[3];  // q's position in cell units
    int ic[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        f[a] = (c[a] - M.glo[a]) * M.ginv[a];
        ic[a] = f[a] > 0.0 ? (f[a] < (double)(M.gdim[a] - 1) ? (int)f[a] : M.gdim[a] - 1) : 0;
    }
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    double best = INFINITY;
    int bid = INT_MAX;
    for (int r = 1; r <= GRID_RMAX; r++) {
        const int w = 2 * r + 1, ncell = w * w * w;
        // this round's cells: the 27 of the 3x3x3 block, then the shell at
        // Chebyshev radius r
        int total = 0;
        for (int k0 = 0; k0 < ncell; k0 += 32) {
            const int k = k0 + lane;
            int a = 0, b = 0;
            int dx, dy, dz;
            bool take;
            if (r == 1) {
                dx = lane % 3 - 1, dy = (lane / 3) % 3 - 1, dz = lane / 9 - 1;
                take = lane < 27;
            } else {
                dx = k % w - r, dy = (k / w) % w - r, dz = k / (w * w) - r;
                take = k < ncell && max(abs(dx), max(abs(dy), abs(dz))) == r;
            }
            const int x = ic[0] + dx, y = ic[1] + dy, z = ic[2] + dz;
            if (take && x >= 0 && y >= 0 && z >= 0 && x < M.gdim[0] && y < M.gdim[1] && z < M.gdim[2]) {
                const int cell = (z * M.gdim[1] + y) * M.gdim[0] + x;
                a = M.gstart[cell];
                b = M.gstart[cell + 1];
            }
            total += __reduce_add_sync(full, b - a);
            if (total > GRID_DENSE) return -1;
            for (int i = a; i < b; i++) {
                const d4 e = M.gitems[i];
                const double d = kd_dist2(e, q);
                const int id = (int)e.w;
                if (d < best || (d == best && id < bid)) {
                    best = d;
                    bid = id;
                }
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const double od = __shfl_xor_sync(full, best, off);
            const int oi = __shfl_xor_sync(full, bid, off);
            if (od < best || (od == best && oi < bid)) {
                best = od;
                bid = oi;
            }
        }
        // distance from q to the block's open sides (not on the grid's boundary)
        double lb = INFINITY;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            if (ic[a] - r > 0) lb = fmin(lb, (f[a] - (double)(ic[a] - r)) * M.gh[a]);
            if (ic[a] + r < M.gdim[a] - 1) lb = fmin(lb, ((double)(ic[a] + r + 1) - f[a]) * M.gh[a]);
        }
        if (lb == INFINITY) return bid == INT_MAX ? -1 : bid;  // the block covers the grid
        const double m = lb - 1e-9 * M.gext;
        if (bid != INT_MAX && m > 0.0 && best < m * m * (1.0 - 1e-12)) return bid;
    }
    return -1;
}

// Which side of tet t's circumsphere q lies on, from the cached circumcentre c
// and squared radius w: 1 inside, -1 outside, 0 where this does not decide.  A
// decision has the sign of natinterp3d's inspherefast and lies outside its
// error bound, because prep_sphere gives only those tets a radius for which
//   6V |d2 - w| > 2 E  for |d2 - w| > SPHERE_REL w and d2 < SPHERE_FAR w,
// d2 = |q - c|^2, E the static error bound of inspherefast; the others have
// w = NaN, which decides nothing.  Nine FP64 operations on one 32-byte record
// for some 80 on four vertices behind the tet's vertex record (the cavity pass
// of 2M rows on 200k keys: 4.55 to 3.3 ms).
constexpr double SPHERE_REL = 1e-6, SPHERE_FAR = 1e4;
__device__ __forceinline__ int sphere_side(const d4 &c, const dv3 &q) {
    const double x = q.x - c.x, y = q.y - c.y, z = q.z - c.z;
    const double d2 = x * x + y * y + z * z;
    const double f = d2 - c.w;
    if (!(fabs(f) > SPHERE_REL * c.w && d2 < SPHERE_FAR * c.w)) return 0;
    return f < 0.0 ? 1 : -1;
}

// The w of sphere_side for a tet with circumcentre c and orientation
// determinant o (6V up to its error), NaN where it cannot be relied on.
//
// With R the radius, s >= every |v_i - q| and V the volume, the exact insphere
// determinant is 6V (|q - C|^2 - R^2), C and R exact, and inspherefast's error
// is at most E <= 24 (16 + 224 eps) eps s^5 < 4.3e-14 s^5 (its permanent: four
// lifts of at most s^2 times six products of at most s^3).  f(q) = |q - c|^2 - w
// and the exact |q - C|^2 - R^2 differ by an affine function that is f(v_i) at
// the vertices: by at most rho = max |f(v_i)| times the sum of |barycentric
// coordinates|, each at most s^3 / 6V.  Evaluating f rounds by less than
// 8 eps (d2 + w).  So a decision is right, and certified, when
//   |f| > 8 eps (d2 + w) + (4 rho s^3 + 8.6e-14 s^5) / 6V.
// For d2 <= 4 w, s <= 3.01 R, the right side is below
// 5e-15 w + (110 rho R^3 + 2.2e-11 R^5) / 6V, which is held to SPHERE_REL w / 2.
// For 4 w < d2 < SPHERE_FAR w, s <= 1.51 d and |f| > 0.75 d2, and with those
// limits on rho and 1 / 6V the right side is below 2e-15 d2 +
// (14 rho + 6.8e-13 d2) d^3 / 6V < 0.1 d2.
__device__ __forceinline__ double prep_sphere(const dv3 &c, const dv3 &p0, const dv3 &p1, const dv3 &p2,
                                              const dv3 &p3, double o, bool uncertain) {
    auto dist2 = [&](const dv3 &p) { return vdot(vsub(p, c), vsub(p, c)); };
    const double w = dist2(p0);
    const double rho = fmax(fmax(fabs(dist2(p1) - w), fabs(dist2(p2) - w)), fabs(dist2(p3) - w)) + 4e-15 * w;
    const double r = sqrt(w), v6 = 0.9 * fabs(o);
    const bool ok = !uncertain && w > 1e-60 && w < 1e60 &&
                    110.0 * rho * r * w + 2.2e-11 * r * w * w <= 0.4e-6 * w * v6;
    return ok ? w : NAN;
}

// Squared circumradius of the located tet below which a row goes to k_rows_general
// straight away: some triangle of its virtual tets will be below natinterp3d's
// threshold, twice the area 1e-15, so that k_rows_volume would give the row up
// after most of its work.  50k uniform keys, 200k queries, median squared radius 9e-15
// / 5e-15 / 2.3e-15 / 6e-16 / 6e-18 (keys 1e-7 to 3e-9 apart), us a call: with
// k_rows_volume first 1,410 / 1,575 / 2,090 / 2,380 / 2,372, straight to the general
// kernel 1,892 / 1,892 / 1,930 / 1,964 / 1,933, by this limit 1,422 / 1,620 / 1,980 /
// 1,962 / 1,930 (and 2,176 / 2,196 / 2,239 / 2,272 / 2,219 with one kernel for both).
constexpr double FLAT_SPHERE = 4e-15;

// Whether a tet is so small that its row is for k_rows_general (FLAT_SPHERE): by
// its cached radius w, or where it has none by its edge p0 p1.
__device__ __forceinline__ bool flat_sized(double w, const dv3 &p0, const dv3 &p1) {
    if (!(w >= 0.0)) w = vdot(vsub(p0, p1), vsub(p0, p1));
    return w < FLAT_SPHERE;
}
__device__ __forceinline__ bool flat_sized(const MeshView &M, int t) {
    const int4 p = M.tv[t];
    return flat_sized(M.tcc[t].w, vload(M, p.x), vload(M, p.y));
}

// Per-group scratch.  The first union member is live during the cavity
// search, the second only during the single-lane replay of natinterp3d's
// visiting order.  Index types are the narrowest that hold each capacity.
template <int HS_, int CAV_, int BF_, int NBR_, int VH_, int G_, class SlotT, class CavT>
struct Workspace {
    static constexpr int HS = HS_;        // tested-tet hash slots (power of two)
    static constexpr int QCAP = HS_ * 3 / 4;
    static constexpr int CAV = CAV_;      // cavity tets
    static constexpr int STACK = 4 * CAV_ + 1;
    static constexpr int BF = BF_;        // boundary faces
    static constexpr int NBR = NBR_;      // natural neighbours
    static constexpr int VH = VH_;        // neighbour hash slots (power of two)
    static constexpr int G = G_;
    using slot_t = SlotT;                 // tested-tet hash slot index
    using cav_t = CavT;                   // signed cavity index
    union U {
        struct {
            int hkey[HS_];
            CavT hval[HS_];
            SlotT queue[HS_ * 3 / 4];
        } a;
        struct {
            CavT stack[4 * CAV_ + 1];
        } r;
    } u;
    double acc[NBR_];            // stolen volume per neighbour
    int cav_tet[CAV_];
    int nbr_vid[NBR_];
    int vh_key[VH_];
    int vh_first[VH_];
    alignas(4) CavT cav_nbr[4 * CAV_];  // cavity index of neighbour f of cavity tet c, -1 outside
    CavT order[CAV_];            // cavity tets in natinterp3d's visiting order
    CavT pos[CAV_];              // inverse of order
    uint16_t bface[BF_];         // (cavity index << 2) | face
    int16_t vh_slot[VH_];
    alignas(16) int4 wave[G_];   // neighbours of the flood wave's cavity tets
};

// Workspace of the split row's cavity phase (flood_pair): one a row, two rows a
// warp.
template <int HS_, int CAV_>
struct alignas(16) CavWorkspace {
    static constexpr int HS = HS_;             // tested-tet hash slots (power of two)
    static constexpr int QCAP = HS_ * 3 / 4;
    static constexpr int CAV = CAV_;
    static_assert(HS_ <= 256 && CAV_ <= 127, "slots and cavity indices are bytes");
    int hkey[HS_];
    int8_t hval[HS_];       // cavity index of a tested tet, -1 outside
    int4 wave[16];          // neighbours of the wave's cavity tets
    int cav_tet[CAV_];
    uint8_t queue[HS_ * 3 / 4];
    union {
        uint8_t nsl[4 * CAV_];                // hash slot of neighbour f of cavity tet c
        alignas(4) int8_t cav_nbr[4 * CAV_];  // then its cavity index, -1 outside
    };
};

// Workspace of the split row's volume phase (split_row): room for BF boundary
// faces.  The phases reuse one arena.  A vertex's id is its number in the row,
// in no particular order: the natural neighbours, then the super-simplex's
// four vertices.
constexpr int VOL_VERTS = 56;      // ids of a row (columns are below 63)
constexpr int VOL_NO_ID = 255;     // a cavity vertex that is on no boundary face
template <int CAV_, int BF_, int VH_, int G_>
struct alignas(16) VolWorkspace {
    static constexpr int CAV = CAV_;
    static constexpr int BF = BF_;
    static constexpr int FW = (BF_ + 63) / 64;  // 64-bit words of a face set
    using edge_t = typename std::conditional<(BF_ <= 85), uint8_t, uint16_t>::type;
    static constexpr unsigned NO_EDGE = (1u << 8 * sizeof(edge_t)) - 1u;
    static constexpr int PAIR_IDS = FW == 1 ? 36 : VOL_VERTS;  // ids of a row that this size takes
    static constexpr int NBR = VOL_VERTS - 4;
    static constexpr int VH = VH_;
    static constexpr int G = G_;
    union U {
        struct {
            int tet[CAV_];       // cavity tets in visiting order
            unsigned lid[CAV_];  // their vertices' ids, one byte each (first: hash slots)
            uint8_t mask[CAV_];  // boundary faces, and << 4 the faces that take a neighbour's copy
            unsigned long long tm[VOL_VERTS];       // per neighbour, the set of its cavity tets
            unsigned firsts[(3 * BF_ + 31) / 32];   // the set of corners that are a vertex's first
            union {
                struct {
                    alignas(16) int vh_key[VH_];
                    int vh_first[VH_];
                } h;
                double term[4 * CAV_];              // cavity terms, by neighbour
            };
        } c;
        // directed boundary edge (u, w) -> 3 * face + corner of u, all ones: none
        edge_t pair[PAIR_IDS * PAIR_IDS + 16 / sizeof(edge_t)];
        struct {
            // circumcentre of (u, q, w) relative to u, per directed boundary edge
            double ec[3 * BF_][3];
            double ct[BF_][3];     // circumcentre of (q, face)
        } v;
    } u;
    union {
        double pos[VOL_VERTS][3];  // vertex positions by id
        struct {
            double acc[64];        // weights by neighbour, once the terms are added
            int vh_first[64];      // scratch of the sinks
        };
    };
    union {
        unsigned long long fm[FW * VOL_VERTS];  // per id, the set of its boundary faces
        double fterm[3 * BF_];   // face terms, by neighbour
    };
    // per face corner: ids of its vertex u, of the next w and the one after x (6
    // bits each), another face's edge u -> x (EB bits, all ones: none), and the
    // place of its term
    using corner_t = typename std::conditional<(BF_ < 43), unsigned, unsigned long long>::type;
    static constexpr int EB = BF_ < 43 ? 7 : 10;
    corner_t corner[3 * BF_];
    int start[VOL_VERTS];        // first term of a neighbour: cavity, face << 16 (first: its first corner)
    int nbr_vid[VOL_VERTS];
    unsigned fid[BF_];           // ids of the face's three vertices, one byte each
    int bff[BF_];                // fcc[] index of the face (first: visiting position << 2 | face); the
                                 // sign bit: its corners' orientation is negative
};

// One row between k_rows_cavity, k_rows_order and k_rows_volume: a header
// and, per cavity tet in the flood's order, the tet, which of its faces bound
// the cavity (bits 0-3) and the cavity indices of its four neighbours (four
// signed bytes, -1 outside the cavity); k_rows_order adds the tet's position in
// natinterp3d's visiting order and which of its faces take a neighbour's copy.
constexpr int REC_CAV = 48;  // cavity tets a record holds (larger cavities take the large kernel)
constexpr int RS_OK = 0, RS_OUTSIDE = 1, RS_WALK = 2, RS_QUEUED = 3;
constexpr int RS_GENERAL = 4;  // a record for k_rows_general (k_rows_order)
constexpr int RS_FLAT = 5;     // the same by its tets' size (k_rows_cavity, for k_rows_order)
struct __align__(16) RowHead {
    int ncav;   // cavity tets (0: the coincident-vertex row)
    int start;  // located tet
    int state;  // RS_*
    int pad;
};
struct __align__(16) RowEntry {
    int tet;
    unsigned bmask;  // boundary faces
    int nbr;         // cavity indices of neighbours 0..3, one signed byte each
    int pos;         // position in natinterp3d's visiting order (bits 0-7); bit 8 + i: face
                     // 3 - i takes the copy of the neighbour visited earlier
};
static_assert(sizeof(RowEntry) == 16, "RowEntry is one 16-byte load");

__device__ __forceinline__ unsigned mix_hash(int key) {
    return (unsigned)key * 2654435761u;
}

// Inserts key; returns its slot, whether newly inserted (fresh = true) or
// already present.  Returns -1 and sets full when every slot was probed.
__device__ __forceinline__ int hash_insert(int *keys, int hs, int key, bool &fresh, bool &full) {
    unsigned h = mix_hash(key) & (unsigned)(hs - 1);
#pragma unroll 1
    for (int probe = 0; probe < hs; ++probe) {
        const int old = atomicCAS(&keys[h], -1, key);
        if (old == -1) {
            fresh = true;
            return (int)h;
        }
        if (old == key) return (int)h;
        h = (h + 1) & (unsigned)(hs - 1);
    }
    full = true;
    return -1;
}

// Slot of key (inserted if absent); -1 and full=true when the table is full.
__device__ __forceinline__ int hash_upsert(int *keys, int hs, int key, bool &full) {
    unsigned h = mix_hash(key) & (unsigned)(hs - 1);
#pragma unroll 1
    for (int probe = 0; probe < hs; ++probe) {
        int old = *(volatile int *)&keys[h];  // most keys are there already
        if (old == -1) old = atomicCAS(&keys[h], -1, key);
        if (old == -1 || old == key) return (int)h;
        h = (h + 1) & (unsigned)(hs - 1);
    }
    full = true;
    return -1;
}

__device__ __forceinline__ int hash_find(const int *keys, int hs, int key) {
    unsigned h = mix_hash(key) & (unsigned)(hs - 1);
#pragma unroll 1
    for (int probe = 0; probe < hs; ++probe) {
        const int k = keys[h];
        if (k == key) return (int)h;
        if (k == -1) return -1;
        h = (h + 1) & (unsigned)(hs - 1);
    }
    return -1;
}

struct RowInfo {
    int status;
    int nnb;
    int steps;
    bool outside;
    bool coincident;  // row from the coincident-vertex path
    double total;     // sum of the stolen volumes (the normaliser), 0 if none
    int nbf;          // boundary faces (ws.bface[0..nbf))
    // PM_RESOLVE only: predicate evaluations natinterp3d performs for this row
    // that the filter could not certify, and those whose decision the exact
    // sign changes (walk orientation tests / cavity in-sphere tests)
    int o_unc, o_flip, i_unc, i_flip;
};

// ---- predicate filters and exact resolution ---------------------------------
__device__ __forceinline__ void to3(const dv3 &v, double *o) {
    o[0] = v.x;
    o[1] = v.y;
    o[2] = v.z;
}

__device__ __forceinline__ int sgn(double x) { return (x > 0.0) - (x < 0.0); }

__device__ __forceinline__ bool orient_uncertain(const dv3 &a, const dv3 &b, const dv3 &c,
                                                 const dv3 &d, double fast) {
    double pa[3], pb[3], pc[3], pd[3];
    to3(a, pa), to3(b, pb), to3(c, pc), to3(d, pd);
    return nif_orient_uncertain(fast, nif_orient_permanent(pa, pb, pc, pd));
}

__device__ __forceinline__ bool insphere_uncertain(const dv3 &a, const dv3 &b, const dv3 &c,
                                                   const dv3 &d, const dv3 &e, double fast) {
    double pa[3], pb[3], pc[3], pd[3], pe[3];
    to3(a, pa), to3(b, pb), to3(c, pc), to3(d, pd), to3(e, pe);
    return nif_insphere_uncertain(fast, nif_insphere_permanent(pa, pb, pc, pd, pe));
}

// Exact orient3d signs for the lanes with unc set, one lane at a time in the
// shared scratch xs (NIF_EXACT_SCRATCH doubles); other lanes keep s.
template <int G>
__device__ __forceinline__ int resolve_orient(const Grp<G> &g, double *xs, bool unc, const dv3 &a,
                                              const dv3 &b, const dv3 &c, const dv3 &d, int s) {
    unsigned um = g.ballot(unc);
    while (um) {
        const int l = __ffs(um) - 1;
        um &= um - 1u;
        if (g.lane == l) {
            double pa[3], pb[3], pc[3], pd[3];
            to3(a, pa), to3(b, pb), to3(c, pc), to3(d, pd);
            s = nif_orient_exact_sign(pa, pb, pc, pd, xs);
        }
        g.sync();
    }
    return s;
}

template <int G>
__device__ __forceinline__ int resolve_insphere(const Grp<G> &g, double *xs, bool unc, const dv3 &a,
                                                const dv3 &b, const dv3 &c, const dv3 &d,
                                                const dv3 &e, int s) {
    unsigned um = g.ballot(unc);
    while (um) {
        const int l = __ffs(um) - 1;
        um &= um - 1u;
        if (g.lane == l) {
            double pa[3], pb[3], pc[3], pd[3], pe[3];
            to3(a, pa), to3(b, pb), to3(c, pc), to3(d, pd), to3(e, pe);
            s = nif_insphere_exact_sign(pa, pb, pc, pd, pe, xs);
        }
        g.sync();
    }
    return s;
}

// PRED_EXACT, query exactly on a face or edge of its located tet: the cavity
// index of the lowest-id cavity tet whose closure contains q (exact signs),
// from which the visiting order is replayed -- the order then no longer
// depends on which of the containing tets the walk reached.
template <int G, class W>
__device__ int canonical_start(const MeshView &M, const W &ws, const Grp<G> &g, double *xs,
                               const dv3 q, int ncav) {
    int best_t = INT_MAX, best_c = 0;
    for (int c0 = 0; c0 < ncav; c0 += G) {
        const int c = c0 + g.lane;
        bool alive = c < ncav;
        const int tt = alive ? ws.cav_tet[c] : 0;
        const int4 p = M.tv[tt];
        for (int f = 0; f < 4; f++) {
            dv3 v1{0.0, 0.0, 0.0}, v2 = v1, v3 = v1;
            int s = 1;
            bool unc = false;
            if (alive) {
                v1 = vload(M, comp(p, face_vslot(f, 0)));
                v2 = vload(M, comp(p, face_vslot(f, 1)));
                v3 = vload(M, comp(p, face_vslot(f, 2)));
                const double o = orient_fast(v1, v2, v3, q);
                s = sgn(o);
                unc = orient_uncertain(v1, v2, v3, q, o);
            }
            s = resolve_orient(g, xs, unc, v1, v2, v3, q, s);
            if (s < 0) alive = false;
        }
        if (alive && tt < best_t) {
            best_t = tt;
            best_c = c;
        }
    }
    for (int off = G / 2; off > 0; off >>= 1) {
        const int ot = g.shfl_xor(best_t, off), oc = g.shfl_xor(best_c, off);
        if (ot < best_t) {
            best_t = ot;
            best_c = oc;
        }
    }
    return best_c;
}

// slot of a data vertex among the natural neighbours, -1 if it is not one
template <class W>
__device__ __forceinline__ int neighbour_slot(const W &ws, int v) {
    const int s = hash_find(ws.vh_key, W::VH, v);
    return s >= 0 ? ws.vh_slot[s] : -1;
}

// Point location (natinterp3d's findContainingSimplex, delaunay.c:383-407):
// the seed is the nearest tet centroid, then natinterp3d's visibility walk.
// Returns the located tet; r.status / r.outside report a walk that hit its
// step limit or left the super-simplex, r.steps counts the steps.  scratch:
// 64 ints of group scratch (the octree search's).  PM selects the predicate
// variant as in sibson_row; *on_face is set in PM_RESOLVE / PRED_EXACT when a
// face test of the located tet is exactly zero.
template <int G, int PM>
__device__ int locate(const MeshView &M, const dv3 q, const Grp<G> &g, int *scratch, RowInfo &r,
                      bool &on_face, double *xs = nullptr) {
    const bool filt = PM != PM_PLAIN && M.pmode != PRED_FAST;
    int t = grid_nearest<G>(M, q);
    if (t < 0) t = nearest_centroid<G>(M, q, g, scratch);
    for (;;) {
        if (r.steps >= WALK_LIMIT) {
            r.status = ST_WALK;
            return t;
        }
        ++r.steps;
        const int4 p = M.tv[t];
        const int4 nbs = M.tn[t];  // loaded with p: no second dependent trip per step
        int sg = 1;
        bool unc = false;
        dv3 v1{0.0, 0.0, 0.0}, v2 = v1, v3 = v1;
        if (g.lane < 4) {
            const int f = g.lane;
            v1 = vload(M, comp(p, face_vslot(f, 0)));
            v2 = vload(M, comp(p, face_vslot(f, 1)));
            v3 = vload(M, comp(p, face_vslot(f, 2)));
            const double o = orient_fast(v1, v2, v3, q);
            sg = sgn(o);
            if (filt) unc = orient_uncertain(v1, v2, v3, q, o);
        }
        unsigned m;
        if constexpr (PM == PM_PLAIN) {
            m = g.ballot(sg < 0);
        } else if constexpr (PM == PM_FILTER) {
            // natinterp3d tests faces 0..3 and moves through the first negative
            // one: only uncertain tests up to that face can change the step
            m = g.ballot(!unc && sg < 0);
            const int fn = m ? __ffs(m) - 1 : 4;
            if (g.ballot(unc) & ((2u << fn) - 1u)) {
                r.status = ST_UNCERTAIN;
                return t;
            }
        } else {
            if (filt) {
                const int xsg = resolve_orient(g, xs, unc, v1, v2, v3, q, sg);
                const int use = M.pmode == PRED_EXACT ? xsg : sg;
                m = g.ballot(use < 0);
                const unsigned seen = (2u << (m ? __ffs(m) - 1 : 3)) - 1u;  // tests natinterp3d makes
                r.o_unc += __popc(g.ballot(unc) & seen);
                r.o_flip += __popc(g.ballot(unc && ((xsg < 0) != (sg < 0))) & seen);
                if (!m) on_face = g.ballot(use == 0) != 0u;
            } else {
                m = g.ballot(sg < 0);
            }
        }
        if (!m) return t;
        const int nb = comp(nbs, __ffs(m) - 1);
        if (nb < 0) {
            r.outside = true;
            return t;
        }
        t = nb;
    }
}

// natinterp3d's walk of up to eight rows at once, four lanes a row (one face
// test each), from the rows' seed tets t: the located tet, or -1 outside the
// super-simplex, -2 at the step limit, -3 (PM_FILTER) at a test that the error
// bound cannot certify and that can change the step.  `act`: the lane's row is
// there; steps counts its steps.  Called by the whole warp, with the rows of one
// mesh.
template <int PM>
__device__ __forceinline__ int walk_rows(const MeshView &M, const dv3 q, int t, bool act, int &steps) {
    const bool filt = PM != PM_PLAIN && M.pmode != PRED_FAST;
    const int f = threadIdx.x & 3, sh = threadIdx.x & 28;
    steps = 0;
    while (__any_sync(0xffffffffu, act)) {
        int4 nbs = make_int4(-1, -1, -1, -1);
        bool neg = false, unc = false;
        if (act) {
            const int4 p = M.tv[t];
            nbs = M.tn[t];  // loaded with p: no second dependent trip per step
            const dv3 v1 = vload(M, comp(p, face_vslot(f, 0)));
            const dv3 v2 = vload(M, comp(p, face_vslot(f, 1)));
            const dv3 v3 = vload(M, comp(p, face_vslot(f, 2)));
            const double o = orient_fast(v1, v2, v3, q);
            if (filt) unc = orient_uncertain(v1, v2, v3, q, o);
            neg = o < 0.0 && !unc;
        }
        // natinterp3d tests faces 0..3 and moves through the first negative one:
        // only uncertain tests up to that face can change the step
        const unsigned m = (__ballot_sync(0xffffffffu, neg) >> sh) & 15u;
        const int first = m ? __ffs(m) - 1 : 4;
        bool open = false;
        if constexpr (PM == PM_FILTER)
            open = (((__ballot_sync(0xffffffffu, unc) >> sh) & 15u) & ((2u << first) - 1u)) != 0u;
        if (act) {
            ++steps;
            if (open) {
                t = -3;
                act = false;
            } else if (!m) {
                act = false;
            } else {
                t = comp(nbs, first);
                act = t >= 0;  // -1: outside
                if (act && steps >= WALK_LIMIT) {
                    t = -2;
                    act = false;
                }
            }
        }
    }
    return t;
}

// Steps 2 of the row: the cavity of q around tet `start` (natinterp3d's
// findCavity, natural_insertionfree.c:486-551) by a parallel flood over the
// tested-tet hash, then natinterp3d's LIFO visiting order replayed on it.
// Returns the number of cavity tets, ws.cav_tet[c] their tets, ws.order[o]
// the cavity index of the o-th visited, ws.pos its inverse and ws.cav_nbr
// [4c + f] the cavity index of neighbour f of cavity tet c (-1 outside).  On
// overflow / an uncertain test (PM_FILTER) r.status is set; an empty cavity
// (0) leaves the order unset.
template <int G, class W, int PM>
__device__ int flood_replay(const MeshView &M, const dv3 q, W &ws, const Grp<G> &g, const int start,
                            RowInfo &r, const bool on_face, double *xs) {
    using cav_t = typename W::cav_t;
    using slot_t = typename W::slot_t;
    const bool filt = PM != PM_PLAIN && M.pmode != PRED_FAST;
    // ---- 2. cavity: parallel flood over the tested-tet hash ----------------
    // While a cavity tet's four neighbours are inserted into the hash, the
    // slot of each is kept in nsl[4c+f] (aliasing cav_nbr, which is filled
    // from it after the flood).  A missing neighbour (hull face of the
    // super-simplex) gets the slot of the key NO_TET, inserted up front with
    // hval = -1 and never queued, so every face has a slot.
    static_assert(sizeof(slot_t) == sizeof(cav_t), "nsl aliases cav_nbr");
    constexpr int NO_TET = -2;
    slot_t *nsl = reinterpret_cast<slot_t *>(ws.cav_nbr);
    static_assert(offsetof(decltype(ws.u.a), hval) == sizeof(ws.u.a.hkey) &&
                      (sizeof(ws.u.a.hkey) + sizeof(ws.u.a.hval)) % 16 == 0,
                  "one run of -1s");
    for (int i = g.lane; i < (int)((sizeof(ws.u.a.hkey) + sizeof(ws.u.a.hval)) / 16); i += G)
        reinterpret_cast<int4 *>(ws.u.a.hkey)[i] = make_int4(-1, -1, -1, -1);
    g.sync();
    int none_slot = 0;
    if (g.lane == 0) {
        const int h = (int)(mix_hash(start) & (unsigned)(W::HS - 1));
        ws.u.a.hkey[h] = start;
        ws.u.a.queue[0] = (slot_t)h;
        bool fresh = false, full = false;
        none_slot = hash_insert(ws.u.a.hkey, W::HS, NO_TET, fresh, full);
    }
    none_slot = g.shfl(none_slot, 0);
    g.sync();
    int qhead = 0, qtail = 1, ncav = 0;
    bool overflow = false;
    // With natinterp3d's signs the located tet's neighbours join its wave:
    // the flood tests them next whenever the located tet is in the cavity, in
    // this same queue order, so the cavity indices are those of a flood that
    // starts with the located tet alone, and one wave of a single lane is
    // saved.  (If the located tet is not in the cavity, their tests are
    // dropped below.)  Filtered modes keep the plain start, so that their
    // predicate counters count the same tests.
    const bool ring = !filt;
    if (ring) {
        int ns = -1;
        bool full = false;
        if (g.lane < 4) {
            const int nb = comp(M.tn[start], g.lane);
            bool fresh = false;
            if (nb >= 0) {
                const int sl = hash_insert(ws.u.a.hkey, W::HS, nb, fresh, full);
                if (fresh) ns = sl;
            }
        }
        const unsigned pm = g.ballot(ns >= 0);
        if (ns >= 0) ws.u.a.queue[qtail + __popc(pm & g.lt())] = (slot_t)ns;
        qtail += __popc(pm);
        if (g.any(full)) overflow = true;
        g.sync();
    }
    while (!overflow && qhead < qtail) {
        const int n = min(G, qtail - qhead);
        int slot = -1, tt = -1;
        bool inc = false, unc = false, open = false;
        int4 nb4 = make_int4(-1, -1, -1, -1);
        dv3 ia{0.0, 0.0, 0.0}, ib = ia, ic = ia, id = ia;
        if (g.lane < n) {
            slot = ws.u.a.queue[qhead + g.lane];
            tt = ws.u.a.hkey[slot];
            nb4 = M.tn[tt];  // with the sphere: no second trip for the tets inside
            const int side = sphere_side(M.tcc[tt], q);
            inc = side > 0;
            open = side == 0;
        }
        // tests that the cached sphere does not decide: the determinant itself
        if (g.any(open)) {
            if (open) {
                const int4 p = M.tv[tt];
                const dv3 a = vload(M, p.x), b = vload(M, p.y);
                ic = vload(M, p.z);
                id = vload(M, p.w);
                // insphere argument order fixed by the tet's orientation
                // (natural_insertionfree.c:511-515); PRED_EXACT uses the exact one
                const uint32_t info = M.tinfo[tt];
                const bool pos = (info & ((PM != PM_PLAIN && M.pmode == PRED_EXACT) ? 4u : 1u)) != 0;
                ia = pos ? a : b;
                ib = pos ? b : a;
                const double sv = insphere_fast(ia, ib, ic, id, q);
                inc = sv > 0;
                if (filt) unc = insphere_uncertain(ia, ib, ic, id, q, sv);
            }
        }
        if constexpr (PM == PM_FILTER) {
            if (g.any(unc)) {
                r.status = ST_UNCERTAIN;
                return 0;
            }
        } else if constexpr (PM == PM_RESOLVE) {
            if (filt && g.any(unc)) {
                const bool xin = resolve_insphere(g, xs, unc, ia, ib, ic, id, q, inc ? 1 : -1) > 0;
                r.i_unc += __popc(g.ballot(unc));
                r.i_flip += __popc(g.ballot(unc && xin != inc));
                if (M.pmode == PRED_EXACT) inc = xin;
            }
        }
        const unsigned cm = g.ballot(inc);
        if (ring && qhead == 0 && !(cm & 1u)) break;  // the located tet is outside: empty cavity
        const int ci = ncav + __popc(cm & g.lt());
        if (g.lane < n) ws.u.a.hval[slot] = (cav_t)(inc ? ci : -1);
        if (inc && ci < W::CAV) {
            ws.cav_tet[ci] = tt;
            ws.wave[ci - ncav] = nb4;
            // the volume phase reads this tet's face circumcentres
            prefetch_l2(&M.fcc[4 * (size_t)tt]);
        }
        const int nnew = __popc(cm);
        const int base = ncav;
        ncav += nnew;
        qhead += n;
        if (ncav > W::CAV) {
            overflow = true;
            break;
        }
        g.sync();
        for (int k0 = 0; k0 < 4 * nnew; k0 += G) {
            const int k = k0 + g.lane;
            int ns = -1;
            bool full = false, fresh = false;
            if (k < 4 * nnew) {
                const int nb = reinterpret_cast<const int *>(ws.wave)[k];
                int sl = none_slot;
                if (nb >= 0) sl = hash_insert(ws.u.a.hkey, W::HS, nb, fresh, full);
                if (fresh) ns = sl;
                nsl[4 * base + k] = (slot_t)(full ? none_slot : sl);
            }
            const unsigned pm = g.ballot(ns >= 0);
            const int qi = qtail + __popc(pm & g.lt());
            if (ns >= 0 && qi < W::QCAP) ws.u.a.queue[qi] = (slot_t)ns;
            qtail += __popc(pm);
            if (g.any(full) || qtail > W::QCAP) overflow = true;
        }
        if (overflow) break;
        g.sync();
    }
    g.sync();
    if (overflow) {
        r.status = ST_CAPACITY;
        return 0;
    }
    if (ncav == 0) return 0;

    // cavity-local neighbour table: cav_nbr[4c+f] = cavity index of s[f] or -1
    // (every neighbour slot recorded by the flood has been tested by now)
    for (int k = g.lane; k < 4 * ncav; k += G) ws.cav_nbr[k] = ws.u.a.hval[nsl[k]];
    for (int c = g.lane; c < ncav; c += G) ws.pos[c] = (cav_t)-1;
    g.sync();

    // cavity index 0 is the located tet, the flood's start
    int start_c = 0;
    if constexpr (PM == PM_RESOLVE) {
        if (on_face && M.pmode == PRED_EXACT) start_c = canonical_start(M, ws, g, xs, q, ncav);
    }

    // replay natinterp3d's LIFO flood on the cavity (its non-cavity tets are
    // leaves and do not change the order in which cavity tets are reached)
    if (g.lane == 0) {
        cav_t *stack = ws.u.r.stack;
        int sp = 0, nord = 0;
        stack[sp++] = (cav_t)start_c;
        if constexpr (W::CAV <= 128) {
            // visited set in two 64-bit registers
            uint64_t v0 = 0, v1 = 0;
            while (sp > 0) {
                const int c = stack[--sp];
                const uint64_t bit = 1ull << (c & 63);
                if ((c < 64 ? v0 : v1) & bit) continue;
                if (c < 64) v0 |= bit; else v1 |= bit;
                int n0, n1, n2, n3;
                if constexpr (sizeof(cav_t) == 1) {
                    // the four signed 8-bit entries of tet c in one 32-bit load
                    const int w = *reinterpret_cast<const int *>(&ws.cav_nbr[4 * c]);
                    n0 = (int8_t)(w & 0xff);
                    n1 = (int8_t)((w >> 8) & 0xff);
                    n2 = (int8_t)((w >> 16) & 0xff);
                    n3 = (int8_t)((unsigned)w >> 24);
                } else {
                    n0 = ws.cav_nbr[4 * c], n1 = ws.cav_nbr[4 * c + 1];
                    n2 = ws.cav_nbr[4 * c + 2], n3 = ws.cav_nbr[4 * c + 3];
                }
                ws.pos[c] = (cav_t)nord;
                ws.order[nord++] = (cav_t)c;
                const int nb[4] = {n0, n1, n2, n3};
    #pragma unroll
                for (int f = 0; f < 4; f++) {
                    const int nc = nb[f];
                    if (nc >= 0 && !(((nc < 64 ? v0 : v1) >> (nc & 63)) & 1ull)) stack[sp++] = (cav_t)nc;
                }
            }
        } else {
            while (sp > 0) {
                const int c = stack[--sp];
                if (ws.pos[c] >= 0) continue;
                ws.pos[c] = (cav_t)nord;
                ws.order[nord++] = (cav_t)c;
                for (int f = 0; f < 4; f++) {
                    const int nc = ws.cav_nbr[4 * c + f];
                    if (nc >= 0 && ws.pos[nc] < 0) stack[sp++] = (cav_t)nc;
                }
            }
        }
    }
    g.sync();

    return ncav;
}

// The coincident-vertex row (natural_insertionfree.c:596-622): an empty
// cavity means the query may sit exactly on a vertex of the start tet; the
// row is 1/n on each of the n data vertices of that tet equal to q.
template <int G, class W>
__device__ void coincident_row(const MeshView &M, const dv3 q, W &ws, const Grp<G> &g, int start,
                               RowInfo &r) {
    bool co = false;
    int v = -1;
    if (g.lane < 4) {
        v = comp(M.tv[start], g.lane);
        co = v < M.n && veq(vload(M, v), q);
    }
    const unsigned cm = g.ballot(co);
    const int nco = __popc(cm);
    if (co) {
        const int s = __popc(cm & g.lt());
        ws.nbr_vid[s] = v;
        ws.acc[s] = fdiv(1.0, (double)nco);
    }
    g.sync();
    r.nnb = nco;
    r.coincident = true;
}

// The circumcentres of the 4 faces of cavity tet c as natinterp3d's face
// cache returns them (natural_insertionfree.c:233-253), as fcc[] indices
// (4 T < 2^31: nif_dmesh_create limits T): for a face shared with another
// cavity tet, the copy cached by whichever of the two natinterp3d visits first
// (its mirror slot is in tinfo), else the tet's own.  Needs ws.pos.
template <class W>
__device__ __forceinline__ void face_cc_choice(const MeshView &M, const W &ws, int c, int (&fp)[4]) {
    const int tt = ws.cav_tet[c];
    const uint32_t info = M.tinfo[tt];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int j = 3 - i;
        const int nc = ws.cav_nbr[4 * c + j];
        if (nc >= 0 && ws.pos[nc] < ws.pos[c]) {
            const int jm = (info >> (8 + 2 * j)) & 3;
            fp[i] = 4 * ws.cav_tet[nc] + (3 - jm);
        } else {
            fp[i] = 4 * tt + i;
        }
    }
}

// Steps 3-5 of the row: boundary faces in visiting order, the natural
// neighbours in first-seen order, and (FULL) the stolen volumes folded in
// natinterp3d's order and normalised.  The caller describes the cavity:
//   face(k, c)       whether face k & 3 of the (k >> 2)-th tet in visiting
//                    order is a boundary face; c = that tet's index into
//                    ws.cav_tet
//   tet_fp(o, c, fp) the o-th tet in visiting order (index c into
//                    ws.cav_tet) and the fcc[] indices of its four faces as
//                    natinterp3d's face cache returns them
//   tet_tv(c)        the vertex record of cavity tet c (M.tv[ws.cav_tet[c]])
template <int G, class W, bool FULL, class FaceFn, class FpFn, class TvFn>
__device__ RowInfo row_volumes(const MeshView &M, const dv3 q, W &ws, const Grp<G> &g, const int ncav,
                               RowInfo r, FaceFn face, FpFn tet_fp, TvFn tet_tv) {
    // ---- 3. boundary faces (cavity order, then face order) ------------------
    int nbf = 0;
    for (int k0 = 0; k0 < 4 * ncav; k0 += G) {
        const int k = k0 + g.lane;
        bool isb = false;
        int c = 0;
        if (k < 4 * ncav) isb = face(k, c);
        const unsigned bm = g.ballot(isb);
        const int b = nbf + __popc(bm & g.lt());
        if (isb && b < W::BF) ws.bface[b] = (uint16_t)((c << 2) | (k & 3));
        nbf += __popc(bm);
    }
    if (nbf > W::BF) {
        r.status = ST_CAPACITY;
        return r;
    }
    r.nbf = nbf;

    // natural neighbours in first-seen order over the boundary-face vertices
    for (int i = g.lane; i < W::VH; i += G) {
        ws.vh_key[i] = -1;
        ws.vh_first[i] = 0x7fffffff;
    }
    g.sync();
    bool vfull = false;
    for (int k = g.lane; k < 3 * nbf; k += G) {
        const int b = k / 3, j = k - 3 * b;
        const int cf = ws.bface[b];
        const int v = comp(tet_tv(cf >> 2), face_vslot(cf & 3, j));
        if (v < M.n) {
            const int s = hash_upsert(ws.vh_key, W::VH, v, vfull);
            if (s >= 0) atomicMin(&ws.vh_first[s], k);
        }
    }
    g.sync();
    if (g.any(vfull)) {
        r.status = ST_CAPACITY;
        return r;
    }
    int nnb = 0;
    for (int k0 = 0; k0 < 3 * nbf; k0 += G) {
        const int k = k0 + g.lane;
        bool first = false;
        int v = -1, s = -1;
        if (k < 3 * nbf) {
            const int b = k / 3, j = k - 3 * b;
            const int cf = ws.bface[b];
            v = comp(tet_tv(cf >> 2), face_vslot(cf & 3, j));
            if (v < M.n) {
                s = hash_find(ws.vh_key, W::VH, v);
                first = (s >= 0) && ws.vh_first[s] == k;
            }
        }
        const unsigned fm = g.ballot(first);
        const int slot = nnb + __popc(fm & g.lt());
        if (first) {
            ws.vh_slot[s] = (int16_t)slot;
            if (slot < W::NBR) {
                ws.nbr_vid[slot] = v;
                ws.acc[slot] = 0.0;
            }
        }
        nnb += __popc(fm);
    }
    if (nnb > W::NBR) {
        r.status = ST_CAPACITY;
        return r;
    }
    g.sync();
    if (nnb == 0) return r;
    if constexpr (!FULL) {
        r.nnb = nnb;
        return r;
    }

    // ---- 4. stolen volumes ----------------------------------------------------
    // Items in natinterp3d's order: the 4 vertices of every cavity tet (cavity
    // order), then the 3 vertices of every boundary face (face order).  One
    // lane computes the items of one cavity tet (4) or one boundary face (3),
    // sharing that tet's loads and face-circumcentre choices, or the face's
    // virtual-tet circumcentre, among them; the terms go to a shared buffer
    // in item order.  Then lanes whose items belong to the same neighbour are
    // folded into acc[] by the lowest of them, in lane order, so every acc[]
    // is a left-to-right sum in item order.
    {
        // the cavity-search scratch is free now: item buffer of one round
        constexpr int PER = 4 * G;  // items of one round (old terms: 4 per lane)
        static_assert(PER * (sizeof(double) + sizeof(int16_t)) <= sizeof(ws.u), "item buffer");
        double *bterm = reinterpret_cast<double *>(&ws.u);
        int16_t *bslot = reinterpret_cast<int16_t *>(bterm + PER);
        // folds buffered items [0, n) into acc[]
        auto fold = [&](int n) {
            for (int k0 = 0; k0 < n; k0 += G) {
                const int k = k0 + g.lane;
                const int s = k < n ? bslot[k] : -1;
                const double term = k < n ? bterm[k] : 0.0;
                const unsigned peers = g.match(s);
                const bool lead = s >= 0 && (__ffs(peers) - 1) == g.lane;
                unsigned rem = lead ? peers : 0u;
                double a = lead ? ws.acc[s] : 0.0;
                while (g.any(rem != 0u)) {
                    const int src = rem ? __ffs(rem) - 1 : g.lane;
                    const double tv = g.shfl(term, src);
                    if (rem) {
                        a = fadd(a, tv);
                        rem &= rem - 1u;
                    }
                }
                if (lead) ws.acc[s] = a;
                g.sync();
            }
        };
        // cavity-tet terms (natural_insertionfree.c:642-676): one lane per
        // item (tet o = k / 4, vertex k % 4), so that a cavity of 18 tets
        // takes 3 lane-steps of 32 items rather than 4 steps of 18 lanes
        for (int k0 = 0; k0 < 4 * ncav; k0 += PER) {
            const int n_round = min(PER, 4 * ncav - k0);
#pragma unroll 1
            for (int k = k0 + g.lane; k < k0 + n_round; k += G) {
                const int o = k >> 2, vi = k & 3;
                int c, fp[4];
                tet_fp(o, c, fp);
                const int tt = ws.cav_tet[c];
                const int4 p = tet_tv(c);
                const int v = comp(p, vi);
                const int sl = v < M.n ? neighbour_slot(ws, v) : -1;
                double term = 0.0;
                if (sl >= 0) {
                    // the other three vertices in ascending slot order
                    const int o0v = (vi == 0) ? 1 : 0;
                    const int o1v = (vi <= 1) ? 2 : 1;
                    const int o2v = (vi <= 2) ? 3 : 2;
                    const dv3 pk = vload(M, v);
                    const dv3 pa = vload(M, comp(p, o0v));
                    const dv3 pb = vload(M, comp(p, o1v));
                    const dv3 pc = vload(M, comp(p, o2v));
                    const dv3 ct = cload(&M.tcc[tt]);
                    // fp[] indexed through selects, so that it stays in registers
                    auto pick = [&](int i) {
                        return i == 0 ? fp[0] : (i == 1 ? fp[1] : (i == 2 ? fp[2] : fp[3]));
                    };
                    const dv3 f1 = cload(&M.fcc[pick(o2v)]);
                    const dv3 f2 = cload(&M.fcc[pick(o1v)]);
                    const dv3 f3 = cload(&M.fcc[pick(o0v)]);
                    term = subcell_volume(pk, pa, pb, pc, ct, f1, f2, f3);
                }
                bterm[k - k0] = term;
                bslot[k - k0] = (int16_t)sl;
            }
            g.sync();
            fold(n_round);
        }
        // virtual-tet terms, query + boundary face (:681-719)
        for (int b0 = 0; b0 < nbf; b0 += G) {
            const int b = b0 + g.lane;
            const int nb_round = min(G, nbf - b0);
            if (b < nbf) {
                const int cf = ws.bface[b];
                const int f = cf & 3;
                const int tt = ws.cav_tet[cf >> 2];
                const int4 p = tet_tv(cf >> 2);
                const int va = comp(p, face_vslot(f, 0));
                const int vb = comp(p, face_vslot(f, 1));
                const int vc = comp(p, face_vslot(f, 2));
                const dv3 ct = tet_cc(q, vload(M, va), vload(M, vb), vload(M, vc));
                const int ffi = 4 * tt + (3 - f);
#pragma unroll 1
                for (int j = 0; j < 3; j++) {
                    const int v = (j == 0) ? va : (j == 1 ? vb : vc);
                    const int sl = v < M.n ? neighbour_slot(ws, v) : -1;
                    double term = 0.0;
                    if (sl >= 0) {
                        // the face's vertices are re-read (L1) rather than held
                        // across the loop, which would spill them
                        const int vn = (j == 0) ? vb : (j == 1 ? vc : va);  // face_verts[(j+1)%3]
                        const int vp = (j == 0) ? vc : (j == 1 ? va : vb);  // face_verts[(j+2)%3]
                        const dv3 pk = vload(M, v), pb = vload(M, vn), pc = vload(M, vp);
                        const dv3 f1 = tri_cc(pk, q, pb);
                        const dv3 f2 = tri_cc(pk, q, pc);
                        term = -subcell_volume(pk, q, pb, pc, ct, f1, f2, cload(&M.fcc[ffi]));
                    }
                    bterm[3 * g.lane + j] = term;
                    bslot[3 * g.lane + j] = (int16_t)sl;
                }
            }
            g.sync();
            fold(3 * nb_round);
        }
    }

    // ---- 5. normalisation -----------------------------------------------------
    double total = 0.0;
    if (g.lane == 0)
        for (int s = 0; s < nnb; s++) total = fadd(total, ws.acc[s]);
    total = g.shfl(total, 0);
    if (!(total > 1e-30)) return r;  // empty row
    const double inv = fdiv(1.0, total);
    for (int s = g.lane; s < nnb; s += G) ws.acc[s] = fmul(ws.acc[s], inv);
    g.sync();
    r.nnb = nnb;
    r.total = total;
    return r;
}

// The Sibson row of centred query q.  On ST_OK the row is ws.nbr_vid[0..nnb)
// with normalised weights ws.acc[0..nnb), in natinterp3d's column order.
// With FULL = false only the combinatorial part is built (cavity, visiting
// order, boundary faces, neighbours in column order) and no volume is
// computed; the query-gradient kernel needs nothing more.  PM selects the
// predicate variant (PM_*); PM_RESOLVE needs xs, NIF_EXACT_SCRATCH doubles of
// global scratch owned by this group.  (The split kernels, k_rows_cavity and
// k_rows_volume, run the same steps on located rows.)
// `located`: the row's located tet, or -1 to find it here.
template <int G, class W, bool FULL = true, int PM = PM_PLAIN>
__device__ RowInfo sibson_row(const MeshView &M, const dv3 q, W &ws, const Grp<G> &g,
                              double *xs = nullptr, int located = -1) {
    RowInfo r{ST_OK, 0, 0, false, false, 0.0, 0, 0, 0, 0, 0};
    bool on_face = false;  // PRED_EXACT: a face test of the located tet is exactly zero

    // ---- 1. point location -------------------------------------------------
    const int start = located >= 0 ? located
                                   : locate<G, PM>(M, q, g, reinterpret_cast<int *>(ws.acc), r, on_face, xs);
    if (r.status != ST_OK || r.outside) return r;

    // ---- 2. cavity and natinterp3d's visiting order ---------------------------
    const int ncav = flood_replay<G, W, PM>(M, q, ws, g, start, r, on_face, xs);
    if (r.status != ST_OK) return r;
    if (ncav == 0) {
        coincident_row<G>(M, q, ws, g, start, r);
        return r;
    }
    auto face = [&](int k, int &c) {
        c = ws.order[k >> 2];
        return ws.cav_nbr[4 * c + (k & 3)] < 0;
    };
    auto tet_fp = [&](int o, int &c, int (&fp)[4]) {
        c = ws.order[o];
        face_cc_choice(M, ws, c, fp);
    };
    auto tet_tv = [&](int c) { return M.tv[ws.cav_tet[c]]; };
    return row_volumes<G, W, FULL>(M, q, ws, g, ncav, r, face, tet_fp, tet_tv);
}

// The split row, part 1: the cavity of q around its located tet (flood_replay's
// flood), written as a record (head, entries[REC_CAV]): REC_DONE, or REC_WIDE where
// the cavity fits the shared-memory capacities but not the record (the caller
// queues the row for the fused row kernel), or REC_LARGE where it exceeds those
// capacities or, with PM_FILTER, where a test the error bound cannot certify
// comes up (the large kernel's).
//
// A flood's waves hold some 8 tets of 32 lanes' room, so that a warp floods two
// rows at once, one a half; both halves go through the same instructions until
// neither has a wave left (rows that diverge by themselves, as with 16-lane
// groups, run one after the other).  Bound by instruction issue (2.8 of 4 a
// cycle): 2M rows, 200k keys take 2.25 ms, 3.03 ms with a warp a row.
// `go`: this half has a row.  Called by the whole warp.
constexpr int REC_DONE = 0, REC_WIDE = 1, REC_LARGE = 2;
template <class W, int PM>
__device__ __forceinline__ int flood_pair(const MeshView &M, const dv3 q, W &ws, const int start, bool go,
                                          RowHead &head, RowEntry *__restrict__ ent) {
    static_assert(REC_CAV <= 127, "neighbour indices are signed bytes");
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int NO_TET = -2;
    const int lane = threadIdx.x & 31, hl = lane & 15, h0 = lane & 16;  // h0: the half's first lane
    const unsigned lt = (1u << hl) - 1u;
    auto ballot = [&](bool p) { return (__ballot_sync(FULL, p) >> h0) & 0xffffu; };
    const bool filt = PM != PM_PLAIN && go && M.pmode != PRED_FAST;

    static_assert(offsetof(W, hval) == sizeof(ws.hkey) && (sizeof(ws.hkey) + sizeof(ws.hval)) % 256 == 0,
                  "one run of -1s");
#pragma unroll
    for (int i = 0; i < (int)((sizeof(ws.hkey) + sizeof(ws.hval)) / 16); i += 16)
        reinterpret_cast<int4 *>(ws.hkey)[i + hl] = make_int4(-1, -1, -1, -1);
    __syncwarp();
    // a missing neighbour (hull face of the super-simplex) has the slot of NO_TET
    int none_slot = 0;
    bool full = false;  // never: the queue's limit is below the table's
    if (hl == 0) {
        const int h = (int)(mix_hash(start) & (unsigned)(W::HS - 1));
        ws.hkey[h] = start;
        ws.queue[0] = (uint8_t)h;
        bool fresh = false;
        none_slot = hash_insert(ws.hkey, W::HS, NO_TET, fresh, full);
    }
    none_slot = __shfl_sync(FULL, none_slot, h0);
    __syncwarp();
    int qhead = 0, qtail = 1, ncav = 0, rc = REC_DONE;
    // With natinterp3d's signs the located tet's neighbours join its wave (see
    // flood_replay)
    const bool ring = !filt;
    {
        bool fresh = false;
        int sl = 0;
        if (go && ring && hl < 4) {
            const int nb = comp(M.tn[start], hl);
            if (nb >= 0) sl = hash_insert(ws.hkey, W::HS, nb, fresh, full);
        }
        const unsigned pm = ballot(fresh);
        if (fresh) ws.queue[qtail + __popc(pm & lt)] = (uint8_t)sl;
        qtail += __popc(pm);
        __syncwarp();
    }
    for (;;) {
        const int n = go ? min(16, qtail - qhead) : 0;
        if (!__any_sync(FULL, n > 0)) break;
        int slot = 0, tt = 0;
        bool inc = false, unc = false, open = false;
        int4 nb4 = make_int4(-1, -1, -1, -1);
        if (hl < n) {
            slot = ws.queue[qhead + hl];
            tt = ws.hkey[slot];
            nb4 = M.tn[tt];  // with the sphere: no second trip for the tets inside
            const int side = sphere_side(M.tcc[tt], q);
            inc = side > 0;
            open = side == 0;
        }
        // tests that the cached sphere does not decide: the determinant itself
        if (__any_sync(FULL, open)) {
            if (open) {
                const int4 p = M.tv[tt];
                const dv3 a = vload(M, p.x), b = vload(M, p.y), c = vload(M, p.z), d = vload(M, p.w);
                // insphere argument order fixed by the tet's orientation
                // (natural_insertionfree.c:511-515); PRED_EXACT uses the exact one
                const bool pos = (M.tinfo[tt] & ((PM != PM_PLAIN && M.pmode == PRED_EXACT) ? 4u : 1u)) != 0;
                const dv3 ia = pos ? a : b, ib = pos ? b : a;
                const double sv = insphere_fast(ia, ib, c, d, q);
                inc = sv > 0;
                if (filt) unc = insphere_uncertain(ia, ib, c, d, q, sv);
            }
            if (PM != PM_PLAIN && ballot(unc)) {
                rc = REC_LARGE;
                go = false;
                inc = false;
            }
        }
        unsigned cm = ballot(inc);
        if (ring && qhead == 0 && !(cm & 1u)) {  // the located tet is outside: empty cavity
            go = false;
            cm = 0;
            inc = false;
        }
        const int i = __popc(cm & lt), ci = ncav + i;
        if (hl < n) ws.hval[slot] = (int8_t)(inc ? ci : -1);
        if (inc && ci < W::CAV) {
            ws.cav_tet[ci] = tt;
            ws.wave[i] = nb4;
            // the volume phase reads this tet's face circumcentres
            prefetch_l2(&M.fcc[4 * (size_t)tt]);
        }
        const int base = ncav;
        ncav += __popc(cm);
        qhead += n;
        if (ncav > W::CAV) {
            rc = REC_LARGE;
            go = false;
        }
        int items = go ? 4 * (ncav - base) : 0;
        __syncwarp();
        for (int k = hl; __any_sync(FULL, k < items); k += 16) {
            bool fresh = false;
            int sl = none_slot;
            if (k < items) {
                const int nb = reinterpret_cast<const int *>(ws.wave)[k];
                if (nb >= 0) sl = hash_insert(ws.hkey, W::HS, nb, fresh, full);
                ws.nsl[4 * base + k] = (uint8_t)sl;
            }
            const unsigned pm = ballot(fresh);
            const int qi = qtail + __popc(pm & lt);
            if (fresh && qi < W::QCAP) ws.queue[qi] = (uint8_t)sl;
            qtail += __popc(pm);
            if (qtail > W::QCAP) {
                rc = REC_LARGE;
                go = false;
                items = 0;
            }
        }
        __syncwarp();
    }
    if (rc == REC_DONE && ncav > REC_CAV) rc = REC_WIDE;
    const int nrec = rc == REC_DONE ? ncav : 0;
    // cavity-local neighbour indices (every neighbour has been tested by now)
    for (int k = hl; k < 4 * nrec; k += 16) ws.cav_nbr[k] = ws.hval[ws.nsl[k]];
    __syncwarp();
    head.ncav = nrec;
    for (int c = hl; c < nrec; c += 16) {
        const int nb = *reinterpret_cast<const int *>(&ws.cav_nbr[4 * c]);
        const unsigned out = (unsigned)nb & 0x80808080u;
        RowEntry e;
        e.tet = ws.cav_tet[c];
        e.bmask = (out >> 7 | out >> 14 | out >> 21 | out >> 28) & 15u;
        e.nbr = nb;
        e.pos = 0;
        ent[c] = e;
    }
    return rc;
}

// The corner term of cavity tet t at its vertex vi (natural_insertionfree.c:
// 642-676): the subcell volume at p[vi] from the tet's circumcentre and those
// of its three faces through p[vi].  Bit i of mask: the face opposite p[i]
// takes the copy of the neighbour across it, as natinterp3d's face cache does
// when that neighbour was visited earlier (:233-253).  A term depends on
// nothing but the mesh and the mask, so that meshes of up to CORNER_TETS_MAX
// tets hold all of them (MeshView::corner, four a tet and mask: a cavity tet
// is one 32-byte sector to a row instead of four vertices, five circumcentres
// and some 110 FP64 operations a corner).  For larger meshes k_rows_terms writes
// them beside the records of a chunk.
__device__ __forceinline__ double corner_term(const MeshView &M, int t, unsigned mask, int vi) {
    const int4 p = M.tv[t];
    const int4 n = M.tn[t];
    const uint32_t info = M.tinfo[t];
    auto face = [&](int i) {
        const int j = 3 - i;
        const int nb = comp(n, j);
        const int k = ((mask >> i) & 1u) && nb >= 0 ? 4 * nb + (3 - (int)((info >> (8 + 2 * j)) & 3u))
                                                    : 4 * t + i;
        return cload(&M.fcc[k]);
    };
    // the other three vertices in ascending slot order
    const int o0 = vi == 0 ? 1 : 0, o1 = vi <= 1 ? 2 : 1, o2 = vi <= 2 ? 3 : 2;
    return subcell_volume(vload(M, comp(p, vi)), vload(M, comp(p, o0)), vload(M, comp(p, o1)),
                          vload(M, comp(p, o2)), cload(&M.tcc[t]), face(o2), face(o1), face(o0));
}

// The same for all eight choices of copies of the three faces through p[vi] (bit
// 0, 1, 2 of the index: the lowest, middle and highest of them takes the
// neighbour's).  A face's copy enters one of the term's three cross products, so
// that the eight share six of them; each is summed in corner_term's order.
__device__ __forceinline__ void corner_terms(const MeshView &M, int t, int vi, double (&out)[8]) {
    const int4 p = M.tv[t];
    const int4 n = M.tn[t];
    const uint32_t info = M.tinfo[t];
    const int o0 = vi == 0 ? 1 : 0, o1 = vi <= 1 ? 2 : 1, o2 = vi <= 2 ? 3 : 2;
    const dv3 pk = vload(M, comp(p, vi));
    const dv3 pa = vload(M, comp(p, o0)), pb = vload(M, comp(p, o1)), pc = vload(M, comp(p, o2));
    const dv3 dt = vsub(cload(&M.tcc[t]), pk);
    const bool swap = vdot(vsub(pa, pk), vcross(vsub(pb, pk), vsub(pc, pk))) < 0;
    auto copy = [&](int i, int taken) {
        const int j = 3 - i;
        const int nb = comp(n, j);
        const int k = taken && nb >= 0 ? 4 * nb + (3 - (int)((info >> (8 + 2 * j)) & 3u)) : 4 * t + i;
        return vsub(cload(&M.fcc[k]), pk);
    };
    auto products = [](dv3 e, dv3 c) { return dv3{fmul(e.x, c.x), fmul(e.y, c.y), fmul(e.z, c.z)}; };
    const dv3 e1 = vsub(pa, pb), e2 = vsub(pa, pc), e3 = vsub(pb, pc);
    double first[2];   // of the face opposite o2
    dv3 next[2], last[2];
#pragma unroll
    for (int c = 0; c < 2; c++) {
        const dv3 m1 = products(e1, vcross(copy(o2, c), dt));
        const dv3 m2 = products(e2, vcross(dt, copy(o1, c)));
        const dv3 m3 = products(e3, vcross(copy(o0, c), dt));
        first[c] = fadd(fadd(m1.x, m1.y), m1.z);
        next[c] = swap ? m3 : m2;
        last[c] = swap ? m2 : m3;
    }
    double sum[2][2][2];
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const double ab = fadd(fadd(fadd(first[a], next[b].x), next[b].y), next[b].z);
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const double v = fadd(fadd(fadd(ab, last[c].x), last[c].y), last[c].z);
                sum[a][b][c] = div12(swap ? -v : v);
            }
        }
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int h = k >> 2, m = (k >> 1) & 1, l = k & 1;
        out[k] = swap ? sum[h][l][m] : sum[h][m][l];
    }
}

// the ids of a face's three vertices, one byte each, from its tet's ids
__device__ __forceinline__ unsigned face_ids(unsigned lid, int f) {
    // byte selectors of getFaceVerticies3's slots: (0, 1, 2), (3, 1, 0), (0, 2, 3), (3, 2, 1)
    const unsigned sel = f == 0 ? 0x0210u : (f == 1 ? 0x0013u : (f == 2 ? 0x0320u : 0x0123u));
    return __byte_perm(lid, 0, sel) & 0xffffffu;
}

__device__ __forceinline__ dv3 sload(const double (&p)[3]) { return dv3{p[0], p[1], p[2]}; }
__device__ __forceinline__ void sstore(double (&p)[3], const dv3 &v) {
    p[0] = v.x;
    p[1] = v.y;
    p[2] = v.z;
}

// The split row, part 2: from a record of part 1 (state RS_OK) the row as
// sibson_row returns it (steps 3-5, or the coincident-vertex row).  With
// FULL = false it stops at the neighbours and the boundary faces.
//
// Bound by the shared-memory pipe (81 % of its wavefronts) and instruction issue
// (70 %, 2,580 warp instructions a row), and by instruction fetch where the code
// outgrows the instruction cache: loops are not unrolled (unrolled 12.2 ms a
// 2M-row call on 200k keys, rolled 8.4), and what a row shares is computed once.
// With what follows such a call's rows take 6.1 ms; 11.7 ms with a tet's terms
// evaluated per row, both of an edge's circumcentres per face and a lane a face.
//  - vertices get their id once per cavity tet (one hash pass over the tets'
//    vertices), and their positions are staged by id;
//  - cavity terms come from the mesh's corner table;
//  - a lane takes a corner of a boundary face;
//  - a triangle circumcentre (u, q, w) belongs to a directed boundary edge:
//    the two faces that share the edge each need both directions, so a corner
//    computes one and reads the other from the face that the sets of u's and
//    w's faces have in common;
//  - a neighbour's terms are stored next to each other, in natinterp3d's item
//    order (a term's place is the number of the neighbour's tets or faces
//    before it, from the same sets), and one lane a neighbour adds them.
// GENERAL = false gives up (ST_GENERAL) on rows of more than 32 neighbours or
// W::BF faces, on flat triangles and tets (natinterp3d's centroid fallbacks)
// and on edges that are not shared by two faces; GENERAL = true, a kernel of
// its own, takes those from the start.
constexpr int ST_GENERAL = 8;

__device__ __forceinline__ int scan_add(int v, int lane) {  // inclusive, over the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// term[0 .. n) added to a in order
__device__ __forceinline__ void add_terms(double &a, const double *term, int n) {
#pragma unroll 1
    for (int i = 0; i < n; i++) a = fadd(a, term[i]);
}

// The row's neighbours as lane l of the warp holds them: neighbour l (and
// l + 32), its vertex, its column and its stolen volume (split_row_body), or its
// weight (split_weights).
template <int IDS>
struct RowLanes {
    double a[IDS];
    int col[IDS], vid[IDS];
    __device__ __forceinline__ RowLanes() {  // no neighbour
#pragma unroll
        for (int i = 0; i < IDS; i++) {
            a[i] = 0.0;
            col[i] = 63;
            vid[i] = 0;
        }
    }
};

// TERMS: the row's corner terms are at ent_terms, by entry, on meshes without the table.
template <int G, class W, bool FULL, bool GENERAL, bool TERMS, int IDS>
__device__ __forceinline__ void split_row_body(const MeshView &M, const dv3 q, W &ws, const Grp<G> &g,
                                               const RowHead &head, const RowEntry *__restrict__ ent,
                                               const d4 *__restrict__ ent_terms, RowInfo &r,
                                               RowLanes<IDS> &out) {
    static_assert(G == 32, "one warp a row");
    constexpr int FW = W::FW;
    static_assert(GENERAL || FW == 1, "a face set is one word of the common rows");
    static_assert(IDS == (GENERAL ? 2 : 1), "neighbours of a lane");
    const int ncav = head.ncav;
    const int lane = g.lane;
    if (ncav == 0) {
        // natural_insertionfree.c:596-622, as coincident_row
        int v = -1;
        bool co = false;
        if (lane < 4) {
            v = comp(M.tv[head.start], lane);
            co = v < M.n && veq(vload(M, v), q);
        }
        const unsigned cm = g.ballot(co);
        r.nnb = __popc(cm);
        r.coincident = true;
        out.vid[0] = v;
        if (co) out.col[0] = __popc(cm & g.lt());
        out.a[0] = r.nnb > 0 ? fdiv(1.0, (double)r.nnb) : 0.0;
        return;
    }
    auto &C = ws.u.c;

    // ---- the cavity's vertices, numbered by hash slot -----------------------
    static_assert(W::VH == 64, "one 8-byte clear a lane");
    reinterpret_cast<int2 *>(C.h.vh_key)[lane] = make_int2(-1, -1);
    reinterpret_cast<int2 *>(C.h.vh_first)[lane] = make_int2(INT_MAX, INT_MAX);
    if (lane < VOL_VERTS / 2)
        reinterpret_cast<ulonglong2 *>(C.tm)[lane] = make_ulonglong2(0ull, 0ull);
#pragma unroll
    for (int w = 0; w < FW; w++)
        if (lane < VOL_VERTS / 2)
            reinterpret_cast<ulonglong2 *>(ws.fm)[w * (VOL_VERTS / 2) + lane] = make_ulonglong2(0ull, 0ull);
    static_assert(sizeof(C.firsts) <= 32 * sizeof(unsigned), "one clear a lane");
    if (lane < (int)(sizeof(C.firsts) / sizeof(unsigned))) C.firsts[lane] = 0u;
    g.sync();
    bool vfull = false;
    d4 terms{0.0, 0.0, 0.0, 0.0};  // the corner terms of the lane's first tet, on their way early
    int first_o = 0;
#pragma unroll 1
    for (int e = lane; e < ncav; e += 32) {
        // the record is in the flood's order: each tet goes to its position in
        // natinterp3d's visiting order
        const RowEntry x = ent[e];
        const int o = min(x.pos & 0xff, ncav - 1);  // a permutation of 0..ncav-1
        const int4 p = M.tv[x.tet];
        if (FULL && e < 32) {
            first_o = o;
            if (!GENERAL) {
                if (TERMS && !M.corner)
                    terms = ent_terms[e];
                else
                    terms = M.corner[16 * (size_t)x.tet + (((unsigned)x.pos >> 8) & 15u)];
            }
        }
        unsigned slots = 0;
        // most vertices get the slot of their hash or the one beside it, all four
        // tried at once
        int s[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int v = comp(p, i);
            s[i] = (int)(mix_hash(v) >> 26);
            if (v < M.n) {
                int old = atomicCAS(&C.h.vh_key[s[i]], -1, v);
                if (old != -1 && old != v) {
                    s[i] ^= 1;
                    old = atomicCAS(&C.h.vh_key[s[i]], -1, v);
                    if (old != -1 && old != v) s[i] = -1;
                }
            } else {
                s[i] = 0x80 | (v - M.n);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) slots |= ((unsigned)s[i] & 0xffu) << (8 * i);
        if ((s[0] | s[1] | s[2] | s[3]) < 0) {
#pragma unroll 1
            for (int i = 0; i < 4; i++)
                if (((slots >> (8 * i)) & 0xffu) == 0xffu) {
                    const int t = hash_upsert(C.h.vh_key, W::VH, comp(p, i), vfull);
                    slots ^= (0xffu ^ ((unsigned)t & 0xffu)) << (8 * i);
                }
        }
        C.tet[o] = x.tet;
        C.lid[o] = slots;
        C.mask[o] = (uint8_t)((x.bmask & 0xfu) | (((unsigned)x.pos >> 4) & 0xf0u));
    }
    if (g.any(vfull)) {
        r.status = ST_CAPACITY;
        return;
    }
    g.sync();

    // ---- 3. boundary faces (visiting order, then face order) -----------------
    int nbf = 0;
#pragma unroll 1
    for (int o0 = 0; o0 < ncav; o0 += 32) {
        const int o = o0 + lane;
        const unsigned m = o < ncav ? C.mask[o] & 15u : 0u;
        const int end = nbf + scan_add(__popc(m), lane);
        int b = end - __popc(m);
#pragma unroll
        for (int f = 0; f < 4; f++)
            if ((m >> f) & 1u) {
                if (b < W::BF) ws.bff[b] = 4 * o + f;
                b++;
            }
        nbf = g.shfl(end, 31);
    }
    if (nbf > W::BF) {
        r.status = GENERAL ? ST_CAPACITY : ST_GENERAL;
        return;
    }
    r.nbf = nbf;
    g.sync();
#pragma unroll 1
    for (int b = lane; b < nbf; b += 32) {
        const int cf = ws.bff[b];
        const unsigned ids = face_ids(C.lid[cf >> 2], cf & 3);
        ws.fid[b] = ids;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const int s = (ids >> (8 * j)) & 0xff;
            if (s < 0x80) atomicMin(&C.h.vh_first[s], 3 * b + j);
        }
    }
    g.sync();

    // ids of the boundary faces' vertices; vh_first becomes the slot's id
    int nnb = 0;
#pragma unroll
    for (int i = 0; i < W::VH; i += 32) {
        const int s = i + lane;
        const int k = C.h.vh_first[s];
        const unsigned m = g.ballot(k != INT_MAX);
        const int id = nnb + __popc(m & g.lt());
        C.h.vh_first[s] = k == INT_MAX ? VOL_NO_ID : id;
        if (k != INT_MAX && id < W::NBR) {
            ws.nbr_vid[id] = C.h.vh_key[s];
            ws.start[id] = k;
            atomicOr(&C.firsts[k >> 5], 1u << (k & 31));
        }
        nnb += __popc(m);
    }
    if (nnb > W::NBR) {
        r.status = ST_CAPACITY;
        return;
    }
    if (!GENERAL && nnb > 32) {
        r.status = ST_GENERAL;
        return;
    }
    g.sync();
    if (nnb == 0) return;

    // the neighbour of each lane: its vertex and column (the order of first corners)
#pragma unroll
    for (int i = 0; i < IDS; i++) {
        const int id = lane + 32 * i;
        if (id < nnb) {
            const int k = ws.start[id];
            const int v = ws.nbr_vid[id];
            sstore(ws.pos[id], vload(M, v));
            out.vid[i] = v;
            int c = __popc(C.firsts[k >> 5] & ((1u << (k & 31)) - 1u));
#pragma unroll 1
            for (int w = 0; w < k >> 5; w++) c += __popc(C.firsts[w]);
            out.col[i] = c;
        }
    }
    if (lane < 4) sstore(ws.pos[nnb + lane], vload(M, M.n + lane));

    // hash slots to ids, and each id's sets of tets and faces
    auto to_id = [&](unsigned s) { return s < 0x80u ? C.h.vh_first[s] : nnb + (int)(s & 3u); };
    if constexpr (FULL) {
#pragma unroll 1
        for (int o = lane; o < ncav; o += 32) {
            const unsigned w = C.lid[o];
            unsigned ids = 0;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int id = to_id((w >> (8 * i)) & 0xffu);
                ids |= (unsigned)id << (8 * i);
                if (id < nnb) atomicOr(reinterpret_cast<unsigned *>(&C.tm[id]) + (o >> 5), 1u << (o & 31));
            }
            C.lid[o] = ids;
        }
    }
#pragma unroll 1
    for (int b = lane; b < nbf; b += 32) {
        const int cf = ws.bff[b];
        const unsigned w = ws.fid[b];
        unsigned ids = 0;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const int id = to_id((w >> (8 * j)) & 0xffu);
            ids |= (unsigned)id << (8 * j);
            atomicOr(reinterpret_cast<unsigned *>(&ws.fm[FW * id]) + (b >> 5), 1u << (b & 31));
        }
        ws.fid[b] = ids;
        ws.bff[b] = 4 * C.tet[cf >> 2] + 3 - (cf & 3);
    }
    g.sync();
    if constexpr (!FULL) {
        // the neighbours in column order, and each id's column
#pragma unroll
        for (int i = 0; i < IDS; i++)
            if (lane + 32 * i < nnb) {
                ws.nbr_vid[out.col[i]] = out.vid[i];
                ws.start[lane + 32 * i] = out.col[i];
            }
        g.sync();
        r.nnb = nnb;
        return;
    }

    // where each neighbour's terms go: lane l adds up those of neighbour l (and l + 32)
    int n[IDS], at[IDS];  // number and first place, cavity terms | face terms << 16
    {
        int base = 0;
#pragma unroll
        for (int i = 0; i < IDS; i++) {
            const int id = lane + 32 * i;
            n[i] = 0;
            if (id < nnb) {
                n[i] = __popcll(C.tm[id]);
#pragma unroll
                for (int w = 0; w < FW; w++) n[i] += __popcll(ws.fm[FW * id + w]) << 16;
            }
            at[i] = base + scan_add(n[i], lane);
            base = g.shfl(at[i], 31);
            at[i] -= n[i];
            if (id < nnb) ws.start[id] = at[i];
        }
    }
    g.sync();

    // ---- 4. stolen volumes -----------------------------------------------------
#pragma unroll 1
    for (int e = lane; e < ncav; e += 32) {
        int o = first_o;
        if (e >= 32) o = min(ent[e].pos & 0xff, ncav - 1);
        if (GENERAL || e >= 32) {
            const int t = C.tet[o];
            const unsigned m = C.mask[o] >> 4;
            if (TERMS && !M.corner)
                terms = ent_terms[e];
            else
                terms = M.corner[16 * (size_t)t + m];
        }
        const unsigned ids = C.lid[o];
        const unsigned long long below = (1ull << o) - 1ull;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int id = (ids >> (8 * i)) & 0xff;
            if (id < nnb)
                C.term[(ws.start[id] & 0xffff) + __popcll(C.tm[id] & below)] =
                    i == 0 ? terms.x : (i == 1 ? terms.y : (i == 2 ? terms.z : terms.w));
        }
    }
    g.sync();
#pragma unroll
    for (int i = 0; i < IDS; i++) {
        add_terms(out.a[i], C.term + (at[i] & 0xffff), n[i] & 0xffff);
    }
    g.sync();

    // virtual-tet terms, query + boundary face (:681-719), a lane a face corner
    bool general = false;  // !GENERAL: the row is not for this body
    auto &V = ws.u.v;
    using corner_t = typename W::corner_t;
    const int ne = 3 * nbf;
    const int S = nnb + 4;
    using edge_t = typename W::edge_t;
#pragma unroll 1
    for (int i = lane; i < (S * S * (int)sizeof(edge_t) + 15) / 16; i += 32)
        reinterpret_cast<uint4 *>(ws.u.pair)[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
    g.sync();
#pragma unroll 1
    for (int k = lane; k < ne; k += 32) {
        const int b = k / 3, j = k - 3 * b;
        const unsigned rot = __byte_perm(ws.fid[b], 0, j == 0 ? 0x3210u : (j == 1 ? 0x3021u : 0x3102u));
        const unsigned u = rot & 0xffu, w = (rot >> 8) & 0xffu, x = rot >> 16;
        ws.u.pair[u * S + w] = (edge_t)k;
        // the faces of u before this one
        int place = 0;
        if (u < (unsigned)nnb) {
            place = ws.start[u] >> 16;
#pragma unroll
            for (int i = 0; i < FW; i++) {
                const unsigned long long mu = ws.fm[FW * u + i];
                if (FW == 1 || b >> 6 == i)
                    place += __popcll(mu & ((1ull << (b & 63)) - 1ull));
                else if (b >> 6 > i)
                    place += __popcll(mu);
            }
        }
        ws.corner[k] = (corner_t)(u | w << 6 | x << 12) | (corner_t)place << (18 + W::EB);
    }
    g.sync();
#pragma unroll 1
    for (int k = lane; k < ne; k += 32) {
        const corner_t cn = ws.corner[k];
        const unsigned e = ws.u.pair[((unsigned)cn & 63) * S + (((unsigned)cn >> 12) & 63)];
        ws.corner[k] = cn | (corner_t)(e & ((1u << W::EB) - 1u)) << 18;
        if (!GENERAL) general |= e == W::NO_EDGE;
    }
    g.sync();
#pragma unroll 1
    for (int k = lane; k < ne; k += 32) {
        const unsigned cn = (unsigned)ws.corner[k];
        const int u = cn & 63;
        if (u < nnb) {
            const dv3 pu = sload(ws.pos[u]), pw = sload(ws.pos[(cn >> 6) & 63]);
            bool flat = false;
            const dv3 c = GENERAL ? tri_cc(pu, q, pw) : tri_cc_regular(pu, q, pw, flat);
            general |= flat;
            sstore(V.ec[k], vsub(c, pu));
        }
    }
#pragma unroll 1
    for (int b = lane; b < nbf; b += 32) {
        const unsigned ids = ws.fid[b];
        const dv3 pa = sload(ws.pos[ids & 0xff]), pb = sload(ws.pos[(ids >> 8) & 0xff]),
                  pc = sload(ws.pos[ids >> 16]);
        if (GENERAL) {
            sstore(V.ct[b], tet_cc(q, pa, pb, pc));
        } else {
            // The orientation of (q, w, x) about each corner u has the exact value
            // -det(a - q, b - q, c - q) = -den / 2.  With l the longest of the three
            // vectors (edges are below 2 l), both computed values are within
            // 200 eps l^3 = 2.3e-14 l^3 of it, so that beyond 1e-13 l^3 they have its
            // sign: one orientation a face instead of one a corner (23 of a corner's
            // 85 FP64 operations).
            bool flat = false;
            double den, l2;
            sstore(V.ct[b], tet_cc_regular(q, pa, pb, pc, flat, den, l2));
            general |= flat || !(den * den > 1e-26 * l2 * l2 * l2);
            if (den > 0.0) ws.bff[b] |= INT_MIN;  // a negative orientation
        }
    }
    if (!GENERAL && g.any(general)) {
        r.status = ST_GENERAL;
        return;
    }
    g.sync();
#pragma unroll 1
    for (int k = lane; k < ne; k += 32) {
        const corner_t cn = ws.corner[k];
        const int u = (unsigned)cn & 63;
        if (u < nnb) {
            const int b = k / 3;
            constexpr unsigned NONE = (1u << W::EB) - 1u;
            const unsigned e = (unsigned)(cn >> 18) & NONE;
            const int ffi = ws.bff[b];
            const dv3 cf = cload(&M.fcc[ffi & INT_MAX]);
            const dv3 pu = sload(ws.pos[u]), pw = sload(ws.pos[((unsigned)cn >> 6) & 63]),
                      px = sload(ws.pos[((unsigned)cn >> 12) & 63]);
            dv3 dac;
            if (GENERAL && e == NONE)
                dac = vsub(tri_cc(pu, q, px), pu);
            else
                dac = sload(V.ec[e]);
            // subcell_volume(u, q, w, x, ct, cc(u, q, w), cc(u, q, x), cf)
            const bool swap = GENERAL ? vdot(vsub(q, pu), vcross(vsub(pw, pu), vsub(px, pu))) < 0 : ffi < 0;
            ws.fterm[(unsigned)(cn >> (18 + W::EB))] =
                -subcell_from(swap, vsub(q, pw), vsub(q, px), vsub(pw, px), sload(V.ec[k]), dac, vsub(cf, pu),
                              vsub(sload(V.ct[b]), pu));
        }
    }
    g.sync();
#pragma unroll
    for (int i = 0; i < IDS; i++) add_terms(out.a[i], ws.fterm + (at[i] >> 16), n[i] >> 16);
    r.nnb = nnb;
}

// ---- 5. normalisation: the lanes' stolen volumes to weights; r.nnb = 0 where
// the row is empty.  The total is added up in column order.
template <int G, class W, int IDS>
__device__ __forceinline__ void split_weights(W &ws, const Grp<G> &g, RowInfo &r, RowLanes<IDS> &out) {
    if (r.coincident || r.nnb == 0) return;
    const int nnb = r.nnb;
#pragma unroll
    for (int i = 0; i < IDS; i++)
        if (out.col[i] < nnb) ws.acc[out.col[i]] = out.a[i];
    g.sync();
    double total = 0.0;
#pragma unroll 4
    for (int s = 0; s < nnb; s++) total = fadd(total, ws.acc[s]);
    if (!(total > 1e-30)) {
        r.nnb = 0;
        return;
    }
    const double inv = frcp(total);
#pragma unroll
    for (int i = 0; i < IDS; i++) out.a[i] = fmul(out.a[i], inv);
    r.total = total;
}

}  // namespace nif
