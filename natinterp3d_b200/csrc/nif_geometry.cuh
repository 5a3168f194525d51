// FP64 geometry for the Sibson query kernels.
//
// Every operation is an explicitly rounded IEEE-754 double operation
// (__dadd_rn / __dsub_rn / __dmul_rn / __ddiv_rn), which the compiler never
// contracts into fused multiply-adds.  Each expression keeps the operand
// grouping of natinterp3d's C code (compiled there with -std=c11 and no
// -march, hence no FMA), so every determinant, circumcentre and volume below
// is bit-identical to natinterp3d's on the same inputs:
//   orient3dfast / inspherefast     predicates.c:1687-1710, 3301-3347
//   circumCenterTri3D               natural_insertionfree.c:24-49
//   circumCenterTet                 natural_insertionfree.c:54-84
//   voronoiSubcellVolume            natural_insertionfree.c:92-146
#pragma once
#include <cuda_runtime.h>

// The four large routines are inlined (measured faster on B200 than calls,
// which spill the FP64 state around each call); NIF_GEOM_OUTLINE compiles
// them out of line instead.
#ifdef NIF_GEOM_OUTLINE
#define NIF_GEOM_FN __device__ __noinline__
#else
#define NIF_GEOM_FN __device__ __forceinline__
#endif

namespace nif {

struct dv3 {
    double x, y, z;
};

__device__ __forceinline__ double fadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double fsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double fmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double fdiv(double a, double b) { return __ddiv_rn(a, b); }

// 1 / x: the correctly rounded reciprocal, the same bits as fdiv(1.0, x)
__device__ __forceinline__ double frcp(double x) { return __drcp_rn(x); }

// x / 12, correctly rounded, in three operations: with y the correctly
// rounded 1/12 and q = x y (within one ulp of the quotient), the residual
// r = x - 12 q is exact and q + r y rounds to x / 12 (Markstein, "Computation
// of elementary functions on the IBM RISC System/6000 processor", 1990,
// theorem on division from a correctly rounded reciprocal).  That needs r
// representable: numbers near the ends of the exponent range, infinities and
// NaN take the plain division.
__device__ __forceinline__ double div12(double x) {
    const double y = 1.0 / 12.0;
    const double q = fmul(x, y);
    const unsigned e = ((unsigned)__double2hiint(x) >> 20) & 0x7ffu;
    if (e - 100u < 1900u) return __fma_rn(__fma_rn(-12.0, q, x), y, q);
    return fdiv(x, 12.0);
}

__device__ __forceinline__ dv3 mk(double x, double y, double z) { return dv3{x, y, z}; }
__device__ __forceinline__ dv3 mk(const double4 &v) { return dv3{v.x, v.y, v.z}; }
__device__ __forceinline__ dv3 vsub(dv3 a, dv3 b) { return dv3{fsub(a.x, b.x), fsub(a.y, b.y), fsub(a.z, b.z)}; }
__device__ __forceinline__ dv3 vadd(dv3 a, dv3 b) { return dv3{fadd(a.x, b.x), fadd(a.y, b.y), fadd(a.z, b.z)}; }
__device__ __forceinline__ dv3 vscale(dv3 a, double s) { return dv3{fmul(a.x, s), fmul(a.y, s), fmul(a.z, s)}; }
// b x c with natinterp3d's component formulas (delaunay.c:986-990)
__device__ __forceinline__ dv3 vcross(dv3 b, dv3 c) {
    return dv3{fsub(fmul(b.y, c.z), fmul(b.z, c.y)), fsub(fmul(b.z, c.x), fmul(b.x, c.z)),
               fsub(fmul(b.x, c.y), fmul(b.y, c.x))};
}
// (a0 b0 + a1 b1) + a2 b2  (delaunay.c:994-996)
__device__ __forceinline__ double vdot(dv3 a, dv3 b) {
    return fadd(fadd(fmul(a.x, b.x), fmul(a.y, b.y)), fmul(a.z, b.z));
}
__device__ __forceinline__ bool veq(dv3 a, dv3 b) { return a.x == b.x && a.y == b.y && a.z == b.z; }

// orient3dfast(a, b, c, d) = det[a-d; b-d; c-d]
__device__ __forceinline__ double orient_fast(dv3 a, dv3 b, dv3 c, dv3 d) {
    dv3 u = vsub(a, d), v = vsub(b, d), w = vsub(c, d);
    double t0 = fmul(u.x, fsub(fmul(v.y, w.z), fmul(v.z, w.y)));
    double t1 = fmul(v.x, fsub(fmul(w.y, u.z), fmul(w.z, u.y)));
    double t2 = fmul(w.x, fsub(fmul(u.y, v.z), fmul(u.z, v.y)));
    return fadd(fadd(t0, t1), t2);
}

// inspherefast(a, b, c, d, e): lifted 4x4 determinant relative to e
NIF_GEOM_FN double insphere_fast(dv3 a, dv3 b, dv3 c, dv3 d, dv3 e) {
    dv3 r0 = vsub(a, e), r1 = vsub(b, e), r2 = vsub(c, e), r3 = vsub(d, e);
    // 2x2 minors of the (x, y) columns: m(i,j) = x_i y_j - x_j y_i
    double m01 = fsub(fmul(r0.x, r1.y), fmul(r1.x, r0.y));
    double m12 = fsub(fmul(r1.x, r2.y), fmul(r2.x, r1.y));
    double m23 = fsub(fmul(r2.x, r3.y), fmul(r3.x, r2.y));
    double m30 = fsub(fmul(r3.x, r0.y), fmul(r0.x, r3.y));
    double m02 = fsub(fmul(r0.x, r2.y), fmul(r2.x, r0.y));
    double m13 = fsub(fmul(r1.x, r3.y), fmul(r3.x, r1.y));
    double abc = fadd(fsub(fmul(r0.z, m12), fmul(r1.z, m02)), fmul(r2.z, m01));
    double bcd = fadd(fsub(fmul(r1.z, m23), fmul(r2.z, m13)), fmul(r3.z, m12));
    double cda = fadd(fadd(fmul(r2.z, m30), fmul(r3.z, m02)), fmul(r0.z, m23));
    double dab = fadd(fadd(fmul(r3.z, m01), fmul(r0.z, m13)), fmul(r1.z, m30));
    double l0 = vdot(r0, r0), l1 = vdot(r1, r1), l2 = vdot(r2, r2), l3 = vdot(r3, r3);
    return fadd(fsub(fmul(l3, abc), fmul(l2, dab)), fsub(fmul(l1, cda), fmul(l0, bcd)));
}

// circumcentre of triangle (a, b, c); centroid when |ab x ac|^2 < 1e-30
// (tri_cc_regular: the circumcentre's own formula, `flat` set where the
// centroid is wanted; tri_cc leaves it out there: where every triangle is flat,
// 200k rows of the fused kernel take 2,958 us, 2,997 with both)
__device__ __forceinline__ dv3 tri_cc_from(dv3 a, dv3 ab, dv3 ac, dv3 n, double n2) {
    double ab2 = vdot(ab, ab), ac2 = vdot(ac, ac);
    dv3 t = dv3{fsub(fmul(ab2, ac.x), fmul(ac2, ab.x)), fsub(fmul(ab2, ac.y), fmul(ac2, ab.y)),
                fsub(fmul(ab2, ac.z), fmul(ac2, ab.z))};
    dv3 cr = vcross(t, n);
    double inv = frcp(fmul(2.0, n2));
    return vadd(a, vscale(cr, inv));
}

__device__ __forceinline__ dv3 tri_cc_regular(dv3 a, dv3 b, dv3 c, bool &flat) {
    const dv3 ab = vsub(b, a), ac = vsub(c, a), n = vcross(ab, ac);
    const double n2 = vdot(n, n);
    flat = n2 < 1e-30;
    return tri_cc_from(a, ab, ac, n, n2);
}

NIF_GEOM_FN dv3 tri_cc(dv3 a, dv3 b, dv3 c) {
    const dv3 ab = vsub(b, a), ac = vsub(c, a), n = vcross(ab, ac);
    const double n2 = vdot(n, n);
    if (n2 < 1e-30)
        return dv3{fdiv(fadd(fadd(a.x, b.x), c.x), 3.0), fdiv(fadd(fadd(a.y, b.y), c.y), 3.0),
                   fdiv(fadd(fadd(a.z, b.z), c.z), 3.0)};
    return tri_cc_from(a, ab, ac, n, n2);
}

// circumcentre of tetrahedron (a, b, c, d); centroid when |denominator| < 1e-30
// (tet_cc_regular: as tri_cc_regular; also the denominator, twice the
// determinant of the edges from a, and the longest edge squared)
__device__ __forceinline__ dv3 tet_cc_regular(dv3 a, dv3 b, dv3 c, dv3 d, bool &flat, double &den,
                                              double &l2) {
    dv3 ba = vsub(b, a), ca = vsub(c, a), da = vsub(d, a);
    dv3 x1 = vcross(ba, ca), x2 = vcross(da, ba), x3 = vcross(ca, da);
    const double lb = vdot(ba, ba), lc = vdot(ca, ca), ld = vdot(da, da);
    l2 = fmax(lb, fmax(lc, ld));
    dv3 m1 = vscale(x1, ld);
    dv3 m2 = vscale(x2, lc);
    dv3 m3 = vscale(x3, lb);
    dv3 s = vadd(m3, vadd(m1, m2));
    den = fmul(2.0, vdot(ba, x3));
    flat = fabs(den) < 1e-30;
    return vadd(vscale(s, frcp(den)), a);
}

NIF_GEOM_FN dv3 tet_cc(dv3 a, dv3 b, dv3 c, dv3 d) {
    bool flat;
    double den, l2;
    const dv3 r = tet_cc_regular(a, b, c, d, flat, den, l2);
    if (flat)
        return dv3{fmul(fadd(fadd(fadd(a.x, b.x), c.x), d.x), 0.25),
                   fmul(fadd(fadd(fadd(a.y, b.y), c.y), d.y), 0.25),
                   fmul(fadd(fadd(fadd(a.z, b.z), c.z), d.z), 0.25)};
    return r;
}

// The subcell volume from the orientation of (pa, pb, pc) about pk (`swap`: it is
// negative), the edges e1 = pa - pb, e2 = pa - pc, e3 = pb - pc, and the face circumcentres
// (dab, dac, dbc) and the tet's (dt), relative to pk.  natinterp3d then swaps pa
// with pb and dac with dbc: that negates e1, exchanges e2 with e3
// and turns the cross products into (c1, -c3, -c2), so that the swapped sum is
// the negated sum of the same nine products in the order 1, 3, 2 (a rounded
// operation on negated operands gives the negated result).
__device__ __forceinline__ double subcell_from(bool swap, dv3 e1, dv3 e2, dv3 e3, dv3 dab, dv3 dac,
                                               dv3 dbc, dv3 dt) {
    const dv3 c1 = vcross(dab, dt), c2 = vcross(dt, dac), c3 = vcross(dbc, dt);
    const dv3 m2{fmul(e2.x, c2.x), fmul(e2.y, c2.y), fmul(e2.z, c2.z)};
    const dv3 m3{fmul(e3.x, c3.x), fmul(e3.y, c3.y), fmul(e3.z, c3.z)};
    double vol = fadd(fadd(fmul(e1.x, c1.x), fmul(e1.y, c1.y)), fmul(e1.z, c1.z));
    if (swap) {
        vol = fadd(fadd(fadd(vol, m3.x), m3.y), m3.z);
        vol = -fadd(fadd(fadd(vol, m2.x), m2.y), m2.z);
    } else {
        vol = fadd(fadd(fadd(vol, m2.x), m2.y), m2.z);
        vol = fadd(fadd(fadd(vol, m3.x), m3.y), m3.z);
    }
    return div12(vol);
}

// Signed volume of the part of tet (pk, pa, pb, pc) closer to pk than to the
// other vertices, from the tet circumcentre ct and the circumcentres of the
// three faces through pk (fab, fac, fbc); derivation in natinterp3d's
// docs/insertion-free.rst:88-165.
NIF_GEOM_FN double subcell_volume(dv3 pk, dv3 pa, dv3 pb, dv3 pc, dv3 ct, dv3 fab,
                                                dv3 fac, dv3 fbc) {
    dv3 ta = vsub(pa, pk), tb = vsub(pb, pk), tc = vsub(pc, pk);
    const double sv = vdot(ta, vcross(tb, tc));
    return subcell_from(sv < 0, vsub(pa, pb), vsub(pa, pc), vsub(pb, pc), vsub(fab, pk), vsub(fac, pk),
                        vsub(fbc, pk), vsub(ct, pk));
}

}  // namespace nif
