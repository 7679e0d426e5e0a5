// sf_voxel.cu -- SDF/CSG voxelisation on the GPU.
//
// Restates SDFPrimitive.voxelize (geometry/sdf.py:99-125 of
// rjwalters/strata-fdtd): the mask is sdf(cell centre) <= 0 with cell centres
// np.arange(n)*res + res/2 (core/grid.py:86-88).  Each thread evaluates one
// cell in FP64 with the reference's operation order and no fused
// multiply-add, so the mask matches NumPy bit for bit:
//   Box      sdf.py:274-293  |p-c| - size/2; norm(max(q,0)) + min(max_d q, 0)
//   Sphere   sdf.py:320-332  norm(p-c) - r
//   Cylinder sdf.py:382-424  projection, clamp, radial/axial distance
//   Union / Intersection / Difference  sdf.py:566-584, 629-647, 704-721
//   Translate / Scale        sdf.py:1225-1236, 1285-1294
//   Rotate                   sdf.py:1351-1355: point @ R (rows of R^T
//                            dotted in the order ((p0 m0 + p1 m1) + p2 m2))
//   Cone                     sdf.py:490-530  projection over the length,
//                            linearly interpolated radius, capped ends
//   Horn                     sdf.py:1085-1133  surface of revolution with
//                            the conical / exponential / hyperbolic /
//                            tractrix radius of sdf.py:1039-1060
//   HelicalTube, SpiralHorn  sdf.py:1666-1695, 1505-1554: distance to a
//                            polyline sampled on the host (paths.py:226-294)
//                            minus the radius at the nearest sample, the
//                            spiral in the xy plane and extruded over z
//   SmoothUnion / SmoothIntersection / SmoothDifference  sdf.py:760-781,
//                            827-847, 903-920: polynomial blends of two
// np.linalg.norm over three components sums ((x0^2 + x1^2) + x2^2).  The
// axis projections of cylinders, cones, horns and path segments use np.dot
// (BLAS), whose rounding depends on the BLAS build; here they are
// ((v0*a0 + v1*a1) + v2*a2), which equals any BLAS result exactly when the
// axis is a coordinate axis.  The horn radii call CUDA's exp, cosh and cos,
// which may differ from NumPy's in the last place: masks can then differ
// only at cells whose distance is within that rounding of zero.
//
// sf_launch_voxelize gets that mask without evaluating every cell in FP64
// (GB300 runs FP64 at about 1/64 of its FP32 rate, and one FP64 evaluation
// per cell was bound by that pipe: 16.2 ms for the 400^3 enclosure, 4 nodes).
// A second evaluator runs the same program, operation for operation, in FP32
// interval arithmetic with directed rounding.  A float bound is itself an
// FP64 number and FP64 rounding is monotonic, so each interval holds what the
// FP64 evaluator computes from any point of the box, roundings included: an
// interval wholly at or below zero, or wholly above, decides every cell in
// the box exactly as the FP64 evaluation would.  Blocks of 4 x 4 x 4 cells
// are decided (or queued) by k_vx_blocks (on large grids super-blocks of 16 x 16 x
// 32 before them, by k_vx_super), the queued blocks' cells one at a
// time by k_vx_cells, and only a cell whose own interval straddles zero is
// evaluated in FP64.  Solids of many parts are mostly decided by a few of them:
// a part of a union, intersection or difference that loses to another everywhere in
// a block is left out inside it.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "sf_common.cuh"
#include "sf_plan_internal.h"

namespace {

constexpr int VX_DSTACK = 32;
constexpr int VX_PSTACK = 12;

// A marker before a child of a union, intersection or difference (mark_program):
// op kSkip, n nodes to pass over, the child's bit in a[0], the value that stands
// for it in s0.
constexpr int kSkip = 30;
constexpr int kMaxParts = 64;
constexpr int kSuperMin = 2048;  // super-blocks from which on they are looked at first

__device__ __forceinline__ double norm3(double a, double b, double c) {
    return __dsqrt_rn(d_add(d_add(d_mul(a, a), d_mul(b, b)), d_mul(c, c)));
}
__device__ __forceinline__ double dmax(double a, double b) {  // np.maximum
    return (a >= b || a != a) ? a : b;
}
__device__ __forceinline__ double dmin(double a, double b) {  // np.minimum
    return (a <= b || a != a) ? a : b;
}

__device__ __forceinline__ double clip01(double t) { return dmin(dmax(t, 0.0), 1.0); }

// distance_to_polyline (paths.py:226-294) from (x, y, z) -- or (x, y) when
// dims == 2 -- to the path in nodes d[0 .. m-1] (a = vertex, b = the vertex's
// segment to the next one and s1 = its squared length, both computed on the
// host as the reference does; s0 = the radius there), minus the radius at the
// nearest vertex (the first of equal distances, as np.argmin).
__device__ double path_distance(const sf_sdf_node* __restrict__ d, int m, int dims, double x,
                                double y, double z) {
    double best = __longlong_as_double(0x7ff0000000000000LL);  // +inf
    double near = best;
    double radius = 0.0;
    for (int q = 0; q < m; ++q) {
        const sf_sdf_node& P = d[q];
        const double w0 = d_sub(x, P.a[0]), w1 = d_sub(y, P.a[1]);
        const double w2 = dims == 3 ? d_sub(z, P.a[2]) : 0.0;
        // nearest vertex: norm(path - point), squares as those of point - path
        const double dv = dims == 3 ? norm3(w0, w1, w2)
                                    : __dsqrt_rn(d_add(d_mul(w0, w0), d_mul(w1, w1)));
        if (dv < near) {
            near = dv;
            radius = P.s0;
        }
        if (q + 1 == m) break;
        double ds;
        if (P.s1 < 1e-14) {  // a degenerate segment is its first vertex
            ds = dv;
        } else {
            double t = d_add(d_mul(w0, P.b[0]), d_mul(w1, P.b[1]));
            if (dims == 3) t = d_add(t, d_mul(w2, P.b[2]));
            const double tc = clip01(__ddiv_rn(t, P.s1));
            const double c0 = d_add(P.a[0], d_mul(tc, P.b[0]));
            const double c1 = d_add(P.a[1], d_mul(tc, P.b[1]));
            if (dims == 3) {
                const double c2 = d_add(P.a[2], d_mul(tc, P.b[2]));
                ds = norm3(d_sub(x, c0), d_sub(y, c1), d_sub(z, c2));
            } else {
                const double e0 = d_sub(x, c0), e1 = d_sub(y, c1);
                ds = __dsqrt_rn(d_add(d_mul(e0, e0), d_mul(e1, e1)));
            }
        }
        best = dmin(best, ds);
    }
    return d_sub(best, radius);
}

template <bool MARKED = false>
__device__ double eval_sdf(const sf_sdf_node* __restrict__ prog, int n, double x, double y,
                           double z, int* err, unsigned long long skip = 0) {
    double ds[VX_DSTACK];
    double px[VX_PSTACK], py[VX_PSTACK], pz[VX_PSTACK];
    int dtop = 0, ptop = 0;
    px[0] = x;
    py[0] = y;
    pz[0] = z;
    for (int q = 0; q < n; ++q) {
        const sf_sdf_node& N = prog[q];
        const double X = px[ptop], Y = py[ptop], Z = pz[ptop];
        switch (N.op) {
            case 1: {  // BOX
                const double q0 = d_sub(fabs(d_sub(X, N.a[0])), d_mul(N.b[0], 0.5));
                const double q1 = d_sub(fabs(d_sub(Y, N.a[1])), d_mul(N.b[1], 0.5));
                const double q2 = d_sub(fabs(d_sub(Z, N.a[2])), d_mul(N.b[2], 0.5));
                const double out = norm3(dmax(q0, 0.0), dmax(q1, 0.0), dmax(q2, 0.0));
                const double ins = dmin(fmax(fmax(q0, q1), q2), 0.0);
                if (dtop >= VX_DSTACK) { *err = 1; return 1.0; }
                ds[dtop++] = d_add(out, ins);
                break;
            }
            case 2: {  // SPHERE
                if (dtop >= VX_DSTACK) { *err = 1; return 1.0; }
                ds[dtop++] = d_sub(norm3(d_sub(X, N.a[0]), d_sub(Y, N.a[1]), d_sub(Z, N.a[2])), N.s0);
                break;
            }
            case 3: {  // CYLINDER: a = p1, b = unit axis, s0 = length, s1 = radius
                const double v0 = d_sub(X, N.a[0]), v1 = d_sub(Y, N.a[1]), v2 = d_sub(Z, N.a[2]);
                const double t = d_add(d_add(d_mul(v0, N.b[0]), d_mul(v1, N.b[1])), d_mul(v2, N.b[2]));
                const double L = N.s0;
                const double tc = dmin(dmax(t, 0.0), L);
                const double c0 = d_add(N.a[0], d_mul(tc, N.b[0]));
                const double c1 = d_add(N.a[1], d_mul(tc, N.b[1]));
                const double c2 = d_add(N.a[2], d_mul(tc, N.b[2]));
                const double radial = norm3(d_sub(X, c0), d_sub(Y, c1), d_sub(Z, c2));
                const double half = d_mul(L, 0.5);
                const double axial = dmax(0.0, d_sub(fabs(d_sub(t, half)), half));
                const bool inside = (t >= 0.0) && (t <= L);
                const double rr = d_sub(radial, N.s1);
                if (dtop >= VX_DSTACK) { *err = 1; return 1.0; }
                ds[dtop++] = inside ? rr : __dsqrt_rn(d_add(d_mul(rr, rr), d_mul(axial, axial)));
                break;
            }
            case 4: {  // CONE: a = p1, b = unit axis, s0 = length, s1 = r1; next node a[0] = r2 - r1
                if (q + 1 >= n || prog[q + 1].op != 27) { *err = 4; return 1.0; }
                const double dr = prog[q + 1].a[0];
                ++q;
                const double v0 = d_sub(X, N.a[0]), v1 = d_sub(Y, N.a[1]), v2 = d_sub(Z, N.a[2]);
                const double L = N.s0;
                const double t = __ddiv_rn(
                    d_add(d_add(d_mul(v0, N.b[0]), d_mul(v1, N.b[1])), d_mul(v2, N.b[2])), L);
                const double tc = clip01(t);
                const double rt = d_add(N.s1, d_mul(tc, dr));
                const double tl = d_mul(tc, L);
                const double c0 = d_add(N.a[0], d_mul(tl, N.b[0]));
                const double c1 = d_add(N.a[1], d_mul(tl, N.b[1]));
                const double c2 = d_add(N.a[2], d_mul(tl, N.b[2]));
                const double radial = norm3(d_sub(X, c0), d_sub(Y, c1), d_sub(Z, c2));
                const double axial = d_mul(dmax(0.0, d_sub(fabs(d_sub(t, 0.5)), 0.5)), L);
                const bool inside = (t >= 0.0) && (t <= 1.0);
                const double rr = d_sub(radial, rt);
                if (dtop >= VX_DSTACK) { *err = 1; return 1.0; }
                ds[dtop++] = inside ? rr : __dsqrt_rn(d_add(d_mul(rr, rr), d_mul(axial, axial)));
                break;
            }
            case 5: {  // HORN: a = throat, b = unit axis, s0 = length, s1 = throat radius,
                       // n = profile; next node a[0] = m, alpha, alpha or R
                if (q + 1 >= n || prog[q + 1].op != 27) { *err = 4; return 1.0; }
                const double k = prog[q + 1].a[0];
                ++q;
                const double v0 = d_sub(X, N.a[0]), v1 = d_sub(Y, N.a[1]), v2 = d_sub(Z, N.a[2]);
                const double L = N.s0;
                const double t = d_add(d_add(d_mul(v0, N.b[0]), d_mul(v1, N.b[1])), d_mul(v2, N.b[2]));
                const double tc = clip01(__ddiv_rn(t, L));
                const double r = norm3(d_sub(v0, d_mul(t, N.b[0])), d_sub(v1, d_mul(t, N.b[1])),
                                       d_sub(v2, d_mul(t, N.b[2])));
                const double xa = d_mul(tc, L);
                double hr;
                if (N.n == 0) hr = d_mul(N.s1, d_add(1.0, d_mul(k, tc)));  // conical
                else if (N.n == 1) hr = d_mul(N.s1, exp(d_mul(k, xa)));   // exponential
                else if (N.n == 2) hr = d_mul(N.s1, cosh(d_mul(k, xa)));  // hyperbolic
                else {                                                     // tractrix
                    const double c = cos(__ddiv_rn(xa, k));
                    hr = __ddiv_rn(N.s1, d_mul(c, c));
                }
                const double rd = d_sub(r, hr);
                const double cap = dmax(-t, d_sub(t, L));
                const bool inside = (t >= 0.0) && (t <= L);
                if (dtop >= VX_DSTACK) { *err = 1; return 1.0; }
                ds[dtop++] = inside ? rd : __dsqrt_rn(d_add(d_mul(rd, rd), d_mul(cap, cap)));
                break;
            }
            case 6:    // TUBE along a 3-D path: n vertices in the next n nodes
            case 7: {  // SPIRAL: the same in the xy plane, extruded over 0 <= z <= s0
                if (N.n < 2 || q + N.n >= n) { *err = 4; return 1.0; }
                const double rd = path_distance(prog + q + 1, N.n, N.op == 6 ? 3 : 2, X, Y, Z);
                double d = rd;
                if (N.op == 7) {
                    const double zd = dmax(0.0, dmax(-Z, d_sub(Z, N.s0)));
                    const bool inside = (Z >= 0.0) && (Z <= N.s0);
                    d = inside ? rd : __dsqrt_rn(d_add(d_mul(rd, rd), d_mul(zd, zd)));
                }
                q += N.n;
                if (dtop >= VX_DSTACK) { *err = 1; return 1.0; }
                ds[dtop++] = d;
                break;
            }
            case 13:    // SMOOTH_UNION: pop b, a; s0 = blend radius
            case 14:    // SMOOTH_INTERSECTION
            case 15: {  // SMOOTH_DIFFERENCE (the subtracted shape negated)
                if (dtop < 2) { *err = 2; return 1.0; }
                const double d1 = ds[dtop - 2];
                const double d2 = (N.op == 15) ? -ds[dtop - 1] : ds[dtop - 1];
                const double k = N.s0;
                const double h = clip01(d_add(0.5, __ddiv_rn(d_mul(0.5, d_sub(d2, d1)), k)));
                const double mix = d_add(d_mul(d2, d_sub(1.0, h)), d_mul(d1, h));
                const double bump = d_mul(d_mul(k, h), d_sub(1.0, h));
                dtop -= 2;
                ds[dtop++] = (N.op == 13) ? d_sub(mix, bump) : d_add(mix, bump);
                break;
            }
            case 10:    // UNION n
            case 11: {  // INTERSECTION n
                if (N.n == 0) {
                    if (dtop >= VX_DSTACK) { *err = 1; return 1.0; }
                    ds[dtop++] = (N.op == 10) ? __longlong_as_double(0x7ff0000000000000LL)
                                              : __longlong_as_double((long long)0xfff0000000000000ULL);
                    break;
                }
                if (N.n > dtop) { *err = 2; return 1.0; }
                const int base = dtop - N.n;
                double r = ds[base];
                for (int c = 1; c < N.n; ++c) r = (N.op == 10) ? dmin(r, ds[base + c]) : dmax(r, ds[base + c]);
                dtop = base;
                ds[dtop++] = r;
                break;
            }
            case 12: {  // DIFFERENCE n: base, then subtracted
                if (N.n > dtop || N.n < 1) { *err = 2; return 1.0; }
                const int base = dtop - N.n;
                double r = ds[base];
                for (int c = 1; c < N.n; ++c) r = dmax(r, -ds[base + c]);
                dtop = base;
                ds[dtop++] = r;
                break;
            }
            case 20:    // PUSH_TRANSLATE
            case 21: {  // PUSH_SCALE
                if (ptop + 1 >= VX_PSTACK) { *err = 3; return 1.0; }
                ++ptop;
                if (N.op == 20) {
                    px[ptop] = d_sub(X, N.a[0]);
                    py[ptop] = d_sub(Y, N.a[1]);
                    pz[ptop] = d_sub(Z, N.a[2]);
                } else {
                    px[ptop] = __ddiv_rn(X, N.a[0]);
                    py[ptop] = __ddiv_rn(Y, N.a[1]);
                    pz[ptop] = __ddiv_rn(Z, N.a[2]);
                }
                break;
            }
            case 25: {  // PUSH_ROTATE: rows 0, 1 here (a, b), row 2 in the next node's a
                if (ptop + 1 >= VX_PSTACK || q + 1 >= n || prog[q + 1].op != 26) { *err = 3; return 1.0; }
                const sf_sdf_node& N2 = prog[q + 1];
                ++ptop;
                px[ptop] = d_add(d_add(d_mul(X, N.a[0]), d_mul(Y, N.a[1])), d_mul(Z, N.a[2]));
                py[ptop] = d_add(d_add(d_mul(X, N.b[0]), d_mul(Y, N.b[1])), d_mul(Z, N.b[2]));
                pz[ptop] = d_add(d_add(d_mul(X, N2.a[0]), d_mul(Y, N2.a[1])), d_mul(Z, N2.a[2]));
                ++q;  // the row-2 node is consumed
                break;
            }
            case 22:
                if (ptop == 0) { *err = 3; return 1.0; }
                --ptop;
                break;
            case 23:
                if (dtop < 1) { *err = 2; return 1.0; }
                ds[dtop - 1] = d_mul(ds[dtop - 1], N.s0);
                break;
            case 24:
                if (dtop < 1) { *err = 2; return 1.0; }
                ds[dtop - 1] = -ds[dtop - 1];
                break;
            default:
                if (MARKED && N.op == kSkip) {
                    if (skip >> (int)N.a[0] & 1) {
                        ds[dtop++] = N.s0;
                        q += N.n;
                    }
                    break;
                }
                *err = 4;
                return 1.0;
        }
    }
    if (dtop != 1) { *err = 2; return 1.0; }
    return ds[0];
}

// ---- FP32 intervals ---------------------------------------------------------

// A node's constants as intervals: the floats at or below / at or above each
// double (rounded on the host).  A marker has its bit, and a union, intersection
// or difference its first child's bit (-1: not marked), in a[0].x as an integer.
struct IvNode {
    int op, n;
    float2 a[3], b[3], s0, s1;
};

// min / max that keep a NaN (a NaN bound must never decide a cell)
__device__ __forceinline__ float nmin(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float nmax(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// Intervals as (lo, hi).  Each function encloses its FP64 counterpart's
// rounded result for operands inside the intervals.
__device__ __forceinline__ float2 iv(float lo, float hi) { return make_float2(lo, hi); }
// decides nothing: NaN bounds stay NaN through every operation
__device__ __forceinline__ float2 iv_unknown() {
    return iv(__int_as_float(0x7fc00000), __int_as_float(0x7fc00000));
}
__device__ __forceinline__ float2 iv_add(float2 a, float2 b) {
    return iv(__fadd_rd(a.x, b.x), __fadd_ru(a.y, b.y));
}
__device__ __forceinline__ float2 iv_sub(float2 a, float2 b) {
    return iv(__fsub_rd(a.x, b.y), __fsub_ru(a.y, b.x));
}
__device__ __forceinline__ float2 iv_neg(float2 a) { return iv(-a.y, -a.x); }
__device__ __forceinline__ float2 iv_min(float2 a, float2 b) {
    return iv(nmin(a.x, b.x), nmin(a.y, b.y));
}
__device__ __forceinline__ float2 iv_max(float2 a, float2 b) {
    return iv(nmax(a.x, b.x), nmax(a.y, b.y));
}
__device__ __forceinline__ float2 iv_hull(float2 a, float2 b) {
    return iv(nmin(a.x, b.x), nmax(a.y, b.y));
}
__device__ __forceinline__ float2 iv_mul(float2 a, float2 b) {
    const float lo = nmin(nmin(__fmul_rd(a.x, b.x), __fmul_rd(a.x, b.y)),
                          nmin(__fmul_rd(a.y, b.x), __fmul_rd(a.y, b.y)));
    const float hi = nmax(nmax(__fmul_ru(a.x, b.x), __fmul_ru(a.x, b.y)),
                          nmax(__fmul_ru(a.y, b.x), __fmul_ru(a.y, b.y)));
    return iv(lo, hi);
}
__device__ __forceinline__ float2 iv_abs(float2 a) {
    const float lo = a.x >= 0.0f ? a.x : (a.y <= 0.0f ? -a.y : (a.x < 0.0f && a.y > 0.0f ? 0.0f : a.x));
    return iv(lo, nmax(fabsf(a.x), fabsf(a.y)));
}
__device__ __forceinline__ float2 iv_sq(float2 a) {
    const float2 m = iv_abs(a);
    return iv(__fmul_rd(m.x, m.x), __fmul_ru(m.y, m.y));
}
__device__ __forceinline__ float2 iv_sqrt(float2 a) {  // of a sum of squares
    return iv(__fsqrt_rd(a.x), __fsqrt_ru(a.y));
}
__device__ __forceinline__ float2 iv_div(float2 a, float2 b) {
    if (!(b.x > 0.0f || b.y < 0.0f)) return iv_unknown();
    const float lo = nmin(nmin(__fdiv_rd(a.x, b.x), __fdiv_rd(a.x, b.y)),
                          nmin(__fdiv_rd(a.y, b.x), __fdiv_rd(a.y, b.y)));
    const float hi = nmax(nmax(__fdiv_ru(a.x, b.x), __fdiv_ru(a.x, b.y)),
                          nmax(__fdiv_ru(a.y, b.x), __fdiv_ru(a.y, b.y)));
    return iv(lo, hi);
}
__device__ __forceinline__ float2 iv_clip01(float2 t) {
    return iv(nmin(nmax(t.x, 0.0f), 1.0f), nmin(nmax(t.y, 0.0f), 1.0f));
}
__device__ __forceinline__ float2 iv_norm3(float2 a, float2 b, float2 c) {
    return iv_sqrt(iv_add(iv_add(iv_sq(a), iv_sq(b)), iv_sq(c)));
}
__device__ __forceinline__ float2 iv_dot3(const float2 v[3], const float2 b[3]) {
    return iv_add(iv_add(iv_mul(v[0], b[0]), iv_mul(v[1], b[1])), iv_mul(v[2], b[2]));
}
__device__ __forceinline__ float2 iv_pos(float2 a) { return iv(nmax(a.x, 0.0f), nmax(a.y, 0.0f)); }
// `in` where 0 <= t <= hi surely, the capped distance where surely not, else both
__device__ __forceinline__ float2 iv_capped(float2 t, float2 hi, float2 in, float2 over) {
    const float2 cap = iv_sqrt(iv_add(iv_sq(in), iv_sq(over)));
    if (t.x >= 0.0f && t.y <= hi.x) return in;
    if (t.y < 0.0f || t.x > hi.y) return cap;
    return iv_hull(in, cap);
}
// A monotonic function's float bounds widened past its error (a few ulp, and
// 1e-37 for results that underflow; an infinite lower bound becomes NaN)
__device__ __forceinline__ float2 iv_widen(float lo, float hi) {
    return iv(__fsub_rd(lo, __fadd_ru(__fmul_ru(fabsf(lo), 1e-5f), 1e-37f)),
              __fadd_ru(hi, __fadd_ru(__fmul_ru(fabsf(hi), 1e-5f), 1e-37f)));
}
// What an interval says of every distance in it: 1 inside, 0 outside, -1 neither
__device__ __forceinline__ int iv_side(float2 d) {
    if (!(d.x <= d.y)) return -1;  // NaN
    return d.y <= 0.0f ? 1 : (d.x > 0.0f ? 0 : -1);
}

// path_distance over the box (X, Y, Z): the radius is the hull of the radii
// of every vertex that could be the nearest one.
__device__ float2 iv_path_distance(const IvNode* __restrict__ d, int m, int dims, float2 X,
                                   float2 Y, float2 Z) {
    const float inf = __int_as_float(0x7f800000);
    float2 best = iv(inf, inf), radius = iv(0.0f, 0.0f);
    float near = inf;
    bool any = false;
    for (int q = 0; q < m; ++q) {
        const IvNode& P = d[q];
        const float2 w0 = iv_sub(X, P.a[0]), w1 = iv_sub(Y, P.a[1]);
        const float2 w2 = dims == 3 ? iv_sub(Z, P.a[2]) : iv(0.0f, 0.0f);
        const float2 dv = iv_norm3(w0, w1, w2);  // adding an exact zero changes nothing
        if (!(dv.x > near)) {
            radius = any ? iv_hull(radius, P.s0) : P.s0;
            any = true;
        }
        near = nmin(near, dv.y);
        if (q + 1 == m) break;
        float2 ds = dv;  // a degenerate segment (squared length below 1e-14) is its first vertex
        if (!(P.s1.y < 0.9e-14f)) {
            float2 t = iv_add(iv_mul(w0, P.b[0]), iv_mul(w1, P.b[1]));
            if (dims == 3) t = iv_add(t, iv_mul(w2, P.b[2]));
            const float2 tc = iv_clip01(iv_div(t, P.s1));
            const float2 e0 = iv_sub(X, iv_add(P.a[0], iv_mul(tc, P.b[0])));
            const float2 e1 = iv_sub(Y, iv_add(P.a[1], iv_mul(tc, P.b[1])));
            const float2 e2 =
                dims == 3 ? iv_sub(Z, iv_add(P.a[2], iv_mul(tc, P.b[2]))) : iv(0.0f, 0.0f);
            ds = iv_norm3(e0, e1, e2);
            if (!(P.s1.x > 1.1e-14f)) ds = iv_hull(ds, dv);
        }
        best = iv_min(best, ds);
    }
    return iv_sub(best, radius);
}

// eval_sdf over a box, operation for operation.  The program has passed
// check_program, so the stacks need no checks here.  Children whose bit is set in
// `skip` are passed over: their markers push a value that cannot win.  RECORD
// sets in *lost the bits of the children that lose to another everywhere in the
// box: whatever box inside it is looked at next, the result does not depend on
// them.  (A NaN bound loses to nothing and nothing loses to it.)
template <bool RECORD>
__device__ float2 eval_iv(const IvNode* __restrict__ prog, int n, float2 x, float2 y, float2 z,
                          unsigned long long skip, unsigned long long* lost) {
    float2 ds[VX_DSTACK];
    float2 px[VX_PSTACK], py[VX_PSTACK], pz[VX_PSTACK];
    int dtop = 0, ptop = 0;
    px[0] = x;
    py[0] = y;
    pz[0] = z;
    const float2 one = iv(1.0f, 1.0f), half1 = iv(0.5f, 0.5f);
    for (int q = 0; q < n; ++q) {
        const IvNode& N = prog[q];
        const float2 X = px[ptop], Y = py[ptop], Z = pz[ptop];
        switch (N.op) {
            case 1: {
                const float2 q0 = iv_sub(iv_abs(iv_sub(X, N.a[0])), iv_mul(N.b[0], half1));
                const float2 q1 = iv_sub(iv_abs(iv_sub(Y, N.a[1])), iv_mul(N.b[1], half1));
                const float2 q2 = iv_sub(iv_abs(iv_sub(Z, N.a[2])), iv_mul(N.b[2], half1));
                const float2 out = iv_norm3(iv_pos(q0), iv_pos(q1), iv_pos(q2));
                const float2 m = iv_max(iv_max(q0, q1), q2);
                ds[dtop++] = iv_add(out, iv(nmin(m.x, 0.0f), nmin(m.y, 0.0f)));
                break;
            }
            case 2:
                ds[dtop++] = iv_sub(iv_norm3(iv_sub(X, N.a[0]), iv_sub(Y, N.a[1]), iv_sub(Z, N.a[2])),
                                    N.s0);
                break;
            case 3: {
                const float2 v[3] = {iv_sub(X, N.a[0]), iv_sub(Y, N.a[1]), iv_sub(Z, N.a[2])};
                const float2 t = iv_dot3(v, N.b);
                const float2 L = N.s0, tc = iv_min(iv_pos(t), L);
                const float2 radial = iv_norm3(iv_sub(X, iv_add(N.a[0], iv_mul(tc, N.b[0]))),
                                               iv_sub(Y, iv_add(N.a[1], iv_mul(tc, N.b[1]))),
                                               iv_sub(Z, iv_add(N.a[2], iv_mul(tc, N.b[2]))));
                const float2 half = iv_mul(L, half1);
                const float2 axial = iv_pos(iv_sub(iv_abs(iv_sub(t, half)), half));
                ds[dtop++] = iv_capped(t, L, iv_sub(radial, N.s1), axial);
                break;
            }
            case 4: {
                const float2 dr = prog[q + 1].a[0];
                ++q;
                const float2 v[3] = {iv_sub(X, N.a[0]), iv_sub(Y, N.a[1]), iv_sub(Z, N.a[2])};
                const float2 L = N.s0, t = iv_div(iv_dot3(v, N.b), L), tc = iv_clip01(t);
                const float2 rt = iv_add(N.s1, iv_mul(tc, dr)), tl = iv_mul(tc, L);
                const float2 radial = iv_norm3(iv_sub(X, iv_add(N.a[0], iv_mul(tl, N.b[0]))),
                                               iv_sub(Y, iv_add(N.a[1], iv_mul(tl, N.b[1]))),
                                               iv_sub(Z, iv_add(N.a[2], iv_mul(tl, N.b[2]))));
                const float2 axial = iv_mul(iv_pos(iv_sub(iv_abs(iv_sub(t, half1)), half1)), L);
                ds[dtop++] = iv_capped(t, one, iv_sub(radial, rt), axial);
                break;
            }
            case 5: {
                const float2 k = prog[q + 1].a[0];
                ++q;
                const float2 v[3] = {iv_sub(X, N.a[0]), iv_sub(Y, N.a[1]), iv_sub(Z, N.a[2])};
                const float2 L = N.s0, t = iv_dot3(v, N.b), tc = iv_clip01(iv_div(t, L));
                const float2 r = iv_norm3(iv_sub(v[0], iv_mul(t, N.b[0])), iv_sub(v[1], iv_mul(t, N.b[1])),
                                          iv_sub(v[2], iv_mul(t, N.b[2])));
                const float2 xa = iv_mul(tc, L);
                float2 hr;
                if (N.n == 0) hr = iv_mul(N.s1, iv_add(one, iv_mul(k, tc)));
                else if (N.n == 1) {
                    const float2 e = iv_mul(k, xa);
                    hr = iv_mul(N.s1, iv_widen(expf(e.x), expf(e.y)));
                } else if (N.n == 2) {
                    const float2 e = iv_abs(iv_mul(k, xa));
                    hr = iv_mul(N.s1, iv_widen(coshf(e.x), coshf(e.y)));
                } else {  // cos falls on [0, pi]; wider arguments decide nothing
                    const float2 e = iv_div(xa, k);
                    if (e.x >= 0.0f && e.y <= 3.1f) {
                        const float2 c = iv(__fsub_rd(cosf(e.y), 1e-6f), __fadd_ru(cosf(e.x), 1e-6f));
                        hr = iv_div(N.s1, iv_sq(c));
                    } else {
                        hr = iv_unknown();
                    }
                }
                ds[dtop++] = iv_capped(t, L, iv_sub(r, hr), iv_max(iv_neg(t), iv_sub(t, L)));
                break;
            }
            case 6:
            case 7: {
                const float2 rd = iv_path_distance(prog + q + 1, N.n, N.op == 6 ? 3 : 2, X, Y, Z);
                float2 d = rd;
                if (N.op == 7)
                    d = iv_capped(Z, N.s0, rd, iv_pos(iv_max(iv_neg(Z), iv_sub(Z, N.s0))));
                q += N.n;
                ds[dtop++] = d;
                break;
            }
            case 13:
            case 14:
            case 15: {
                const float2 d1 = ds[dtop - 2];
                const float2 d2 = (N.op == 15) ? iv_neg(ds[dtop - 1]) : ds[dtop - 1];
                const float2 k = N.s0;
                const float2 h = iv_clip01(iv_add(half1, iv_div(iv_mul(half1, iv_sub(d2, d1)), k)));
                const float2 g = iv_sub(one, h);
                const float2 mix = iv_add(iv_mul(d2, g), iv_mul(d1, h));
                const float2 bump = iv_mul(iv_mul(k, h), g);
                dtop -= 2;
                ds[dtop++] = (N.op == 13) ? iv_sub(mix, bump) : iv_add(mix, bump);
                break;
            }
            case 10:
            case 11: {
                const float inf = __int_as_float(0x7f800000);
                if (N.n == 0) {
                    ds[dtop++] = (N.op == 10) ? iv(inf, inf) : iv(-inf, -inf);
                    break;
                }
                const int base = dtop - N.n;
                float2 r = ds[base];
                for (int c = 1; c < N.n; ++c)
                    r = (N.op == 10) ? iv_min(r, ds[base + c]) : iv_max(r, ds[base + c]);
                const int bit = __float_as_int(N.a[0].x);
                if (RECORD && bit >= 0)
                    for (int c = 0; c < N.n; ++c)
                        if (N.op == 10 ? ds[base + c].x > r.y : ds[base + c].y < r.x)
                            *lost |= 1ull << (bit + c);
                dtop = base;
                ds[dtop++] = r;
                break;
            }
            case 12: {
                const int base = dtop - N.n;
                float2 r = ds[base];
                for (int c = 1; c < N.n; ++c) r = iv_max(r, iv_neg(ds[base + c]));
                const int bit = __float_as_int(N.a[0].x);
                if (RECORD && bit >= 0)
                    for (int c = 0; c < N.n; ++c)
                        if ((c == 0 ? ds[base].y : -ds[base + c].x) < r.x) *lost |= 1ull << (bit + c);
                dtop = base;
                ds[dtop++] = r;
                break;
            }
            case 20:
                ++ptop;
                px[ptop] = iv_sub(X, N.a[0]);
                py[ptop] = iv_sub(Y, N.a[1]);
                pz[ptop] = iv_sub(Z, N.a[2]);
                break;
            case 21:
                ++ptop;
                px[ptop] = iv_div(X, N.a[0]);
                py[ptop] = iv_div(Y, N.a[1]);
                pz[ptop] = iv_div(Z, N.a[2]);
                break;
            case 25: {
                const float2 P[3] = {X, Y, Z};
                ++ptop;
                px[ptop] = iv_dot3(P, N.a);
                py[ptop] = iv_dot3(P, N.b);
                pz[ptop] = iv_dot3(P, prog[q + 1].a);
                ++q;
                break;
            }
            case 22:
                --ptop;
                break;
            case 23:
                ds[dtop - 1] = iv_mul(ds[dtop - 1], N.s0);
                break;
            case 24:
                ds[dtop - 1] = iv_neg(ds[dtop - 1]);
                break;
            case kSkip:
                if (skip >> __float_as_int(N.a[0].x) & 1) {
                    ds[dtop++] = N.s0;
                    q += N.n;
                }
                break;
        }
    }
    return ds[0];
}

// ---- the mask -----------------------------------------------------------------

struct VxGrid {
    int nx, ny, nz, invert;
    int first, planes;     // the grid's plane that is plane 0 here (a slab), its planes
    double res;
    const double* coords;  // planes + ny + nz cell centres of a nonuniform grid, or null
    float2* axis;          // the same centres as intervals (k_vx_axes)
    unsigned* count;       // queued blocks
    unsigned* queue;
    int si, sj, sk;               // super-blocks of 16 x 16 x 32 cells per axis
    unsigned long long* lost;     // per queue entry, in front of them one per super-block: the
    unsigned char* side;          // parts that do not matter there; per super-block its side + 1
    uint8_t* out;
};

__device__ __forceinline__ double cell_centre(const VxGrid& g, int axis, int i) {
    if (axis == 0) i += g.first;
    if (g.coords) return g.coords[(axis > 0 ? g.planes : 0) + (axis > 1 ? g.ny : 0) + i];
    return d_add(d_mul((double)i, g.res), d_mul(g.res, 0.5));
}

// Cell centres as intervals, and an empty queue.
__global__ void k_vx_axes(VxGrid g) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0) *g.count = 0;
    if (t >= g.nx + g.ny + g.nz) return;
    const int axis = t < g.nx ? 0 : (t < g.nx + g.ny ? 1 : 2);
    const double c = cell_centre(g, axis, t - (axis > 0 ? g.nx : 0) - (axis > 1 ? g.ny : 0));
    g.axis[t] = iv(__double2float_rd(c), __double2float_ru(c));
}

__device__ __forceinline__ float2 axis_hull(const float2* __restrict__ a, int i0, int cells, int n) {
    float2 h = a[i0];
    for (int e = 1; e < cells; ++e)
        if (i0 + e < n) h = iv_hull(h, a[i0 + e]);
    return h;
}

// A program of up to kStaged nodes is read from shared memory: a thread that walks
// it alone otherwise waits for each node in turn (k_vx_super on 900 super-blocks,
// a program of 16 resonators: 69 -> 43 us).
constexpr int kStaged = 256;
__device__ __forceinline__ const IvNode* stage(IvNode* to, const IvNode* __restrict__ prog, int n) {
    if (n > kStaged) return prog;
    float2* d = reinterpret_cast<float2*>(to);
    const float2* f = reinterpret_cast<const float2*>(prog);
    for (int e = threadIdx.x; e < n * (int)(sizeof(IvNode) / sizeof(float2)); e += blockDim.x) d[e] = f[e];
    __syncthreads();
    return to;
}

// One thread per super-block of 16 x 16 x 32 cells: its side, and the parts of the
// program that matter nowhere in it.
__global__ void __launch_bounds__(32) k_vx_super(VxGrid g, const IvNode* __restrict__ program, int n) {
    __shared__ IvNode staged[kStaged];
    const IvNode* prog = stage(staged, program, n);
    const int t = blockIdx.x * 32 + threadIdx.x;
    if (t >= g.si * g.sj * g.sk) return;
    const int k0 = 32 * (t % g.sk), j0 = 16 * (t / g.sk % g.sj), i0 = 16 * (t / g.sk / g.sj);
    unsigned long long lost = 0;
    const float2 d = eval_iv<true>(prog, n, axis_hull(g.axis, i0, 16, g.nx),
                                   axis_hull(g.axis + g.nx, j0, 16, g.ny),
                                   axis_hull(g.axis + g.nx + g.ny, k0, 32, g.nz), 0, &lost);
    g.lost[t] = lost;
    g.side[t] = (unsigned char)(iv_side(d) + 1);
}

// One thread block per super-block, one thread per 4 x 4 x 4 block of cells, with
// k fastest, so that 8 threads write 32 consecutive bytes of a row.  A decided
// block is filled, any other is queued with the parts that do not matter in it.
// Bound by instruction issue of the interval program; the block edge is the
// smallest whose row fits one 32-bit store.  Measured on GB300, whole sf_voxelize
// calls: 400^3 enclosure (4 nodes) 16.3 ms with one FP64 evaluation per cell, 0.154
// with blocks and cells over the whole program, 0.12 now; 180 x 240 x 157 with 16
// resonators 18.2, 0.53 and 0.27 (of which 0.17 is the host's).
__global__ void __launch_bounds__(128) k_vx_blocks(VxGrid g, const IvNode* __restrict__ program, int n, int supers) {
    __shared__ IvNode staged[kStaged];
    const int sb = blockIdx.x, t = threadIdx.x;
    const int k0 = 32 * (sb % g.sk) + 4 * (t & 7), j0 = 16 * (sb / g.sk % g.sj) + 4 * (t >> 3 & 3),
              i0 = 16 * (sb / g.sk / g.sj) + 4 * (t >> 5);
    const bool real = k0 < g.nz && j0 < g.ny && i0 < g.nx;
    int side = supers ? (int)g.side[sb] - 1 : -1;  // (else the super-blocks were not looked at)
    const bool open = side < 0;
    const IvNode* prog = open ? stage(staged, program, n) : program;  // (the whole block is open or not)
    unsigned long long lost = 0;
    if (!real) side = 0;
    if (real && open) {
        const unsigned long long skip = supers ? g.lost[sb] : 0;
        lost = skip;
        side = iv_side(eval_iv<true>(prog, n, axis_hull(g.axis, i0, 4, g.nx),
                                     axis_hull(g.axis + g.nx, j0, 4, g.ny),
                                     axis_hull(g.axis + g.nx + g.ny, k0, 4, g.nz), skip, &lost));
    }
    const int lane = t & 31;
    const unsigned m = __ballot_sync(0xffffffffu, side < 0);
    if (m) {  // one atomic per warp
        unsigned at = 0;
        if (lane == 0) at = atomicAdd(g.count, (unsigned)__popc(m));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1));
        if (side < 0) {
            g.queue[at] = (unsigned)(((long long)(i0 / 4) * ((g.ny + 3) / 4) + j0 / 4) * ((g.nz + 3) / 4) + k0 / 4);
            g.lost[(size_t)g.si * g.sj * g.sk + at] = lost;
        }
    }
    if (!real || side < 0) return;
    const uint8_t v = (uint8_t)((side == 1) != (g.invert != 0));
    const int i1 = min(i0 + 4, g.nx), j1 = min(j0 + 4, g.ny), k1 = min(k0 + 4, g.nz);
    const bool word = g.nz % 4 == 0 && (reinterpret_cast<uintptr_t>(g.out) & 3u) == 0;
    for (int i = i0; i < i1; ++i)
        for (int j = j0; j < j1; ++j) {
            uint8_t* o = g.out + ((long long)i * g.ny + j) * g.nz + k0;
            if (word) *reinterpret_cast<unsigned*>(o) = v * 0x01010101u;
            else
                for (int e = 0; e < k1 - k0; ++e) o[e] = v;
        }
}

// The cell of thread t of the queued blocks.
__device__ __forceinline__ bool queued_cell(const VxGrid& g, unsigned long long t, int& i, int& j, int& k) {
    const int bj_n = (g.ny + 3) / 4, bk_n = (g.nz + 3) / 4;
    const unsigned b = g.queue[t >> 6];
    const int e = (int)(t & 63);
    k = 4 * (int)(b % bk_n) + (e & 3);
    j = 4 * (int)(b / bk_n % bj_n) + (e >> 2 & 3);
    i = 4 * (int)(b / bk_n / bj_n) + (e >> 4);
    return i < g.nx && j < g.ny && k < g.nz;
}

// The queued blocks' cells, one thread each: the cell's own interval, and the
// FP64 evaluation where that straddles zero.  Straddling cells lie in planes (a
// face through cell centres), a few to a warp, and the FP64 pipe takes as long for
// a few lanes as for 32: a thread block collects them and evaluates them side by
// side (180 x 240 x 157 with 32 resonators: 289 -> 243 us; with 16, where the
// interval program bounds it, 30 -> 32).  Both evaluators pass over the parts that
// do not matter in the block: 365 -> 332 us for 16 with the intervals alone, then 47
// with the FP64 program too.
__global__ void __launch_bounds__(128) k_vx_cells(VxGrid g, const IvNode* __restrict__ program,
                                                  const sf_sdf_node* __restrict__ prog, int n) {
    __shared__ IvNode staged[kStaged];
    __shared__ unsigned long long open[256];
    __shared__ int n_open;
    const unsigned long long cells = (unsigned long long)*g.count * 64;
    const unsigned long long* lost = g.lost + (size_t)g.si * g.sj * g.sk;
    if (threadIdx.x == 0) n_open = 0;
    const IvNode* ivp = stage(staged, program, n);
    auto put = [&](int i, int j, int k, bool inside) {
        g.out[((long long)i * g.ny + j) * g.nz + k] = (uint8_t)(inside != (g.invert != 0));
    };
    auto exact = [&](unsigned long long t) {
        int i, j, k, err = 0;  // the program has passed check_program
        queued_cell(g, t, i, j, k);
        put(i, j, k,
            eval_sdf<true>(prog, n, cell_centre(g, 0, i), cell_centre(g, 1, j), cell_centre(g, 2, k), &err,
                           lost[t >> 6]) <= 0.0);
    };
    __syncthreads();
    for (unsigned long long first = (unsigned long long)blockIdx.x * 128; first < cells;
         first += (unsigned long long)gridDim.x * 128) {
        const unsigned long long t = first + threadIdx.x;
        int i, j, k;
        if (t < cells && queued_cell(g, t, i, j, k)) {
            const int side = iv_side(eval_iv<false>(ivp, n, g.axis[i], g.axis[g.nx + j],
                                                    g.axis[g.nx + g.ny + k], lost[t >> 6], nullptr));
            if (side < 0) open[atomicAdd(&n_open, 1)] = t;  // at most 127 + 128
            else put(i, j, k, side == 1);
        }
        __syncthreads();
        const int have = n_open;
        if (have >= 128) exact(open[have - 128 + threadIdx.x]);
        __syncthreads();
        if (have >= 128 && threadIdx.x == 0) n_open = have - 128;
        __syncthreads();
    }
    if ((int)threadIdx.x < n_open) exact(open[threadIdx.x]);
}

// MaterializedGeometry.voxelize_with_materials (geometry/
// material_assignment.py:133-171) in one pass: program 0 (nodes
// off[0]..off[1]-1) is the geometry, inside = air; programs 1..n_regions are
// the material regions in assignment order, region r giving id ids[r-1].  A
// cell's id is that of the last region containing it, within air only, else
// 0 -- the reference's ordered overwrites.  Regions are tried from the last
// down and the first hit wins, which gives the same id with fewer programs
// evaluated.
__global__ void k_voxelize_materials(const sf_sdf_node* __restrict__ prog,
                                     const int* __restrict__ off, const uint8_t* __restrict__ ids,
                                     int n_regions, int nx, int ny, int nz, double res,
                                     const double* __restrict__ coords,
                                     uint8_t* __restrict__ geom, uint8_t* __restrict__ mat,
                                     int* __restrict__ err_flag) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= nz || j >= ny) return;
    double x, y, z;
    if (coords) {
        x = coords[i];
        y = coords[nx + j];
        z = coords[nx + ny + k];
    } else {
        const double half = d_mul(res, 0.5);
        x = d_add(d_mul((double)i, res), half);
        y = d_add(d_mul((double)j, res), half);
        z = d_add(d_mul((double)k, res), half);
    }
    int err = 0;
    const bool air = eval_sdf(prog + off[0], off[1] - off[0], x, y, z, &err) <= 0.0;
    uint8_t m = 0;
    if (air) {
        for (int r = n_regions; r >= 1; --r) {
            if (eval_sdf(prog + off[r], off[r + 1] - off[r], x, y, z, &err) <= 0.0) {
                m = ids[r - 1];
                break;
            }
        }
    }
    if (err) atomicExch(err_flag, err);
    const long long c = ((long long)i * ny + j) * nz + k;
    geom[c] = (uint8_t)air;
    mat[c] = m;
}

__global__ void k_sdf_points(const sf_sdf_node* __restrict__ prog, int n_nodes,
                             const double* __restrict__ pts, long long n, double* __restrict__ out,
                             int* __restrict__ err_flag) {
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n;
         q += (long long)gridDim.x * blockDim.x) {
        int err = 0;
        out[q] = eval_sdf(prog, n_nodes, pts[3 * q], pts[3 * q + 1], pts[3 * q + 2], &err);
        if (err) atomicExch(err_flag, err);
    }
}

}  // namespace

int sf_launch_sdf_points(const sf_sdf_node* prog_dev, int n_nodes, const double* pts, long long n,
                         double* out, int* err_dev, cudaStream_t st) {
    long long blocks = (n + 255) / 256;
    if (blocks > 152 * 32) blocks = 152 * 32;
    if (blocks < 1) blocks = 1;
    k_sdf_points<<<(int)blocks, 256, 0, st>>>(prog_dev, n_nodes, pts, n, out, err_dev);
    return cudaGetLastError() == cudaSuccess ? 0 : sf_fail("k_sdf_points launch failed");
}

namespace {

// The stack checks eval_sdf makes, which depend on the program alone.
bool check_program(const sf_sdf_node* prog, int n) {
    int dtop = 0, ptop = 0;
    for (int q = 0; q < n; ++q) {
        const sf_sdf_node& N = prog[q];
        switch (N.op) {
            case 4:
            case 5:
                if (q + 1 >= n || prog[q + 1].op != 27) return false;
                ++q;  // fall through
            case 1:
            case 2:
            case 3:
                if (dtop >= VX_DSTACK) return false;
                ++dtop;
                break;
            case 6:
            case 7:
                if (N.n < 2 || N.n >= n - q || dtop >= VX_DSTACK) return false;
                q += N.n;
                ++dtop;
                break;
            case 13:
            case 14:
            case 15:
                if (dtop < 2) return false;
                --dtop;
                break;
            case 10:
            case 11:
                if (N.n == 0) {
                    if (dtop >= VX_DSTACK) return false;
                    ++dtop;
                    break;
                }
                if (N.n < 0 || N.n > dtop) return false;
                dtop -= N.n - 1;
                break;
            case 12:
                if (N.n > dtop || N.n < 1) return false;
                dtop -= N.n - 1;
                break;
            case 20:
            case 21:
                if (ptop + 1 >= VX_PSTACK) return false;
                ++ptop;
                break;
            case 25:
                if (ptop + 1 >= VX_PSTACK || q + 1 >= n || prog[q + 1].op != 26) return false;
                ++ptop;
                ++q;
                break;
            case 22:
                if (ptop == 0) return false;
                --ptop;
                break;
            case 23:
            case 24:
                if (dtop < 1) return false;
                break;
            default:
                return false;
        }
    }
    return dtop == 1;
}

// The floats around a double (rounding toward zero or away does not matter:
// the neighbours are checked).
float2 bounds_of(double v) {
    const float f = (float)v;
    float2 r = make_float2(f, f);
    if ((double)f > v) r.x = std::nextafterf(f, -INFINITY);
    if ((double)f < v) r.y = std::nextafterf(f, INFINITY);
    return r;
}

IvNode interval_node(const sf_sdf_node& N) {
    IvNode v;
    v.op = N.op;
    v.n = N.n;
    for (int e = 0; e < 3; ++e) {
        v.a[e] = bounds_of(N.a[e]);
        v.b[e] = bounds_of(N.b[e]);
    }
    v.s0 = bounds_of(N.s0);
    v.s1 = bounds_of(N.s1);
    return v;
}

// A checked program with a skip marker before each child of its unions,
// intersections and differences: the outer ones first, up to kMaxParts children
// (an operation whose children do not fit has none).  first_bit[q] is the bit of
// the marker at node q of the result, or of the first child of the operation there,
// or -1.  A child is the run of nodes that leaves its value, from the transforms it
// opens with to the last of those it closes with; where a transform encloses
// anything but one value made inside it, no child of the program is marked.
std::vector<sf_sdf_node> mark_program(const sf_sdf_node* nodes, int n, std::vector<int>& first_bit) {
    struct Child {
        int op, index, start, end;  // its operation's node, its place there, its nodes
    };
    struct Open {
        int node;
        size_t values;
    };
    std::vector<Child> children;
    std::vector<int> value;  // first node of each value on the stack
    std::vector<Open> open;
    auto inside = [&] { return open.empty() ? 0 : open.back().values; };  // values below the transform
    bool clean = true;
    for (int q = 0; q < n; ++q) {
        const sf_sdf_node& N = nodes[q];
        const int at = q;
        switch (N.op) {
            case 4: case 5: ++q; value.push_back(at); break;
            case 6: case 7: q += N.n; value.push_back(at); break;
            case 13: case 14: case 15:
                value.pop_back();
                clean = clean && value.size() > inside();
                break;
            case 10: case 11: case 12: {
                if (N.n == 0) {
                    value.push_back(at);
                    break;
                }
                const size_t base = value.size() - N.n;
                clean = clean && base >= inside();
                for (int c = 0; c < N.n; ++c)
                    children.push_back({at, c, value[base + c], c + 1 < N.n ? value[base + c + 1] : at});
                value.resize(base + 1);
                break;
            }
            case 20: case 21: open.push_back({at, value.size()}); break;
            case 25: ++q; open.push_back({at, value.size()}); break;
            case 22:
                if (value.size() == open.back().values + 1) value.back() = open.back().node;
                else clean = false;
                open.pop_back();
                break;
            case 23: case 24: clean = clean && value.size() > inside(); break;
            default: value.push_back(at); break;  // 1, 2, 3
        }
    }
    std::vector<int> bit(n, -1), last(n, -1), before(children.size(), -1);
    int used = 0;
    for (size_t c = children.size(); clean && c-- > 0;) {  // an outer operation stands after its children's
        const int op = children[c].op, k = nodes[op].n;
        if (children[c].index != 0 || k < 2 || used + k > kMaxParts) continue;
        bit[op] = used;
        used += k;
    }
    for (size_t c = 0; c < children.size(); ++c) {  // children by first node, the outermost first
        before[c] = last[children[c].start];
        last[children[c].start] = (int)c;
    }
    std::vector<sf_sdf_node> out;
    first_bit.clear();
    auto put = [&](const sf_sdf_node& N, int b) {
        out.push_back(N);
        first_bit.push_back(b);
    };
    std::vector<int> place(n + 1);
    std::vector<std::pair<int, int>> jumps;  // marker, the node it passes over to
    for (int q = 0; q < n; ++q) {
        place[q] = (int)out.size();
        for (int c = last[q]; c >= 0; c = before[c]) {
            const Child& C = children[c];
            if (bit[C.op] < 0) continue;
            sf_sdf_node m{};
            const int op = nodes[C.op].op;
            const bool high = op == 10 || (op == 12 && C.index > 0);  // what never wins there
            m.op = kSkip;
            m.a[0] = bit[C.op] + C.index;
            m.s0 = high ? INFINITY : -INFINITY;
            jumps.push_back({(int)out.size(), C.end});
            put(m, bit[C.op] + C.index);
        }
        const int op = nodes[q].op;
        put(nodes[q], bit[q]);
        const int data = op == 4 || op == 5 || op == 25 ? 1 : (op == 6 || op == 7 ? nodes[q].n : 0);
        for (int e = 0; e < data; ++e) put(nodes[++q], -1);
    }
    for (const auto& j : jumps) out[j.first].n = place[j.second] - j.first - 1;
    return out;
}

// Device memory of a voxelisation, kept between calls (one block per device
// of at most kKeepBytes, lent to one call at a time; released with the
// deferred frees): a call's allocation took longer than its kernels.  Grids that
// need more are done in slabs of planes.
constexpr size_t kKeepBytes = size_t(72) << 20;  // 500^3 cells: 25 MB
constexpr int kKeepDevices = 64;
struct Kept {
    char* p = nullptr;
    size_t bytes = 0;
    bool lent = false;
};
std::mutex g_keep_mu;
Kept g_keep[kKeepDevices];

class Scratch {
  public:
    char* p = nullptr;
    bool idle = true;  // nothing queued uses it
    int take(size_t bytes, cudaStream_t st) {
        st_ = st;
        cudaGetDevice(&dev_);
        if (bytes <= kKeepBytes && dev_ >= 0 && dev_ < kKeepDevices) {
            std::lock_guard<std::mutex> lock(g_keep_mu);
            Kept& k = g_keep[dev_];
            if (!k.lent) {
                if (k.bytes < bytes) {  // at least doubled; the old one is queued for release
                    size_t grown = 2 * k.bytes < (size_t(1) << 20) ? size_t(1) << 20 : 2 * k.bytes;
                    if (grown < bytes) grown = bytes;
                    if (grown > kKeepBytes) grown = kKeepBytes;
                    sf_defer_free(k.p, k.bytes);
                    k = Kept{};
                    if (cudaMalloc(&k.p, grown) == cudaSuccess) k.bytes = grown;
                    else (void)cudaGetLastError();
                }
                if (k.bytes >= bytes) {
                    k.lent = kept_ = true;
                    p = k.p;
                    return 0;
                }
            }
        }
        if (const cudaError_t e = cudaMallocAsync(reinterpret_cast<void**>(&p), bytes, st)) {
            p = nullptr;
            (void)cudaGetLastError();
            return sf_fail_cuda(e, "sf_voxelize: scratch memory", __FILE__, __LINE__);
        }
        return 0;
    }
    ~Scratch() {
        if (kept_) {
            if (!idle) (void)cudaStreamSynchronize(st_);  // a call that failed on its way
            std::lock_guard<std::mutex> lock(g_keep_mu);
            g_keep[dev_].lent = false;
        } else if (p) {
            cudaFreeAsync(p, st_);
        }
    }

  private:
    cudaStream_t st_ = nullptr;
    int dev_ = 0;
    bool kept_ = false;
};

size_t up16(size_t b) { return (b + 15) / 16 * 16; }

}  // namespace

void sf_voxel_release_kept() {
    std::lock_guard<std::mutex> lock(g_keep_mu);
    int prev = -1;
    cudaGetDevice(&prev);
    for (int d = 0; d < kKeepDevices; ++d) {
        if (!g_keep[d].p || g_keep[d].lent) continue;
        if (d != prev) cudaSetDevice(d);
        cudaFree(g_keep[d].p);
        if (d != prev) cudaSetDevice(prev);
        g_keep[d] = Kept{};
    }
}

// The mask of a program over a grid (coords: the cell centres per axis of a
// nonuniform grid, or null), complete when the call returns.
int sf_launch_voxelize(const sf_sdf_node* nodes, int n_nodes, int nx, int ny, int nz, double res,
                       const double* const* coords, int invert, uint8_t* out, cudaStream_t st) {
    if (!check_program(nodes, n_nodes))
        return sf_fail("sf_voxelize: malformed SDF program (stack error)");
    const int sj = (ny + 15) / 16, sk = (nz + 31) / 32;
    std::vector<int> first_bit;
    const std::vector<sf_sdf_node> marked = mark_program(nodes, n_nodes, first_bit);
    const int n_marked = (int)marked.size();
    const size_t n_axis = (size_t)nx + ny + nz;
    const size_t off_iv = up16(sizeof(sf_sdf_node) * n_marked);
    const size_t off_co = off_iv + up16(sizeof(IvNode) * n_marked);
    const size_t sent = off_co + (coords ? up16(sizeof(double) * n_axis) : 0);
    // Large grids are done in slabs of planes, so that the scratch memory (12 bytes a
    // block) stays within what is kept; a device with less room gets smaller slabs.
    struct Slab {
        long long supers, blocks;
        size_t ax, ct, sd, l, q, end;
    };
    auto slab_of = [&](int planes) {
        Slab b;
        b.supers = (long long)((planes + 15) / 16) * sj * sk;
        b.blocks = (long long)((planes + 3) / 4) * ((ny + 3) / 4) * ((nz + 3) / 4);
        b.ax = sent;
        b.ct = b.ax + up16(sizeof(float2) * n_axis);
        b.sd = b.ct + 16;
        b.l = b.sd + up16((size_t)b.supers);
        b.q = b.l + 8 * (size_t)(b.supers + b.blocks);
        b.end = b.q + sizeof(unsigned) * (size_t)b.blocks;
        return b;
    };
    auto half = [](int planes) {  // in whole blocks, from 32 planes on in whole super-blocks
        const int h = (planes + 1) / 2, unit = h > 16 ? 16 : 4;
        return (h + unit - 1) / unit * unit;
    };
    int planes = nx;
    Slab slab = slab_of(planes);
    while (planes > 4 && (slab.end - slab.ct > kKeepBytes || slab.blocks > 0xffffffffLL))
        slab = slab_of(planes = half(planes));
    if (slab.blocks > 0xffffffffLL) return sf_fail("sf_voxelize: grid too large");
    std::vector<char> host(sent);
    std::memcpy(host.data(), marked.data(), sizeof(sf_sdf_node) * n_marked);
    for (int q = 0; q < n_marked; ++q) {
        const int op = marked[q].op;
        IvNode v = interval_node(marked[q]);
        if (op == kSkip || op == 10 || op == 11 || op == 12) std::memcpy(&v.a[0].x, &first_bit[q], 4);
        std::memcpy(host.data() + off_iv + sizeof(IvNode) * q, &v, sizeof(v));
    }
    if (coords) {
        size_t o = off_co;
        const int n3[3] = {nx, ny, nz};
        for (int a = 0; a < 3; ++a) {
            std::memcpy(host.data() + o, coords[a], sizeof(double) * n3[a]);
            o += sizeof(double) * n3[a];
        }
    }
    SfRelaxedCapture relaxed;  // (the call allocates and waits)
    Scratch scratch;
    while (int rc = scratch.take(slab.end, st)) {
        if (planes <= 4) return rc;
        slab = slab_of(planes = half(planes));
    }
    char* b = scratch.p;
    scratch.idle = false;
    if (cudaMemcpyAsync(b, host.data(), sent, cudaMemcpyHostToDevice, st) != cudaSuccess)
        return sf_fail("sf_voxelize: upload failed");
    const sf_sdf_node* prog = reinterpret_cast<const sf_sdf_node*>(b);
    const IvNode* ivp = reinterpret_cast<const IvNode*>(b + off_iv);
    for (int first = 0; first < nx; first += planes) {
        const int n = nx - first < planes ? nx - first : planes, si = (n + 15) / 16;
        const VxGrid g{n, ny, nz, invert, first, nx, res,
                       coords ? reinterpret_cast<const double*>(b + off_co) : nullptr,
                       reinterpret_cast<float2*>(b + slab.ax), reinterpret_cast<unsigned*>(b + slab.ct),
                       reinterpret_cast<unsigned*>(b + slab.q), si, sj, sk,
                       reinterpret_cast<unsigned long long*>(b + slab.l),
                       reinterpret_cast<unsigned char*>(b + slab.sd), out + (long long)first * ny * nz};
        const long long supers = (long long)si * sj * sk;
        k_vx_axes<<<(unsigned)(((long long)n + ny + nz + 127) / 128), 128, 0, st>>>(g);
        // One thread walks the whole program for a super-block, so that takes its
        // latency however few there are, and pays where they fill the chip.  Calls with
        // and without (16 resonators): 180 x 240 x 157 (900 super-blocks) 293 and 273
        // us, 300^3 (3610) 313 and 481, 400^3 313 and 747; enclosure 200^3 (1183) 129
        // and 112 to 131, 400^3 (8125) 138 and 172.
        const bool look = supers >= kSuperMin;
        if (look) k_vx_super<<<(unsigned)((supers + 31) / 32), 32, 0, st>>>(g, ivp, n_marked);
        k_vx_blocks<<<(unsigned)supers, 128, 0, st>>>(g, ivp, n_marked, look);
        k_vx_cells<<<152 * 16, 128, 0, st>>>(g, ivp, prog, n_marked);
    }
    if (cudaGetLastError() != cudaSuccess) return sf_fail("k_voxelize launch failed");
    if (cudaStreamSynchronize(st) != cudaSuccess) return sf_fail("sf_voxelize: kernel failed");
    scratch.idle = true;
    return 0;
}

int sf_launch_voxelize_materials(const sf_sdf_node* prog_dev, const int* off_dev,
                                 const uint8_t* ids_dev, int n_regions, int nx, int ny, int nz,
                                 double res, const double* coords_dev, uint8_t* geom,
                                 uint8_t* mat, int* err_dev, cudaStream_t st) {
    dim3 blk(32, 8, 1), grd((nz + 31) / 32, (ny + 7) / 8, nx);
    k_voxelize_materials<<<grd, blk, 0, st>>>(prog_dev, off_dev, ids_dev, n_regions, nx, ny, nz,
                                              res, coords_dev, geom, mat, err_dev);
    return cudaGetLastError() == cudaSuccess ? 0 : sf_fail("k_voxelize_materials launch failed");
}
