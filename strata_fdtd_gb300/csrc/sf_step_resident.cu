// sf_step_resident.cu -- many steps of one small grid in one launch, its state
// held on the chip.
//
// A step of a small grid is short of work: 100^3 took 9.1 us per launch of the
// warp-tile kernel, of which reading and writing the state accounts for less
// than half.  k_resident cuts the grid into at most one block per SM, loads
// each block's state once, and advances it n steps: the two velocity
// components along x and z stay in registers, the pressure and the y component
// in shared memory, and only the pressures on the faces between blocks travel
// through L2.
//
// Block: `nci` chunks of L planes x `nj` rows x `nq` quads of 4 k cells; one
// thread owns a chunk of one row's quad (4 L cells).  A step is two phases with
// a block barrier after each:
//   V  send the block's outermost pressures to the neighbouring blocks; update
//      the high faces inside the block (the messages travel meanwhile);
//      receive the neighbours' pressures and update the faces between blocks.
//   P  update the pressures from those faces.
// Sending, receiving and the faces between blocks are shared out over all
// threads in units of four values, whoever owns the cells (threads of their own
// for them, 96 beside 512, were the longest path of a step).
// A face between two blocks is updated by both, with the same operations on
// the same values, so no face velocity is ever sent.  Velocities are kept
// before their PML decay (the pressure update uses that value) and decayed
// when the next step reads them.  Every cell sees the operations of k_step
// (sf_step.cu) in their order: results are bit-identical.
//
// Bound by latency and shared-memory traffic: what a step waits for is one
// message through L2 (about 1 us) and two barriers; the shared-memory reads and
// writes of 15 000 cells take about 3 us of an SM.  Measured on GB300, whole
// run_steps calls per step, single-step kernels -> this one: 52 x 44 x 48 7.1 ->
// 2.3 us, 100^3 9.7 -> 3.9 us, stretched 144 x 120 x 132 20.3 -> 10.0 us.
//
// Messages carry each 32-bit value beside a 32-bit step tag in one 64-bit
// word, so a reader that sees the tag has the value: no fence and no flag.
// Two sets of mailboxes alternate; a block sends step t + 2 only after the
// neighbour has sent t + 1, hence has read t.  The launch is cooperative (all
// blocks resident), launches of a device run one after another (sf_api.cu),
// and every wait is bounded: when one expires the kernel raises the plan's
// error flag and returns without writing the state.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "sf_common.cuh"
#include "sf_kernels.h"

namespace {

typedef unsigned long long u64;

__device__ __forceinline__ u64 tagged(float v, unsigned tag) {
    return ((u64)tag << 32) | __float_as_uint(v);
}
__device__ __forceinline__ void send2(u64* p, u64 a, u64 b) {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ ulonglong2 recv2(const u64* p) {
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}

// Where a block lies: chunk, row and quad ranges and their counts.
struct Box {
    int c0, nci, j0, nj, q0, nq;
    bool lo[3], hi[3];  // a neighbouring block on that side
};

__device__ __forceinline__ Box box_of(const SfResArgs& A) {
    Box b;
    const int bk = blockIdx.x % A.bk, bj = blockIdx.x / A.bk % A.bj, bi = blockIdx.x / A.bk / A.bj;
    b.c0 = (int)((long long)bi * A.chunks / A.bi);
    b.nci = (int)((long long)(bi + 1) * A.chunks / A.bi) - b.c0;
    b.j0 = (int)((long long)bj * A.a.ny / A.bj);
    b.nj = (int)((long long)(bj + 1) * A.a.ny / A.bj) - b.j0;
    b.q0 = (int)((long long)bk * A.quads / A.bk);
    b.nq = (int)((long long)(bk + 1) * A.quads / A.bk) - b.q0;
    b.lo[0] = bi > 0;
    b.lo[1] = bj > 0;
    b.lo[2] = bk > 0;
    b.hi[0] = bi + 1 < A.bi;
    b.hi[1] = bj + 1 < A.bj;
    b.hi[2] = bk + 1 < A.bk;
    return b;
}

// Flag bits of cell (i, j, k): the plan's byte, or all open inside the grid.
__device__ __forceinline__ unsigned cell_flags(const SfStepArgs& a, int i, int j, int k) {
    if (i >= a.nx || j >= a.ny || k >= a.nz) return 0;
    if (a.flags) return a.flags[(long long)i * a.plane + (long long)j * a.nz + k] & 15u;
    return SF_AIR | (i < a.nx - 1 ? SF_OPX : 0) | (j < a.ny - 1 ? SF_OPY : 0) |
           (k < a.nz - 1 ? SF_OPZ : 0);
}

__device__ __forceinline__ float cell_value(const SfStepArgs& a, const float* f, int i, int j, int k) {
    return i < a.nx && j < a.ny && k < a.nz ? f[(long long)i * a.plane + (long long)j * a.nz + k] : 0.0f;
}

__device__ __forceinline__ void load4(const SfStepArgs& a, const float* f, int i, int j, int k,
                                      float (&v)[4]) {
    if (i < a.nx && a.nz % 4 == 0) {
        const float4 t = *reinterpret_cast<const float4*>(f + (long long)i * a.plane + (long long)j * a.nz + k);
        v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
        return;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = cell_value(a, f, i, j, k + e);
}

__device__ __forceinline__ void store4(const SfStepArgs& a, float* f, int i, int j, int k,
                                       const float (&v)[4]) {
    if (i >= a.nx) return;
    float* o = f + (long long)i * a.plane + (long long)j * a.nz + k;
    if (a.nz % 4 == 0) {
        *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
        return;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e)
        if (k + e < a.nz) o[e] = v[e];
}

typedef SfResLayout Layout;  // of the largest block: the same offsets in every block

// Message units of 4 values over one side of a block (sides: x low, x high, y
// low, ...).  Within a side the words are numbered (j, k) or (i, k); on the z
// sides (chunk, j, plane) when a thread has 4 planes or more, else (i, j), so that
// a unit's values lie at one stride.
__host__ __device__ inline int side_units(int side, int planes, int nj, int nq) {
    return side < 2 ? nj * nq : (side < 4 ? planes * nq : (planes * nj + 3) / 4);
}

// Kinds with many planes per thread keep the z velocities in shared memory
// too (UZ then holds every z face; otherwise only those at quad ends, the rest
// in registers): vx and vz of 8 planes would need 64 registers and spill.
__host__ __device__ constexpr bool z_shared(int L) { return L >= 8; }

// Floats of one row of UZ, and the places of the low and the high boundary
// face in it.  Quad-end rows: slot q + 1 is the high face of quad q.  Full rows:
// the face above cell k is at 4 + k, so that quads are aligned.
__host__ __device__ constexpr int z_row(int L, int nq) { return z_shared(L) ? 4 * nq + 4 : nq + 1; }
__host__ __device__ constexpr int z_low(int L) { return z_shared(L) ? 3 : 0; }
__host__ __device__ constexpr int z_high(int L, int nq) { return z_shared(L) ? 4 * nq + 3 : nq; }

// Cells of a block's share of the plane perpendicular to an axis
__host__ __device__ inline int plane_cells(int axis, int planes, int nj, int row) {
    return axis == 0 ? nj * row : (axis == 1 ? planes * row : planes * nj);
}

inline Layout layout(int L, int nci, int nj, int nq, int n_probe, bool nu, const SfResExtra* x) {
    const int planes = nci * L;
    Layout l;
    int o = 0;
    auto take = [&](int floats) {
        const int at = o;
        o += (floats + 3) & ~3;
        return at;
    };
    l.src = take(2 * SF_MAX_SOURCES);
    l.ctl = take(4);
    l.side = take(12);
    l.P = take(planes * nj * nq * 4);
    l.UX = take((nci + 1) * nj * nq * 4);
    l.UY = take(planes * (nj + 1) * nq * 4);
    l.UZ = take(planes * nj * z_row(L, nq));
    l.dx = take(planes);
    l.dy = take(nj);
    l.dz = take(nq * 4);
    l.cx = l.cy = l.cz = l.sx = l.sy = l.sz = 0;
    if (nu) {
        l.cx = take(planes);
        l.cy = take(nj);
        l.cz = take(nq * 4);
        l.sx = take(planes);
        l.sy = take(nj);
        l.sz = take(nq * 4);
    }
    l.probe = take(n_probe * 2);
    for (int q = 0; q < SF_MAX_PLANE_OPS; ++q)
        for (int side = 0; side < 2; ++side)
            l.prev[q][side] =
                x && q < x->n_plane ? take(plane_cells(x->ops[q].axis, planes, nj, nq * 4)) : 0;
    int listed = 0;
    for (int q = 0; x && q < x->n_plane; ++q)
        listed += (x->ops[q].kind == 0 ? 2 : 1) * plane_cells(x->ops[q].axis, planes, nj, nq * 4);
    l.plist = take((listed + 1) / 2);  // two to a word
    long long wcap = 0;  // entries a block can have: its overlap with the sources' box
    if (x && x->w_slots > 0) {
        const int dims[3] = {planes, nj, nq * 4};
        wcap = x->w_slots;
        for (int a = 0; a < 3; ++a) {
            const int e = x->wbox[3 + a] - x->wbox[a];
            wcap *= e < dims[a] ? e : dims[a];
        }
    }
    l.wlist = wcap > 16000 ? (o = 1 << 28) : take((int)wcap * 4);
    l.mic = take(x ? x->n_mic * 8 * 4 : 0);
    l.end = o;
    return l;
}

extern __shared__ __align__(16) float smem[];

// Geometry of the block a thread works in.
struct Place {
    Box b;
    int planes, row, plane, gi0, gk0;
};

// Pairs of floats for the packed FP32 instructions: two results per issue slot
// (the phases were bound by issue), each lane rounded as the scalar operation.
__device__ __forceinline__ u64 pair(float a, float b) {
    return ((u64)__float_as_uint(b) << 32) | __float_as_uint(a);
}
__device__ __forceinline__ float lo_of(u64 p) { return __uint_as_float((unsigned)p); }
__device__ __forceinline__ float hi_of(u64 p) { return __uint_as_float((unsigned)(p >> 32)); }
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// a * b, as a * b + (-0): rounded as the product, signed zeros included.  The
// assembler fuses a packed mul and a following packed add into one rounding,
// even with .rn and -fmad=false (94 of 512 random sums differed), also when the
// -0 is a literal; with a -0 that it cannot see it does not (0 of 512).
__constant__ u64 kNegZero = 0x8000000080000000ull;
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(kNegZero));
    return r;
}
__device__ __forceinline__ u64 sub2(u64 a, u64 b) {  // a + (-b): the same rounding and zero signs
    u64 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Four consecutive cells.
struct Quad {
    u64 a, b;
    __device__ __forceinline__ float operator[](int e) const {
        return e == 0 ? lo_of(a) : (e == 1 ? hi_of(a) : (e == 2 ? lo_of(b) : hi_of(b)));
    }
};
__device__ __forceinline__ Quad quad(float x, float y, float z, float w) { return {pair(x, y), pair(z, w)}; }
__device__ __forceinline__ Quad lds_q(int at) {
    const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(smem + at);
    return {t.x, t.y};
}
__device__ __forceinline__ void sts_q(int at, const Quad& v) {
    *reinterpret_cast<ulonglong2*>(smem + at) = make_ulonglong2(v.a, v.b);
}
__device__ __forceinline__ Quad operator+(const Quad& x, const Quad& y) { return {add2(x.a, y.a), add2(x.b, y.b)}; }
__device__ __forceinline__ Quad operator-(const Quad& x, const Quad& y) { return {sub2(x.a, y.a), sub2(x.b, y.b)}; }
__device__ __forceinline__ Quad operator*(const Quad& x, const Quad& y) { return {mul2(x.a, y.a), mul2(x.b, y.b)}; }
__device__ __forceinline__ Quad operator*(u64 c, const Quad& y) { return {mul2(c, y.a), mul2(c, y.b)}; }
__device__ __forceinline__ Quad load_q(const SfStepArgs& a, const float* f, int i, int j, int k) {
    float t[4];
    load4(a, f, i, j, k, t);
    return quad(t[0], t[1], t[2], t[3]);
}
__device__ __forceinline__ void store_q(const SfStepArgs& a, float* f, int i, int j, int k, const Quad& v) {
    const float t[4] = {v[0], v[1], v[2], v[3]};
    store4(a, f, i, j, k, t);
}
// v where bit (4 e) of f is set, else zero
__device__ __forceinline__ Quad where(unsigned f, const Quad& v) {
    return quad(f & 1u ? v[0] : 0.0f, f & 0x10u ? v[1] : 0.0f, f & 0x100u ? v[2] : 0.0f,
                f & 0x1000u ? v[3] : 0.0f);
}

// What a compute thread keeps between the phases.
template <int L>
struct Own {
    Quad vx[L], vz[z_shared(L) ? 1 : L];
    unsigned flags[(L + 1) / 2];  // 16 bits per plane
};

// Where a compute thread works: its tile, its places in shared memory and the
// strides from plane to plane.
struct Tile {
    int ci, j, q;
    int p, ux, uy, uz;         // own pressure, low x face slot, high y face, high z face
    int row, dp, duy, duz;
    bool next_x, next_y, next_z;  // the next tile along the axis is in the block
    bool own_x, own_y, own_z;     // the high face is this thread's (not a message unit's)
};

// Phase V of one compute thread.  MODE 0: every face open; 1: some closed (a
// wall, or outside the grid); 2: also some at the grid's high edges, which no
// step updates.  PML: some decay is not 1 (taken as 1 on the first step).
template <int L, bool NU, int MODE, bool PML>
__device__ __forceinline__ void phase_v(const SfStepArgs& a, const Layout& S, const Tile& T, const Place& g,
                                        Own<L>& o, bool first) {
    const int i0 = g.gi0 + T.ci * L, gj = g.b.j0 + T.j, k0 = g.gk0 + T.q * 4;
    const u64 cv = pair(a.cv, a.cv);
    u64 cvy = cv, dj = 0;
    Quad dk{}, cvz{cv, cv};
    if (NU) {
        const float c = smem[S.cy + T.j];
        cvy = pair(c, c);
        cvz = lds_q(S.cz + T.q * 4);
    }
    if (PML) {
        const float d = first ? 1.0f : smem[S.dy + T.j];
        dj = pair(d, d);
        dk = first ? quad(1.0f, 1.0f, 1.0f, 1.0f) : lds_q(S.dz + T.q * 4);
    }
    int p = T.p, uy = T.uy, uz = T.uz;
    Quad pc = lds_q(p);
#pragma unroll
    for (int l = 0; l < L; ++l) {
        const Quad pn = l + 1 < L || T.next_x ? lds_q(p + T.dp) : pc;
        const Quad pj = T.next_y ? lds_q(p + T.row) : pc;
        const float pk = T.next_z ? smem[p + 4] : pc[3];
        const unsigned f = MODE ? o.flags[l / 2] >> (16 * (l & 1)) : 0u;
        {  // x
            u64 c = cv;
            if (NU) {
                const float t = smem[S.cx + T.ci * L + l];
                c = pair(t, t);
            }
            Quad v = o.vx[l];
            if (PML) {
                const float d = first ? 1.0f : smem[S.dx + T.ci * L + l];
                v = pair(d, d) * v;
            }
            Quad u = v + c * (pn - pc);
            if (MODE) u = where(f >> 1, u);  // SF_OPX
            if (MODE == 2 && i0 + l == a.nx - 1) u = v;
            if (l + 1 < L || T.own_x) o.vx[l] = u;
            if (l + 1 == L && T.next_x) sts_q(T.ux + g.plane, u);
        }
        if (T.own_y) {
            Quad v = lds_q(uy);
            if (PML) v = dj * v;
            Quad u = v + cvy * (pj - pc);
            if (MODE) u = where(f >> 2, u);  // SF_OPY
            if (MODE == 2 && gj == a.ny - 1) u = v;
            sts_q(uy, u);
        }
        {  // z
            Quad v = z_shared(L) ? lds_q(uz) : o.vz[z_shared(L) ? 0 : l];
            const Quad was = v;
            if (PML) v = dk * v;
            const Quad d = quad(f_sub(pc[1], pc[0]), f_sub(pc[2], pc[1]), f_sub(pc[3], pc[2]), f_sub(pk, pc[3]));
            Quad u = v + cvz * d;
            if (MODE) u = where(f >> 3, u);  // SF_OPZ
            if (MODE == 2 && k0 + 3 >= a.nz - 1)
                u = quad(k0 == a.nz - 1 ? v[0] : u[0], k0 + 1 == a.nz - 1 ? v[1] : u[1],
                         k0 + 2 == a.nz - 1 ? v[2] : u[2], k0 + 3 == a.nz - 1 ? v[3] : u[3]);
            if (z_shared(L)) {
                if (T.own_z) {
                    sts_q(uz, u);
                } else {  // the last one is a message unit's
                    *reinterpret_cast<u64*>(smem + uz) = u.a;
                    smem[uz + 2] = u[2];
                }
            } else {
                o.vz[z_shared(L) ? 0 : l] = T.own_z ? u : Quad{u.a, pair(u[2], was[3])};
                if (T.next_z) smem[uz] = u[3];
            }
        }
        pc = pn;
        p += T.dp;
        uy += T.duy;
        uz += T.duz;
    }
}

// Phase P of one compute thread.
template <int L, bool NU, bool MASK, bool PML>
__device__ __forceinline__ void phase_p(const SfStepArgs& a, const Layout& S, const Tile& T, const Place& g,
                                        const Own<L>& o) {
    const u64 cp = pair(a.cp, a.cp);
    u64 dj = 0, sy = 0;
    Quad dk{}, sz{};
    if (PML) {
        const float d = smem[S.dy + T.j];
        dj = pair(d, d);
        dk = lds_q(S.dz + T.q * 4);
    }
    if (NU) {
        const float t = smem[S.sy + T.j];
        sy = pair(t, t);
        sz = lds_q(S.sz + T.q * 4);
    }
    int p = T.p, uy = T.uy, uz = T.uz;
    Quad lo = lds_q(T.ux);
#pragma unroll
    for (int l = 0; l < L; ++l) {
        const Quad ylo = lds_q(uy - T.row), yhi = lds_q(uy), pc = lds_q(p);
        const float zlo = smem[uz - 1];
        Quad z = z_shared(L) ? lds_q(uz) : o.vz[z_shared(L) ? 0 : l];
        if (!z_shared(L) && !T.own_z) z.b = pair(z[2], smem[uz]);
        const Quad hi = l + 1 < L || T.own_x ? o.vx[l] : lds_q(T.ux + g.plane);
        Quad ex = hi - lo, ey = yhi - ylo;
        Quad ez = quad(f_sub(z[0], zlo), f_sub(z[1], z[0]), f_sub(z[2], z[1]), f_sub(z[3], z[2]));
        if (NU) {
            const float t = smem[S.sx + T.ci * L + l];
            ex = pair(t, t) * ex;
            ey = sy * ey;
            ez = sz * ez;
        }
        Quad pn = pc + cp * ((ex + ey) + ez);
        if (MASK) pn = where(o.flags[l / 2] >> (16 * (l & 1)), pn);  // SF_AIR
        if (PML) {
            const float d = smem[S.dx + T.ci * L + l];
            pn = dk * (dj * (pair(d, d) * pn));
        }
        sts_q(p, pn);
        lo = hi;
        p += T.dp;
        uy += T.duy;
        uz += T.duz;
    }
}

// ---- between the steps --------------------------------------------------------

// float(double(was) + coeff * double(d)), the two FP64 operations rounded, with
// coeff = c.x + c.y to 2^-47 (c.x = 0: no such split).  In FP32 x = zh + zl is was
// + coeff d to 2^-44 (|c.x d| + |s|), and the FP64 result differs from it by less;
// where everything within 2^-43 of that scale rounds to zh, zh is the answer.
// Elsewhere (one in 2^17, and below 2^-70, where a product's low part could be
// lost) the FP64 pipe decides: it has 2 lanes a clock, and took 0.5 us of a step
// for a corner block's 1344 plane cells (112 x 96 x 120, three absorbing axes).
__device__ __forceinline__ float plane_value(float was, double coeff, float2 c, float d) {
    const float ph = f_mul(c.x, d);
    if (d == 0.0f && c.x != 0.0f) return f_add(was, ph);  // exact, the sign of zero too
    const float pl = __fmaf_rn(c.y, d, __fmaf_rn(c.x, d, -ph));
    const float s = f_add(was, ph), bv = f_sub(s, was);
    const float t = f_add(f_add(f_sub(was, f_sub(s, bv)), f_sub(ph, bv)), pl);
    const float zh = f_add(s, t), tv = f_sub(zh, s);
    const float zl = f_add(f_sub(s, f_sub(zh, tv)), f_sub(t, tv));
    const float err = f_mul(f_add(fabsf(ph), fabsf(s)), 0x1p-43f);
    if (fabsf(ph) >= 0x1p-70f && f_add(zh, f_add(zl, err)) == zh && f_add(zh, f_sub(zl, err)) == zh)
        return zh;
    return __double2float_rn(d_add((double)was, d_mul(coeff, (double)d)));
}

// The places in shared memory of the block's cells in the grid's absorbing planes,
// by operation and end, each list as long as its stored plane (kNoCell: past the
// grid).  Built once: with the places worked out at each step an operation took
// 0.65 us of a step, of two cells a thread (112 x 96 x 120, three operations, two
// sources and two microphones: 7.84 us a step, 7.16 with the lists; 9.56 with four
// cells' loads before their stores, which spilled).
constexpr unsigned short kNoCell = 0xffff;
__device__ __forceinline__ bool has_plane(const Place& g, const sf_plane_bc& op, int side) {
    return !(side ? g.b.hi[op.axis] : g.b.lo[op.axis]) && (op.kind == 0 || op.side == side);
}
__device__ __forceinline__ void list_planes(const SfStepArgs& a, const SfResExtra& x, const Layout& S,
                                            const Place& g) {
    unsigned short* list = reinterpret_cast<unsigned short*>(smem + S.plist);
    for (int q = 0; q < x.n_plane; ++q) {
        const sf_plane_bc& op = x.ops[q];
        const int ax = op.axis, cnt = plane_cells(ax, g.planes, g.b.nj, g.row);
        const int n = ax == 0 ? a.nx - g.gi0 : (ax == 1 ? g.b.nj : a.nz - g.gk0);  // cells up to the grid's end
        const int stride = ax == 0 ? g.plane : (ax == 1 ? g.row : 1);
        for (int side = 0; side < 2; ++side) {
            if (!has_plane(g, op, side)) continue;
            for (int t = threadIdx.x; t < cnt; t += blockDim.x) {
                const int per = ax == 2 ? g.b.nj : g.row, u = t / per, v = t % per;
                const bool live = (ax == 0 || g.gi0 + u < a.nx) && (ax == 2 || g.gk0 + v < a.nz);
                const int cell = u * (ax == 0 ? g.row : g.plane) + v * (ax == 2 ? g.row : 1);
                list[t] = live ? (unsigned short)(S.P + cell + (side ? n - 1 : 0) * stride) : kNoCell;
            }
            list += cnt;
        }
    }
}

// One plane boundary over one end's list (k_plane_bc's arithmetic): its inner
// neighbours lie at `inner`, its stored values at `prev`.
__device__ __forceinline__ void plane_op(const sf_plane_bc& op, float2 coeff, const unsigned short* list,
                                         int cnt, int inner, int prev) {
    for (int t = threadIdx.x; t < cnt; t += blockDim.x) {
        const unsigned cell = list[t];
        if (cell == kNoCell) continue;
        float& pb = smem[cell];
        const float pi = smem[(int)cell + inner];
        float& was = smem[prev + t];
        if (op.kind == 0) {
            pb = plane_value(was, op.coeff, coeff, f_sub(pi, pb));
        } else {
            const double abc = d_add((double)was, d_mul(op.coeff, (double)f_sub(pi, pb)));
            const float rig = f_mul(__double2float_rn(op.reflection), pi);
            pb = __double2float_rn(d_add((double)rig, d_mul(d_sub(1.0, op.reflection), abc)));
        }
        was = pi;
    }
}

// The stored planes between global memory (t over the grid's plane) and the block.
__device__ __forceinline__ void move_prev(const SfStepArgs& a, const SfResExtra& x, const Layout& S,
                                          const Place& g, bool store) {
    for (int q = 0; q < x.n_plane; ++q) {
        const sf_plane_bc& op = x.ops[q];
        const int ax = op.axis, nv = ax == 2 ? a.ny : a.nz;
        const int cnt = plane_cells(ax, g.planes, g.b.nj, g.row);
        for (int side = 0; side < 2; ++side) {
            if (side ? g.b.hi[ax] : g.b.lo[ax]) continue;
            if (op.kind == 1 && op.side != side) continue;
            float* f = op.kind == 1 ? x.prev[q][0] : x.prev[q][side];
            for (int t = threadIdx.x; t < cnt; t += blockDim.x) {
                const int per = ax == 2 ? g.b.nj : g.row;
                const int u = (ax == 0 ? g.b.j0 : g.gi0) + t / per, v = (ax == 2 ? g.b.j0 : g.gk0) + t % per;
                if (u >= (ax == 0 ? a.ny : a.nx) || v >= nv) continue;
                float& here = smem[S.prev[q][side] + t];
                float& there = f[(long long)u * nv + v];
                if (store) there = here;
                else here = there;
            }
        }
    }
}

// The place of cell c in the block's P, or -1 outside the block.
__device__ __forceinline__ int place_of(const SfStepArgs& a, const Place& g, long long c) {
    const int i = (int)(c / a.plane), r = (int)(c % a.plane), j = r / a.nz, k = r % a.nz;
    if (i < g.gi0 || i >= g.gi0 + g.planes || j < g.b.j0 || j >= g.b.j0 + g.b.nj || k < g.gk0 ||
        k >= g.gk0 + g.row)
        return -1;
    return (i - g.gi0) * g.plane + (j - g.b.j0) * g.row + (k - g.gk0);
}

// The sources that reach this thread's cells, in order, after the decays.
template <int L>
__device__ void add_sources(const SfSources& src, const Layout& S, const Tile& T, int i0, int k0,
                            const unsigned (&flags)[(L + 1) / 2], unsigned mask) {
    for (; mask != 0; mask &= mask - 1) {
        const int s = __ffs(mask) - 1;
        const sf_source& Q = src.s[s];
        const double v = reinterpret_cast<const double*>(smem + S.src)[s];
#pragma unroll
        for (int l = 0; l < L; ++l) {
            if (Q.kind == 0 ? i0 + l != Q.a : (Q.a == 0 && i0 + l != Q.b)) continue;
            const unsigned f = flags[l / 2] >> (16 * (l & 1));
            for (int e = 0; e < 4; ++e) {
                if (Q.kind == 0 ? k0 + e != Q.c : (Q.a == 2 && k0 + e != Q.b)) continue;
                if (!(f >> (4 * e) & SF_AIR)) continue;
                float& p = smem[T.p + l * T.dp + e];
                p = __double2float_rn(d_add((double)p, v));
            }
        }
    }
}

template <int L, bool NU>
__device__ __forceinline__ void v_any(const SfStepArgs& a, const Layout& S, const Tile& T, const Place& g,
                                      Own<L>& o, bool first, int mode, bool pml) {
    if (mode == 0) {
        if (pml) phase_v<L, NU, 0, true>(a, S, T, g, o, first);
        else phase_v<L, NU, 0, false>(a, S, T, g, o, first);
    } else if (mode == 1) {
        if (pml) phase_v<L, NU, 1, true>(a, S, T, g, o, first);
        else phase_v<L, NU, 1, false>(a, S, T, g, o, first);
    } else {
        phase_v<L, NU, 2, true>(a, S, T, g, o, first);
    }
}
template <int L, bool NU>
__device__ __forceinline__ void p_any(const SfStepArgs& a, const Layout& S, const Tile& T, const Place& g,
                                      const Own<L>& o, int mode, bool pml) {
    if (mode == 0) {
        if (pml) phase_p<L, NU, false, true>(a, S, T, g, o);
        else phase_p<L, NU, false, false>(a, S, T, g, o);
    } else {
        if (pml) phase_p<L, NU, true, true>(a, S, T, g, o);
        else phase_p<L, NU, true, false>(a, S, T, g, o);
    }
}

// Message units a thread has at most.
constexpr int kUnits = 2;

// A mailbox holds the first two words of every unit of its side, then the last
// two, so that neighbouring threads' 16-byte accesses are adjacent.
//
// A message unit: its first pressure and first face in shared memory, its words in
// the neighbour's mailbox and in this block's, and
// side | open faces << 3 | values in the unit << 7 (0: no unit).
struct Unit {
    unsigned at;  // pressure | face << 16
    unsigned d;
    int send, recv;
    __device__ __forceinline__ int side() const { return d & 7; }
    __device__ __forceinline__ bool z() const { return (d & 4) != 0; }
    __device__ __forceinline__ int n() const { return d >> 7; }
    __device__ __forceinline__ int p() const { return at & 0xffffu; }
    __device__ __forceinline__ int f() const { return at >> 16; }
};

// Waits for the words of this thread's units to carry the tag `want`; false when
// the wait ran out (or another thread's did).
__device__ __forceinline__ bool receive(const u64* mail, const Unit (&U)[kUnits], int half, unsigned want,
                                        long long limit, const volatile int* stop, Quad (&r)[kUnits]) {
    for (long long polls = 0;; ++polls) {
        ulonglong2 m[kUnits][2];
        bool ready = true;
#pragma unroll
        for (int w = 0; w < kUnits; ++w) {
            m[w][0] = recv2(mail + U[w].recv);  // a missing unit reads word 0
            m[w][1] = recv2(mail + U[w].recv + half);
        }
#pragma unroll
        for (int w = 0; w < kUnits; ++w) {
            // (a short unit's last words carry its last pressure)
            ready = ready && (U[w].d == 0 || ((unsigned)(m[w][0].x >> 32) == want &&
                                              (unsigned)(m[w][0].y >> 32) == want &&
                                              (unsigned)(m[w][1].x >> 32) == want &&
                                              (unsigned)(m[w][1].y >> 32) == want));
            r[w] = {(m[w][0].x & 0xffffffffu) | (m[w][0].y << 32), (m[w][1].x & 0xffffffffu) | (m[w][1].y << 32)};
        }
        if (ready) return true;
        if (polls >= limit || *stop) return false;
    }
}

template <int L>
__device__ __forceinline__ Unit make_unit(const SfResArgs& A, const Place& g, int u) {
    const SfStepArgs& a = A.a;
    const Layout& S = A.lay;
    const Box& b = g.b;
    struct {
        int p, f;
    } t{S.P, S.UX};
    int side = 0;
    for (; side < 6; ++side) {
        if (!(side & 1 ? b.hi[side >> 1] : b.lo[side >> 1])) continue;
        const int n = side_units(side, g.planes, b.nj, b.nq);
        if (u < n) break;
        u -= n;
    }
    if (side == 6) return Unit{0, 0, 0, 0};
    const int ax = side >> 1, zr = z_row(L, b.nq);
    const bool high = side & 1;
    unsigned open = 0;
    int n = 4;
    if (ax == 0) {
        const int jj = u / b.nq, qq = u % b.nq, gi = high ? g.gi0 + g.planes - 1 : g.gi0 - 1;
        t.p = S.P + (high ? (g.planes - 1) * g.plane : 0) + jj * g.row + qq * 4;
        t.f = S.UX + (high ? b.nci * g.plane : 0) + jj * g.row + qq * 4;
        for (int e = 0; e < 4; ++e) {
            smem[t.f + e] = cell_value(a, a.vx, gi, b.j0 + jj, g.gk0 + qq * 4 + e);
            if (cell_flags(a, gi, b.j0 + jj, g.gk0 + qq * 4 + e) & SF_OPX) open |= 1u << e;
        }
    } else if (ax == 1) {
        const int i = u / b.nq, qq = u % b.nq, gj = high ? b.j0 + b.nj - 1 : b.j0 - 1;
        t.p = S.P + i * g.plane + (high ? (b.nj - 1) * g.row : 0) + qq * 4;
        t.f = S.UY + (i * (b.nj + 1) + (high ? b.nj : 0)) * g.row + qq * 4;
        for (int e = 0; e < 4; ++e) {  // (a high face's compute thread loads the same value)
            smem[t.f + e] = cell_value(a, a.vy, g.gi0 + i, gj, g.gk0 + qq * 4 + e);
            if (cell_flags(a, g.gi0 + i, gj, g.gk0 + qq * 4 + e) & SF_OPY) open |= 1u << e;
        }
    } else {
        const int gk = high ? g.gk0 + g.row - 1 : g.gk0 - 1;
        n = min(4, g.planes * b.nj - u * 4);
        for (int e = n - 1; e >= 0; --e) {
            const int r = u * 4 + e;
            const int i = L >= 4 ? r / L / b.nj * L + r % L : r / b.nj;
            const int jj = L >= 4 ? r / L % b.nj : r % b.nj;
            t.p = S.P + i * g.plane + jj * g.row + (high ? g.row - 1 : 0);
            t.f = S.UZ + (i * b.nj + jj) * zr + (high ? z_high(L, b.nq) : z_low(L));
            smem[t.f] = cell_value(a, a.vz, g.gi0 + i, b.j0 + jj, gk);
            if (cell_flags(a, g.gi0 + i, b.j0 + jj, gk) & SF_OPZ) open |= 1u << e;
        }
    }
    const int step[3] = {A.bj * A.bk, A.bk, 1}, words = A.side_max * 4;
    const int to = (int)blockIdx.x + (high ? step[ax] : -step[ax]);
    return Unit{(unsigned)t.p | ((unsigned)t.f << 16), (unsigned)side | (open << 3) | ((unsigned)n << 7),
                (to * 6 + (side ^ 1)) * words + u * 2, ((int)blockIdx.x * 6 + side) * words + u * 2};
}

// EXTRA: plane boundaries, weighted sources or microphones between the steps
// (sources then follow the plane boundaries, as in sf_plan_step).
template <int L, int MAXT, bool NU, bool EXTRA>
__global__ void __launch_bounds__(MAXT, 1) k_resident(const __grid_constant__ SfResArgs A,
                                                      const __grid_constant__ SfSources src) {
    const SfStepArgs& a = A.a;
    const Layout& S = A.lay;
    Place g;
    g.b = box_of(A);
    const Box& b = g.b;
    g.planes = b.nci * L;
    g.row = b.nq * 4;
    g.plane = b.nj * g.row;
    g.gi0 = b.c0 * L;
    g.gk0 = b.q0 * 4;
    const int tid = threadIdx.x, nthreads = blockDim.x;
    const int planes = g.planes, row = g.row, plane = g.plane, gi0 = g.gi0, gk0 = g.gk0;
    const int zr = z_row(L, b.nq);

    // ---- tables
    for (int t = tid; t < planes; t += nthreads) {
        const int i = gi0 + t;
        smem[S.dx + t] = i < a.nx ? a.dx[i] : 1.0f;
        if (NU) {
            smem[S.cx + t] = i < a.nx ? a.nu_cv[0][i] : 0.0f;
            smem[S.sx + t] = i < a.nx ? a.nu_inv[0][i] : 0.0f;
        }
    }
    for (int t = tid; t < b.nj; t += nthreads) {
        smem[S.dy + t] = a.dy[b.j0 + t];
        if (NU) {
            smem[S.cy + t] = a.nu_cv[1][b.j0 + t];
            smem[S.sy + t] = a.nu_inv[1][b.j0 + t];
        }
    }
    for (int t = tid; t < row; t += nthreads) {
        const int k = gk0 + t;
        smem[S.dz + t] = k < a.nz ? a.dz[k] : 1.0f;
        if (NU) {
            smem[S.cz + t] = k < a.nz ? a.nu_cv[2][k] : 0.0f;
            smem[S.sz + t] = k < a.nz ? a.nu_inv[2][k] : 0.0f;
        }
    }
    volatile int* ctl = reinterpret_cast<volatile int*>(smem + S.ctl);
    if (tid < 4) ctl[tid] = 0;
    if (tid < 6) {  // per side: the decay and the coefficient of its faces
        const int ax = tid >> 1;
        const bool high = tid & 1;
        float d = 1.0f, c = a.cv;
        if (high ? b.hi[ax] : b.lo[ax]) {
            const int gl = ax == 0 ? (high ? gi0 + planes - 1 : gi0 - 1)
                                   : (ax == 1 ? (high ? b.j0 + b.nj - 1 : b.j0 - 1)
                                              : (high ? gk0 + row - 1 : gk0 - 1));
            d = (ax == 0 ? a.dx : (ax == 1 ? a.dy : a.dz))[gl];
            if (NU) c = a.nu_cv[ax][gl];
        }
        smem[S.side + tid * 2] = d;
        smem[S.side + tid * 2 + 1] = c;
    }
    // low faces at the grid's edge are zero; those between blocks come with the units
    for (int t = tid; t < plane; t += nthreads) smem[S.UX + t] = 0.0f;
    for (int t = tid; t < planes * row; t += nthreads)
        smem[S.UY + t / row * (b.nj + 1) * row + t % row] = 0.0f;
    for (int t = tid; t < planes * b.nj; t += nthreads) smem[S.UZ + t * zr + z_low(L)] = 0.0f;
    __syncthreads();

    // ---- message units, probes
    int2* probe = reinterpret_cast<int2*>(smem + S.probe);
    Unit U[kUnits];
#pragma unroll
    for (int w = 0; w < kUnits; ++w) U[w] = make_unit<L>(A, g, tid + w * nthreads);
    for (int t = tid; t < a.n_probe; t += nthreads) {
        const long long c = a.probe_cells[t];
        const int i = (int)(c / a.plane), r = (int)(c % a.plane), jj = r / a.nz, k = r % a.nz;
        if (i < gi0 || i >= gi0 + planes || jj < b.j0 || jj >= b.j0 + b.nj || k < gk0 || k >= gk0 + row)
            continue;
        probe[atomicAdd(const_cast<int*>(ctl) + 1, 1)] =
            make_int2(t, (i - gi0) * plane + (jj - b.j0) * row + (k - gk0));
    }

    // ---- what acts between the steps
    const SfResExtra& x = A.x;
    // microphone corners: (number, value, its decay, -1) in shared memory, or
    // (number, field << 8 | plane << 2 | cell, its decay, thread) in a thread's registers
    // (walked as lists: every owner passing over the 40 corners of two microphones, one
    // a cardioid, took 1.5 us a step)
    int4* mics = reinterpret_cast<int4*>(smem + S.mic);
    int4* wlist = reinterpret_cast<int4*>(smem + S.wlist);  // (place in P, source, weight)
    if (EXTRA) {
        move_prev(a, x, S, g, false);
        list_planes(a, x, S, g);
        for (int q = 0; q < src.n; ++q)
            if (src.s[q].kind == 2)
                for (int t = tid; t < x.wn[q]; t += nthreads) {
                    const int at = place_of(a, g, x.wcells[q][t]);
                    if (at < 0) continue;
                    const long long w = __double_as_longlong(x.ww[q][t]);
                    wlist[atomicAdd(const_cast<int*>(ctl), 1)] = make_int4(at, q, (int)w, (int)(w >> 32));
                }
        for (int t = tid; t < x.n_mic * 8; t += nthreads) {
            const int at = place_of(a, g, x.mic_idx[t]);
            if (at < 0) continue;
            const int i = at / plane, r = at % plane, jj = r / row, k = r % row, l = i % L;
            const int f = x.mic_field ? x.mic_field[t / 8] : 0;
            int4 m = make_int4(t, S.P + at, -1, -1);
            if (f == 2) {
                m.y = S.UY + (i * (b.nj + 1) + jj + 1) * row + k;
                m.z = S.dy + jj;
            } else if (f != 0) {
                m.z = f == 1 ? S.dx + i : S.dz + k;
                const bool slot = f == 1 ? i == planes - 1 && b.hi[0] : z_shared(L) || (k == row - 1 && b.hi[2]);
                if (slot) {
                    m.y = f == 1 ? S.UX + b.nci * plane + jj * row + k
                                 : S.UZ + (i * b.nj + jj) * zr + (z_shared(L) ? 4 + k : b.nq);
                } else {
                    m.y = f << 8 | l << 2 | (k % 4);
                    m.w = (i / L * b.nj + jj) * b.nq + k / 4;
                }
            }
            mics[atomicAdd(const_cast<int*>(ctl) + 3, 1)] = m;
        }
    }

    // ---- this thread's cells
    const bool active = tid < b.nci * b.nj * b.nq;
    Tile T;
    T.q = tid % b.nq;
    T.j = tid / b.nq % b.nj;
    T.ci = tid / b.nq / b.nj;
    T.row = row;
    T.dp = plane;
    T.duy = (b.nj + 1) * row;
    T.duz = b.nj * zr;
    T.p = S.P + (T.ci * L) * T.dp + T.j * row + T.q * 4;
    T.ux = S.UX + (T.ci * b.nj + T.j) * row + T.q * 4;
    T.uy = S.UY + (T.ci * L) * T.duy + (T.j + 1) * row + T.q * 4;
    T.uz = S.UZ + (T.ci * L) * T.duz + T.j * zr + (z_shared(L) ? 4 + 4 * T.q : T.q + 1);
    T.next_x = T.ci + 1 < b.nci;
    T.next_y = T.j + 1 < b.nj;
    T.next_z = T.q + 1 < b.nq;
    T.own_x = T.next_x || !b.hi[0];
    T.own_y = T.next_y || !b.hi[1];
    T.own_z = T.next_z || !b.hi[2];
    const int gj = b.j0 + T.j, k0 = gk0 + T.q * 4, i0 = gi0 + T.ci * L;
    Own<L> o;
    int mode = 0;
    bool pml = false;
    unsigned smask = 0;
#pragma unroll
    for (int w = 0; w < (L + 1) / 2; ++w) o.flags[w] = 0;
    if (active) {
#pragma unroll
        for (int l = 0; l < L; ++l) {
            sts_q(T.p + l * T.dp, load_q(a, a.p, i0 + l, gj, k0));
            // (a face between blocks: its unit's thread loads the same value)
            sts_q(T.uy + l * T.duy, load_q(a, a.vy, i0 + l, gj, k0));
            o.vx[l] = load_q(a, a.vx, i0 + l, gj, k0);
            const Quad z = load_q(a, a.vz, i0 + l, gj, k0);
            if (z_shared(L)) sts_q(T.uz + l * T.duz, z);
            else o.vz[z_shared(L) ? 0 : l] = z;
            unsigned f = 0;
            for (int e = 0; e < 4; ++e) f |= cell_flags(a, i0 + l, gj, k0 + e) << (4 * e);
            o.flags[l / 2] |= f << (16 * (l & 1));
            if (f != 0xffffu) mode = 1;
            pml = pml || smem[S.dx + T.ci * L + l] != 1.0f;
        }
        pml = pml || smem[S.dy + T.j] != 1.0f;
        for (int e = 0; e < 4; ++e) pml = pml || smem[S.dz + T.q * 4 + e] != 1.0f;
        if (i0 + L >= a.nx || gj == a.ny - 1 || k0 + 4 >= a.nz) mode = 2;
        for (int s = 0; s < src.n; ++s) {
            const sf_source& Q = src.s[s];
            if (EXTRA && Q.kind == 2) continue;
            const int at = Q.kind == 0 ? Q.a : Q.b;
            const bool in_i = at >= i0 && at < i0 + L;
            bool can;
            if (Q.kind == 0) can = in_i && Q.b == gj && Q.c >= k0 && Q.c < k0 + 4;
            else if (Q.a == 0) can = in_i;
            else if (Q.a == 1) can = Q.b == gj;
            else can = Q.b >= k0 && Q.b < k0 + 4;
            if (can) smask |= 1u << s;
        }
    }
    // a warp takes one path: the plainest that suits all its lanes
    mode = __reduce_max_sync(0xffffffffu, mode);
    pml = __any_sync(0xffffffffu, pml);
    __syncthreads();
    const int probes = ctl[1];
    const bool has_units = U[0].d != 0;
    const int n_w = EXTRA ? ctl[0] : 0, n_mics = EXTRA ? ctl[3] : 0;
    // a thread's own corners as a list (the next one + 1 in bits 16 up of .y)
    int my_mics = -1;
    for (int t = n_mics - 1; t >= 0; --t)
        if (mics[t].w == tid) {
            mics[t].y |= (my_mics + 1) << 16;
            my_mics = t;
        }
    // the state's values at the microphone corners after step s
    auto record_mics = [&](int s) {
        float* out = x.corners + (size_t)s * x.n_mic * 8;
        for (int t = tid; t < n_mics; t += nthreads) {
            const int4 m = mics[t];
            if (m.w >= 0) continue;
            out[m.x] = m.z < 0 ? smem[m.y] : f_mul(smem[m.y], smem[m.z]);
        }
        for (int t = my_mics; t >= 0;) {
            const int4 m = mics[t];
            t = (m.y >> 16) - 1;
            float v = 0.0f;
#pragma unroll
            for (int l = 0; l < L; ++l) {
                if (l != (m.y >> 2 & 63)) continue;
                const Quad f = (m.y >> 8 & 255) == 1 ? o.vx[l] : o.vz[z_shared(L) ? 0 : l];
                const int e = m.y & 3;
                v = e == 0 ? f[0] : (e == 1 ? f[1] : (e == 2 ? f[2] : f[3]));
            }
            out[m.x] = f_mul(v, smem[m.z]);
        }
    };
    const int z_ps = L >= 4 ? plane : row, z_fs = L >= 4 ? b.nj * zr : zr;
    const size_t parity = (size_t)gridDim.x * 6 * A.side_max * 4;
    const int half = A.side_max * 2;

    for (int s = 0; s < A.n_steps; ++s) {
        // ---- V
        const unsigned tag = A.tag + (unsigned)s;
        u64* mail = A.mail + (tag & 1) * parity;
        double sv = 0.0;
        if (tid < src.n) sv = a.src_val[(size_t)s * src.n + tid];
        if (has_units) {
#pragma unroll
            for (int w = 0; w < kUnits; ++w) {
                if (U[w].d == 0) continue;
                Quad v;
                if (!U[w].z()) {
                    v = lds_q(U[w].p());
                } else {  // a short unit's last words repeat its last pressure
                    const int n = U[w].n() - 1, p = U[w].p();
                    v = quad(smem[p], smem[p + min(1, n) * z_ps], smem[p + min(2, n) * z_ps],
                             smem[p + min(3, n) * z_ps]);
                }
                send2(mail + U[w].send, tagged(v[0], tag), tagged(v[1], tag));
                send2(mail + U[w].send + half, tagged(v[2], tag), tagged(v[3], tag));
            }
        }
        if (s > 0)
            for (int t = tid; t < probes; t += nthreads)
                a.trace_prev[(size_t)(s - 1) * a.n_probe + probe[t].x] = smem[S.P + probe[t].y];
        if (active) v_any<L, NU>(a, S, T, g, o, s == 0, mode, pml);
        if (has_units) {
            const unsigned want = tag + ((A.hold && blockIdx.x == 0) ? 0x40000000u : 0u);
            Quad r[kUnits];
            if (!receive(mail, U, half, want, A.poll_limit, ctl + 2, r)) ctl[2] = 1;
#pragma unroll
            for (int w = 0; w < kUnits; ++w) {
                if (U[w].d == 0) continue;
                const int side = U[w].side(), p = U[w].p(), f = U[w].f(), n = U[w].n();
                const float d = s == 0 ? 1.0f : smem[S.side + side * 2];
                const float c = NU ? smem[S.side + side * 2 + 1] : a.cv;
                Quad own, v;
                if (!U[w].z()) {
                    own = lds_q(p);
                    v = lds_q(f);
                } else {
                    own = quad(smem[p], smem[p + min(1, n - 1) * z_ps], smem[p + min(2, n - 1) * z_ps],
                               smem[p + min(3, n - 1) * z_ps]);
                    v = quad(smem[f], smem[f + min(1, n - 1) * z_fs], smem[f + min(2, n - 1) * z_fs],
                             smem[f + min(3, n - 1) * z_fs]);
                }
                const Quad dp = side & 1 ? r[w] - own : own - r[w];
                Quad u = pair(d, d) * v + pair(c, c) * dp;
                const unsigned open = U[w].d >> 3 & 15u;
                if (open != 15u)
                    u = quad(open & 1u ? u[0] : 0.0f, open & 2u ? u[1] : 0.0f, open & 4u ? u[2] : 0.0f,
                             open & 8u ? u[3] : 0.0f);
                if (!U[w].z()) {
                    sts_q(f, u);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (e < n) smem[f + e * z_fs] = u[e];
                }
            }
        }
        if (tid < src.n) reinterpret_cast<double*>(smem + S.src)[tid] = sv;
        __syncthreads();
        if (ctl[2]) {  // block-uniform: the state in global memory stays as it was
            if (tid == 0) *A.err = 1;
            return;
        }
        // ---- P
        if (active) {
            p_any<L, NU>(a, S, T, g, o, mode, pml);
            if (!EXTRA && smask) add_sources<L>(src, S, T, i0, k0, o.flags, smask);
        }
        __syncthreads();
        if (EXTRA) {
            const unsigned short* list = reinterpret_cast<const unsigned short*>(smem + S.plist);
            for (int q = 0; q < x.n_plane; ++q) {
                const sf_plane_bc& op = x.ops[q];
                const int ax = op.axis, cnt = plane_cells(ax, planes, b.nj, row);
                const int stride = ax == 0 ? plane : (ax == 1 ? row : 1);
                for (int side = 0; side < 2; ++side) {  // (an axis has 4 cells or more: no common ones)
                    if (!has_plane(g, op, side)) continue;
                    plane_op(op, x.coeff[q], list, cnt, side ? -stride : stride, S.prev[q][side]);
                    list += cnt;
                }
                __syncthreads();
            }
            for (int q = 0; q < src.n; ++q) {
                if (src.s[q].kind == 2) {  // k_inject_weighted's arithmetic
                    const double v = reinterpret_cast<const double*>(smem + S.src)[q];
                    for (int t = tid; t < n_w; t += nthreads) {
                        const int4 w = wlist[t];
                        if (w.y != q) continue;
                        float& p = smem[S.P + w.x];
                        const double ww = __longlong_as_double(((long long)w.w << 32) | (unsigned)w.z);
                        p = __double2float_rn(d_add((double)p, d_mul(v, ww)));
                    }
                } else if (smask >> q & 1u) {
                    add_sources<L>(src, S, T, i0, k0, o.flags, 1u << q);
                }
                __syncthreads();
            }
            if (n_mics > 0) {  // before the next step moves the faces between blocks
                record_mics(s);
                __syncthreads();
            }
        }
    }

    // ---- back to global memory, velocities decayed
    for (int t = tid; t < probes; t += nthreads)
        a.trace_prev[(size_t)(A.n_steps - 1) * a.n_probe + probe[t].x] = smem[S.P + probe[t].y];
    if (EXTRA) move_prev(a, x, S, g, true);
    if (!active) return;
    const Quad dk = lds_q(S.dz + T.q * 4);
    const float fj = smem[S.dy + T.j];
    const u64 dj = pair(fj, fj);
#pragma unroll
    for (int l = 0; l < L; ++l) {
        const int i = i0 + l;
        const float fi = smem[S.dx + T.ci * L + l];
        store_q(a, a.po, i, gj, k0, lds_q(T.p + l * T.dp));
        const Quad x = l + 1 < L || T.own_x ? o.vx[l] : lds_q(T.ux + plane);
        store_q(a, a.vxo, i, gj, k0, pair(fi, fi) * x);
        store_q(a, a.vyo, i, gj, k0, dj * lds_q(T.uy + l * T.duy));
        Quad z;
        if (z_shared(L)) z = lds_q(T.uz + l * T.duz);
        else z = T.own_z ? o.vz[z_shared(L) ? 0 : l]
                         : Quad{o.vz[z_shared(L) ? 0 : l].a,
                                pair(o.vz[z_shared(L) ? 0 : l][2], smem[T.uz + l * T.duz])};
        store_q(a, a.vzo, i, gj, k0, dk * z);
    }
}

// ---- partition ----------------------------------------------------------------

// Planes per thread, threads at most (512 of 128 registers: with 640 to 768 the
// kernels spilled more, 52 x 44 x 48 0.73 ms against 0.69 for 250 steps, 100^3 2.44
// against 2.22 for 500; loading operands ahead of the stores too, 2.36 to 2.46.  At
// 128 the variants of one and two planes do not spill, those of four store 32 to 52
// bytes, those of eight 24 to 136).
// More planes hold more cells per SM (the registers of a thread grow more
// slowly than its cells) but make a longer chain per phase: the smallest L
// whose blocks fit is taken.
struct ResKind {
    int L, threads;
};
const ResKind kKinds[] = {{1, 512}, {2, 512}, {4, 512}, {8, 512}};
constexpr int kKindCount = sizeof(kKinds) / sizeof(kKinds[0]);
constexpr size_t kSmemMax = 227 * 1024;

template <int L, int MAXT>
const void* kernel_of(bool nu, bool extra) {
    if (extra)
        return nu ? reinterpret_cast<const void*>(k_resident<L, MAXT, true, true>)
                  : reinterpret_cast<const void*>(k_resident<L, MAXT, false, true>);
    return nu ? reinterpret_cast<const void*>(k_resident<L, MAXT, true, false>)
              : reinterpret_cast<const void*>(k_resident<L, MAXT, false, false>);
}
const void* kernel_of(int kind, bool nu, bool extra) {
    switch (kind) {
        case 0: return kernel_of<1, 512>(nu, extra);
        case 1: return kernel_of<2, 512>(nu, extra);
        case 2: return kernel_of<4, 512>(nu, extra);
        default: return kernel_of<8, 512>(nu, extra);
    }
}

// Microphone rows from the recorded corners (k_mic_gather's sum).
__global__ void k_resident_mics(const float* __restrict__ corners, const float* __restrict__ w, int n_mic,
                                long long total, float* __restrict__ out) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const int m = (int)(t % n_mic);
    float s = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; ++q) s = f_add(s, f_mul(w[8 * m + q], corners[8 * t + q]));
    out[t] = s;
}

}  // namespace

// Whether each plane boundary's end plane and the one inside it lie in one block.
static bool planes_fit(const SfResExtra& x, int nx, int ny, int nz, int L, int chunks, int quads, int bi,
                       int bj, int bk) {
    for (int q = 0; q < x.n_plane; ++q) {
        const int ax = x.ops[q].axis;
        const int n = ax == 0 ? nx : (ax == 1 ? ny : nz);
        if (n < 4) return false;
        const int units = ax == 0 ? chunks : (ax == 1 ? ny : quads), b = ax == 0 ? bi : (ax == 1 ? bj : bk);
        const int per = ax == 0 ? L : (ax == 1 ? 1 : 4);
        const int first = (int)((long long)units / b) * per;
        const int last = n - (int)((long long)(b - 1) * units / b) * per;
        if ((first < n ? first : n) < 2 || last < 2) return false;
    }
    return true;
}

// The cut of an nx x ny x nz grid into at most `sms` blocks, or kind < 0 when
// no kind's blocks hold it.
SfResCut sf_resident_cut(int nx, int ny, int nz, int n_probe, bool nu, int sms, const SfResExtra* x) {
    SfResCut best{};
    best.kind = -1;
    const int quads = (nz + 3) / 4;
    for (int kind = 0; kind < kKindCount && best.kind < 0; ++kind) {
        const ResKind& K = kKinds[kind];
        const int chunks = (nx + K.L - 1) / K.L;
        if ((long long)chunks * ny * quads > (long long)K.threads * sms) continue;
        long long best_cost = 0;
        for (int bi = 1; bi <= chunks && bi <= sms; ++bi)
            for (int bj = 1; bj <= ny && bi * bj <= sms; ++bj) {
                const int bk_max = sms / (bi * bj) < quads ? sms / (bi * bj) : quads;
                for (int bk = 1; bk <= bk_max; ++bk) {
                    const int nci = (chunks + bi - 1) / bi, nj = (ny + bj - 1) / bj,
                              nq = (quads + bk - 1) / bk;
                    if (x && !planes_fit(*x, nx, ny, nz, K.L, chunks, quads, bi, bj, bk)) continue;
                    const long long tiles = (long long)nci * nj * nq;
                    if (tiles > K.threads) continue;
                    // (only sides that a cut crosses have messages: 1000 x 1 x 1000 would
                    // need 93 MB of mailboxes for its y sides, which nothing is sent over)
                    int units = 0, side = 1;
                    const int split[3] = {bi, bj, bk};
                    for (int s = 0; s < 6; ++s) {
                        if (split[s >> 1] == 1) continue;
                        const int n = side_units(s, nci * K.L, nj, nq);
                        side = std::max(side, n);
                        units += n;
                    }
                    if (sf_resident_mail_bytes(bi * bj * bk, side) > kSfResMailMax) continue;
                    // the phases' cells, and the messages
                    const long long cost = (tiles + 31) / 32 * 32 * K.L + units;
                    if (best.kind >= 0 && cost >= best_cost) continue;
                    const Layout lay = layout(K.L, nci, nj, nq, n_probe, nu, x);
                    const size_t bytes = sizeof(float) * (size_t)lay.end;
                    if (bytes > kSmemMax) continue;
                    const long long need = std::max<long long>(tiles, (units + kUnits - 1) / kUnits);
                    if (need > K.threads) continue;
                    best_cost = cost;
                    best.kind = kind;
                    best.extra = x != nullptr;
                    best.bi = bi;
                    best.bj = bj;
                    best.bk = bk;
                    best.chunks = chunks;
                    best.quads = quads;
                    best.threads = (int)((need + 31) / 32 * 32);
                    best.side_max = side;
                    best.smem = bytes;
                    best.lay = lay;
                    best.units = units;
                }
            }
    }
    return best;
}

int sf_launch_resident(SfResArgs& A, const SfSources& src, const SfResCut& c, cudaStream_t st) {
    A.bi = c.bi;
    A.bj = c.bj;
    A.bk = c.bk;
    A.chunks = c.chunks;
    A.quads = c.quads;
    A.side_max = c.side_max;
    A.lay = c.lay;
    const void* k = kernel_of(c.kind, A.a.nu_cv[0] != nullptr, c.extra);
    SF_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax));
    SfSources s = src;
    void* args[] = {&A, &s};
    const cudaError_t e = cudaLaunchCooperativeKernel(k, dim3(c.bi * c.bj * c.bk), dim3(c.threads), args,
                                                      c.smem, st);
    return e == cudaSuccess ? 0 : sf_fail_cuda(e, "k_resident launch", __FILE__, __LINE__);
}

int sf_launch_resident_mics(const float* corners, const float* w, int n_mic, long long n_steps,
                            float* mic_trace, cudaStream_t st) {
    const long long total = n_steps * n_mic;
    k_resident_mics<<<(unsigned)((total + 127) / 128), 128, 0, st>>>(corners, w, n_mic, total, mic_trace);
    return cudaGetLastError() == cudaSuccess ? 0 : sf_fail("k_resident_mics launch failed");
}
