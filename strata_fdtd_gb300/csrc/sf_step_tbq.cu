// sf_step_tbq.cu -- two time steps per pass over the state, a block per window
// of rows and quads (four k cells per thread).
//
// A step of a grid larger than L2 is bound by HBM, which sees the whole state
// read and written; a pass of two steps sees it once (15 B of DRAM a cell and step
// at 200 x 256 x 256, against 33).  A block owns NR rows x NQ quads, marches planes
// along i, and outputs the rows 2 .. NR - 3 and quads 1 .. NQ - 2 of its window;
// neighbouring windows overlap by 4 rows and 2 quads, whose first step both compute,
// with the same operations (no block waits for another).  At plane t a block forms
// the first step of plane t and the second of plane t - 1:
//
//   1  faces of the first step at t (x from p of t + 1, y from the row above in shared
//      memory, z by a shuffle)
//   2  p of the first step at t; from it the x faces, p and output of the
//      second step at t - 1
//   3  y and z faces of the second step at t
//
// with a barrier after 1 and after 2: 3 and the next plane's 1 share an interval.
// The input arrives by cp.async, three planes ahead, in rings of which each thread
// copies its own quads; row r - 1's y faces and row r + 1's p come through shared
// memory, what belongs to neighbouring planes stays in registers.
//
// What bounds it are the barriers and the data path to shared memory, then HBM:
// 400^3 with walls, us a step: 420 with loads in registers one plane ahead (one block
// of 40 rows per SM), 368 in packed FP32, 333 and 320 (two blocks of 16 rows) with
// the thread's own values kept in shared memory, 327 and 304 (24 rows) with the rings,
// 277 with two blocks of 16 rows, own values in registers and the decays read ahead,
// 270 with the next plane's velocities read behind the barrier before it; the
// single-step kernel takes 332.  Three and four blocks of 16 rows 312 to 448, 32
// to 64 rows 310 to 436, 32 quads 353 to 414.
//
// The per-cell operations are those of tile4_run (sf_tile.cuh), in the same order.
// Uniform grids, nz % 4 == 0 and 16-byte aligned fields, at most 32 probes.
#include <cuda_runtime.h>

#include <climits>

#include "sf_common.cuh"
#include "sf_kernels.h"

namespace {

typedef unsigned long long u64;

// Four consecutive cells, as two pairs for the packed FP32 instructions.
struct Q4 {
    u64 a, b;
    __device__ __forceinline__ float at(int e) const {
        return e == 0 ? sf_lo(a) : (e == 1 ? sf_hi(a) : (e == 2 ? sf_lo(b) : sf_hi(b)));
    }
    static __device__ __forceinline__ float sf_lo(u64 p) { return __uint_as_float((unsigned)p); }
    static __device__ __forceinline__ float sf_hi(u64 p) { return __uint_as_float((unsigned)(p >> 32)); }
};
__device__ __forceinline__ u64 pr(float x, float y) {
    return ((u64)__float_as_uint(y) << 32) | __float_as_uint(x);
}
__device__ __forceinline__ Q4 q4(float x, float y, float z, float w) { return Q4{pr(x, y), pr(z, w)}; }
__device__ __forceinline__ Q4 zero4() { return Q4{0, 0}; }
__device__ __forceinline__ Q4 ldq(const float* f, int c) {
    const float4 t = __ldg(reinterpret_cast<const float4*>(f + c));
    return q4(t.x, t.y, t.z, t.w);
}
__device__ __forceinline__ void stq(float* f, int c, const Q4& q) {
    *reinterpret_cast<float4*>(f + c) = make_float4(q.at(0), q.at(1), q.at(2), q.at(3));
}
__device__ __forceinline__ Q4 lds4(const float4* s) {
    const float4 t = *s;
    return q4(t.x, t.y, t.z, t.w);
}
__device__ __forceinline__ void sts4(float4* s, const Q4& q) { *s = make_float4(q.at(0), q.at(1), q.at(2), q.at(3)); }

// Each lane of a packed operation rounds as the scalar one; a product is a b + (-0)
// with a -0 that the assembler cannot see (it fuses a packed mul and add into one
// rounding otherwise).
__constant__ u64 kNegZero4 = 0x8000000080000000ull;
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 sub2(u64 a, u64 b) {
    u64 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(kNegZero4));
    return r;
}
__device__ __forceinline__ Q4 operator+(const Q4& x, const Q4& y) { return {add2(x.a, y.a), add2(x.b, y.b)}; }
__device__ __forceinline__ Q4 operator-(const Q4& x, const Q4& y) { return {sub2(x.a, y.a), sub2(x.b, y.b)}; }
__device__ __forceinline__ Q4 operator*(const Q4& x, const Q4& y) { return {mul2(x.a, y.a), mul2(x.b, y.b)}; }
__device__ __forceinline__ Q4 operator*(u64 c, const Q4& y) { return {mul2(c, y.a), mul2(c, y.b)}; }

constexpr uint32_t kOpen4 = 0x01010101u * SF_ALL;

// u where the faces `bit` of the four cells are open (cells: air), else zero
__device__ __forceinline__ Q4 close4(const Q4& u, uint32_t f, uint32_t bit) {
    float v[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = f >> (8 * e) & bit ? u.at(e) : 0.0f;
    return q4(v[0], v[1], v[2], v[3]);
}

// The sources into quad (j, k .. k + 3) of plane i, in order, into air cells.
__device__ __noinline__ float4 inject4(float4 p4, const SfSources& src, unsigned smask, const double* val, int i,
                                       int j, int k, uint32_t f) {
    float p[4] = {p4.x, p4.y, p4.z, p4.w};
    for (unsigned m = smask; m != 0; m &= m - 1) {
        const int q = __ffs(m) - 1;
        const sf_source& S = src.s[q];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            bool hit;
            if (S.kind == 0) hit = i == S.a && j == S.b && k + e == S.c;
            else hit = (S.a == 0 ? i : (S.a == 1 ? j : k + e)) == S.b;
            if (hit && (f >> (8 * e) & SF_AIR)) p[e] = __double2float_rn(d_add((double)p[e], val[q]));
        }
    }
    return make_float4(p[0], p[1], p[2], p[3]);
}

__device__ __forceinline__ void copy16(float4* to, const float* from) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from)
                 : "memory");
}
__device__ __forceinline__ void copy4(unsigned* to, const uint8_t* from) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from)
                 : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Shared memory of a block: rings of p (4 planes) and of the velocities and flags (3),
// of which a thread copies its own quads; p and y faces of the first step and y faces
// of the second, of one plane.
extern __shared__ __align__(16) float4 tbq_smem[];
constexpr int tbq_bytes(int threads) { return threads * (16 * (4 + 9 + 3) + 4 * 3); }

template <bool GEOM, int NQ, int NR, int MINB>
__global__ void __launch_bounds__(NQ* NR, MINB) k_step_tbq(SfStepArgs a, SfSources src, int ich, float* trace1) {
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int NT = NQ * NR;
    const int tid = threadIdx.x, q = tid % NQ, r = tid / NQ;
    const int nx = a.nx, ny = a.ny, nz = a.nz;
    const int j = (int)blockIdx.y * (NR - 4) - 2 + r, k = (int)blockIdx.x * (4 * NQ - 8) - 4 + 4 * q;
    const int chunk = a.reverse ? (int)(gridDim.z - 1 - blockIdx.z) : (int)blockIdx.z;
    const int i0 = chunk * ich, i1 = min(i0 + ich, nx);
    if (a.trace_prev != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0)
        for (int t = tid; t < a.n_probe; t += NQ * NR) a.trace_prev[t] = a.p[a.probe_cells[t]];
    const bool in = j >= 0 && j < ny && k >= 0 && k < nz;
    const bool mine = in && r >= 2 && r < NR - 2 && q >= 1 && q < NQ - 1;
    // a quad past the grid reads the nearest one of the grid: nothing that is kept
    // depends on it (the faces at the low ends are set to zero where they are used)
    const int jc = min(max(j, 0), ny - 1), kc = min(max(k, 0), nz - 4);
    const bool jf = j < ny - 1, last_k = k + 4 >= nz;
    // faces of an axis' last plane carry no update: they are not closed either
    const uint32_t kept = (jf ? 0u : 0x01010101u * SF_OPY) | (last_k ? (uint32_t)SF_OPZ << 24 : 0u);
    const u64 cv = pr(a.cv, a.cv), cp = pr(a.cp, a.cp);
    const u64 dj = pr(a.dy[jc], a.dy[jc]);
    const Q4 dk = ldq(a.dz, kc);
    const int plane = ny * nz, at = jc * nz + kc;

    // sources that reach the window's planes i0 - 1 .. i1, probes in this quad
    // (hot: the plane in which they act, as a call at every plane made their blocks the
    // last of a wave: 300^3 in one wave 168 us a step against 109)
    constexpr int kNever = -1, kEvery = -2;
    unsigned smask = 0;
    int hot = kNever;
    for (int s = 0; s < src.n; ++s) {
        const sf_source& S = src.s[s];
        bool can;
        if (S.kind == 0)
            can = S.a >= i0 - 1 && S.a <= i1 && S.b == j && S.c >= k && S.c < k + 4;
        else if (S.a == 0) can = S.b >= i0 - 1 && S.b <= i1;
        else if (S.a == 1) can = S.b == j;
        else can = S.b >= k && S.b < k + 4;
        if (!can || !in) continue;
        smask |= 1u << s;
        const int at_plane = S.kind == 0 ? S.a : (S.a == 0 ? S.b : kEvery);
        hot = hot == kNever || hot == at_plane ? at_plane : kEvery;
    }
    const double* val1 = a.src_val;
    const double* val2 = a.src_val != nullptr ? a.src_val + src.n : nullptr;
    unsigned pmask = 0;
    if (trace1 != nullptr && mine)
        for (int t = 0; t < a.n_probe; ++t) {
            const int c = (int)a.probe_cells[t], w = c % plane;
            if (c >= i0 * plane && c < i1 * plane && w >= at && w < at + 4) pmask |= 1u << t;
        }

    auto flags4 = [&](int c) -> uint32_t {
        return GEOM ? __ldg(reinterpret_cast<const unsigned*>(a.flags + c)) : kOpen4;
    };
    auto face = [&](const Q4& u, const Q4& hi, const Q4& lo) { return u + cv * (hi - lo); };
    // z faces of a quad: the cell above the last one by a shuffle
    auto zface = [&](const Q4& u, const Q4& p) -> Q4 {
        const float up = __shfl_down_sync(kAll, p.at(0), 1, NQ);
        Q4 o = face(u, q4(p.at(1), p.at(2), p.at(3), up), p);
        if (last_k) o.b = pr(o.at(2), u.at(3));
        return o;
    };
    auto inject = [&](const Q4& p, const double* val, int i, uint32_t f) -> Q4 {
        const float4 o = inject4(make_float4(p.at(0), p.at(1), p.at(2), p.at(3)), src, smask, val, i, j, k, f);
        return q4(o.x, o.y, o.z, o.w);
    };
    // p + cp (d/dx + d/dy + d/dz), z faces with the one below the quad by a shuffle
    auto pressure = [&](const Q4& p, const Q4& xh, const Q4& xl, const Q4& yh, const float4* ylow, const Q4& zh) {
        const Q4 yl = j <= 0 || r == 0 ? zero4() : lds4(ylow);
        float zl = __shfl_up_sync(kAll, zh.at(3), 1, NQ);
        if (k == 0) zl = 0.0f;
        return p + cp * (((xh - xl) + (yh - yl)) + (zh - q4(zl, zh.at(0), zh.at(1), zh.at(2))));
    };

    float4* const r_p = tbq_smem + tid;  // (rows past the last one read what follows: unused)
    float4* const r_v = r_p + 4 * NT;
    float4* const s_p1 = r_v + 9 * NT;
    float4* const s_y1 = s_p1 + NT;
    float4* const s_y2 = s_y1 + NT;
    unsigned* const r_f = reinterpret_cast<unsigned*>(tbq_smem + 16 * NT) + tid;
    const int ts = i0 > 0 ? i0 - 1 : 0;
    int c = ts * plane + at;
    // p of plane t + d, velocities and flags of plane t + d, at c + d plane
    auto fetch_p = [&](int t, int d, int slot) {
        if (t + d < nx && t + d <= i1 + 1) copy16(r_p + slot * NT, a.p + c + d * plane);
    };
    auto fetch_v = [&](int t, int d, int slot) {
        if (t + d >= nx || t + d > i1) return;
        const int at_d = c + d * plane;
        copy16(r_v + (3 * slot) * NT, a.vx + at_d);
        copy16(r_v + (3 * slot + 1) * NT, a.vy + at_d);
        copy16(r_v + (3 * slot + 2) * NT, a.vz + at_d);
        if (GEOM) copy4(r_f + slot * NT, a.flags + at_d);
    };
    fetch_p(ts, 0, 0);
    for (int d = 0; d < 3; ++d) {  // plane t's velocities and plane t + 1's p: the group of iteration t - 3
        fetch_v(ts, d, d);
        fetch_p(ts, d + 1, d + 1);
        copies_commit();
    }
    uint32_t Fm = kOpen4;
    Q4 u1x = zero4();  // x faces of the first step at t - 1
    if (ts > 0) {
        u1x = face(ldq(a.vx, c - plane), ldq(a.p, c), ldq(a.p, c - plane));
        if (GEOM) u1x = close4(u1x, flags4(c - plane), SF_OPX);
    }
    Q4 p1m = zero4(), u2x = zero4(), u2y = zero4(), u2z = zero4(), Pn = zero4();
    float d_prev = 1.0f, d_t = a.dx[ts];
    bool wallm = false;
    int sp = 0, sv = 0;  // this plane's places in the rings
    copies_wait<2>();
    __syncthreads();
    Q4 P = lds4(r_p);
    // with registers to spare, a plane's velocities are read behind the barrier before it
    constexpr bool AHEAD = NT * MINB <= 512;
    Q4 nx1 = lds4(r_v), ny1 = lds4(r_v + NT), nz1 = lds4(r_v + 2 * NT);

    for (int t = ts; t <= i1; ++t, c += plane) {
        const bool first = t < nx;
        // ---- 1
        Q4 x1, y1, z1, p1;
        const float d_next = a.dx[min(t + 1, nx - 1)];  // (its wait lies in the next plane)
        uint32_t Ft = kOpen4;
        bool walls = false;
        if (first) {
            const float4* const s_p0 = r_p + sp * NT;
            const float4* const s_v = r_v + 3 * sv * NT;
            x1 = AHEAD ? nx1 : lds4(s_v);
            if (t < nx - 1) {
                Pn = lds4(r_p + (sp + 1 & 3) * NT);
                x1 = face(x1, Pn, P);
            }
            y1 = AHEAD ? ny1 : lds4(s_v + NT);
            if (jf) y1 = face(y1, lds4(s_p0 + NQ), P);
            z1 = zface(AHEAD ? nz1 : lds4(s_v + 2 * NT), P);
            if (GEOM) Ft = r_f[sv * NT] | kept | (t == nx - 1 ? 0x01010101u * SF_OPX : 0u);
            walls = GEOM && __any_sync(kAll, Ft != kOpen4);
            if (walls) {
                x1 = close4(x1, Ft, SF_OPX);
                y1 = close4(y1, Ft, SF_OPY);
                z1 = close4(z1, Ft, SF_OPZ);
            }
            sts4(s_y1, y1);
        }
        fetch_v(t, 3, sv);
        __syncthreads();
        // ---- 2
        if (first) {
            p1 = pressure(P, x1, u1x, y1, s_y1 - NQ, z1);
            if (walls) p1 = close4(p1, Ft, SF_AIR);
            p1 = dk * (dj * (pr(d_t, d_t) * p1));
            if (hot == t || hot == kEvery) p1 = inject(p1, val1, t, Ft);
            sts4(s_p1, p1);
            for (unsigned m = pmask; m != 0; m &= m - 1) {
                const int s = __ffs(m) - 1, w = (int)a.probe_cells[s] - c;
                if (w >= 0 && w < 4) trace1[s] = p1.at(w);
            }
        }
        if (t > ts) {
            const u64 dm = pr(d_prev, d_prev);
            Q4 x2 = dm * u1x;
            if (t < nx) x2 = face(x2, p1, p1m);
            if (wallm) x2 = close4(x2, Fm, SF_OPX);
            if (t > i0) {
                Q4 p2 = pressure(p1m, x2, u2x, u2y, s_y2 - NQ, u2z);
                if (wallm) p2 = close4(p2, Fm, SF_AIR);
                p2 = dk * (dj * (dm * p2));
                if (hot == t - 1 || hot == kEvery) p2 = inject(p2, val2, t - 1, Fm);
                if (mine) {
                    stq(a.po, c - plane, p2);
                    stq(a.vxo, c - plane, dm * x2);
                    stq(a.vyo, c - plane, dj * u2y);
                    stq(a.vzo, c - plane, dk * u2z);
                }
            }
            u2x = x2;
        }
        fetch_p(t, 4, sp);
        copies_commit();
        __syncthreads();
        // ---- 3
        copies_wait<2>();
        sp = sp + 1 & 3;
        sv = sv == 2 ? 0 : sv + 1;
        if (AHEAD) {
            const float4* const s_v = r_v + 3 * sv * NT;
            nx1 = lds4(s_v);
            ny1 = lds4(s_v + NT);
            nz1 = lds4(s_v + 2 * NT);
        }
        if (first) {
            u2y = dj * y1;
            if (jf) u2y = face(u2y, lds4(s_p1 + NQ), p1);
            u2z = zface(dk * z1, p1);
            if (walls) {
                u2y = close4(u2y, Ft, SF_OPY);
                u2z = close4(u2z, Ft, SF_OPZ);
            }
            sts4(s_y2, u2y);
            p1m = p1;
            P = Pn;
            u1x = x1;
            Fm = Ft;
            wallm = walls;
        }
        d_prev = d_t;
        d_t = d_next;
    }
}

template <int NQ, int NR, int MINB>
int launch_tbq(const SfStepArgs& a, const SfSources& src, bool geom, int ich, float* trace1, cudaStream_t st) {
    const dim3 grid((a.nz + 4 * NQ - 9) / (4 * NQ - 8), (a.ny + NR - 5) / (NR - 4), (a.nx + ich - 1) / ich);
    auto kernel = geom ? k_step_tbq<true, NQ, NR, MINB> : k_step_tbq<false, NQ, NR, MINB>;
    SF_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, tbq_bytes(NQ * NR)));
    kernel<<<grid, NQ * NR, tbq_bytes(NQ * NR), st>>>(a, src, ich, trace1);
    return cudaGetLastError() == cudaSuccess ? 0 : sf_fail("k_step_tbq launch failed");
}

}  // namespace

// Windows of 16 or 20 rows x 16 quads, two blocks per SM.
int sf_launch_step_tbq(const SfStepArgs& a, const SfSources& src, bool geom, int rows, int ich, float* trace1,
                       cudaStream_t st) {
    if (ich < 1) ich = 1;
    if (rows == 20) return launch_tbq<16, 20, 2>(a, src, geom, ich, trace1, st);
    return launch_tbq<16, 16, 2>(a, src, geom, ich, trace1, st);
}
