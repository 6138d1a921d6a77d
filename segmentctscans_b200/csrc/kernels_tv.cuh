// TV-L2 (ROF) denoising by Chambolle's projection algorithm on the cylinder
// (totalvarmin/chambolle.cpp:33-218): the next row of the reference's scope
// table after the Potts solve, on the same layout and neighbour tables.
// State: xi (3 planes) and v (1 plane) laid out like g (the mapping's stride).
// Arithmetic as in the reference's clang build: a multiply and an add are
// fused for the sum of squares, 1 + tau |G|, xi + tau G and g - lambda d; the
// rest are IEEE single operations in source order (the library is compiled
// with -fmad=false).
#pragma once

#include <cuda.h>

#include <cstdint>

#include "block.cuh"
#include "geometry.cuh"
#include "kernels_plain.cuh"
#include "tma.cuh"
#include "voxel.cuh"

namespace potts {

// div_kernel (:33-87): d = -xi_n(x-e_n) + xi_n(x) - xi_r(x-e_r) + xi_r(x) - xi_c(x-e_c) + xi_c(x),
// each term only where that neighbour exists, in this order.
__device__ __forceinline__ float tv_div_at(const Geometry &g, const float *__restrict__ xi, int64_t o, int n,
                                           const LineInfo &li)
{
    const float *x0 = xi, *x1 = xi + g.plane_w, *x2 = xi + 2 * g.plane_w;
    float d = 0.0f;
    if (n > 0) d -= x0[o - 1];
    if (n + 1 < g.ns) d += x0[o];
    if (li.flags & kHasPrevRow) d -= x1[o - g.nstride_w];
    if (li.flags & kHasNextRow) d += x1[o];
    if (li.prev_col >= 0) d -= x2[(int64_t)li.prev_col * g.nstride_w + n];
    if (li.next_col >= 0) d += x2[o];
    return d;
}

__global__ void __launch_bounds__(kPlainThreads) tv_div_kernel(Geometry g, const float *__restrict__ xi,
                                                               float *__restrict__ v)
{
    const PlainIndex p = plain_index(g, 0, g.ns);
    if (!p.valid) return;
    const LineInfo li = load_line(g, p.line);
    const int64_t o = p.line * g.nstride_w + p.n;
    v[o] = tv_div_at(g, xi, o, p.n, li);
}

// grad_kernel (:89-166): G = grad+ v - (grad+ g) / lambda, xi <- (xi + tau G) / (1 + tau |G|),
// max |dxi|^2 into *dq.
__global__ void __launch_bounds__(kPlainThreads) tv_grad_kernel(Geometry g, const float *__restrict__ gin,
                                                                float *__restrict__ xi, const float *__restrict__ v,
                                                                float lam, float tau, float *dq)
{
    const PlainIndex p = plain_index(g, 0, g.ns);
    float d = 0.0f;
    if (p.valid) {
        const LineInfo li = load_line(g, p.line);
        const int64_t o = p.line * g.nstride_w + p.n;
        float g1 = 0.0f, g2 = 0.0f, g3 = 0.0f;
        if (p.n + 1 < g.ns) g1 = (v[o + 1] - v[o]) - __fdiv_rn(gin[o + 1] - gin[o], lam);
        if (li.flags & kHasNextRow) {
            const int64_t q = o + g.nstride_w;
            g2 = (v[q] - v[o]) - __fdiv_rn(gin[q] - gin[o], lam);
        }
        if (li.next_col >= 0) {
            const int64_t q = (int64_t)li.next_col * g.nstride_w + p.n;
            g3 = (v[q] - v[o]) - __fdiv_rn(gin[q] - gin[o], lam);
        }
        float s = g1 * g1;
        s = fmaf(g2, g2, s);
        s = fmaf(g3, g3, s);
        const float denom = fmaf(tau, __fsqrt_rn(s), 1.0f);
        float *x0 = xi + o, *x1 = xi + g.plane_w + o, *x2 = xi + 2 * g.plane_w + o;
        const float q1 = __fdiv_rn(fmaf(tau, g1, *x0), denom);
        const float q2 = __fdiv_rn(fmaf(tau, g2, *x1), denom);
        const float q3 = __fdiv_rn(fmaf(tau, g3, *x2), denom);
        const float e1 = *x0 - q1, e2 = *x1 - q2, e3 = *x2 - q3;
        d = e1 * e1;
        d = fmaf(e2, e2, d);
        d = fmaf(e3, e3, d);
        *x0 = q1;
        *x1 = q2;
        *x2 = q3;
    }
    if (dq) block_max_to(d, dq);
}

// One fused iteration: the div and grad kernels in one launch.  Each thread
// rebuilds v = div xi at its voxel and at the three forward neighbours from
// xi_in (neighbour reads are L1/L2 hits), so v is never stored, and writes
// xi_out (ping-pong: other threads still read xi_in).  Same operations in the
// same order as tv_div_kernel + tv_grad_kernel, so the same bits; DRAM traffic
// xi in (3) + g (1) + xi out (3) = 28 B per voxel instead of 48 B.
__global__ void __launch_bounds__(kPlainThreads) tv_fused_kernel(Geometry g, const float *__restrict__ gin,
                                                                 const float *__restrict__ xi_in,
                                                                 float *__restrict__ xi_out, float lam, float tau,
                                                                 float *dq)
{
    const PlainIndex p = plain_index(g, 0, g.ns);
    float d = 0.0f;
    if (p.valid) {
        const LineInfo li = load_line(g, p.line);
        const int64_t o = p.line * g.nstride_w + p.n;
        const float v0 = tv_div_at(g, xi_in, o, p.n, li);
        float g1 = 0.0f, g2 = 0.0f, g3 = 0.0f;
        if (p.n + 1 < g.ns) {
            const float vn = tv_div_at(g, xi_in, o + 1, p.n + 1, li);
            g1 = (vn - v0) - __fdiv_rn(gin[o + 1] - gin[o], lam);
        }
        if (li.flags & kHasNextRow) {
            const int64_t q = o + g.nstride_w;
            const float vr = tv_div_at(g, xi_in, q, p.n, load_line(g, p.line + 1));
            g2 = (vr - v0) - __fdiv_rn(gin[q] - gin[o], lam);
        }
        if (li.next_col >= 0) {
            const int64_t q = (int64_t)li.next_col * g.nstride_w + p.n;
            const float vc = tv_div_at(g, xi_in, q, p.n, load_line(g, li.next_col));
            g3 = (vc - v0) - __fdiv_rn(gin[q] - gin[o], lam);
        }
        float s = g1 * g1;
        s = fmaf(g2, g2, s);
        s = fmaf(g3, g3, s);
        const float denom = fmaf(tau, __fsqrt_rn(s), 1.0f);
        const float x0 = xi_in[o], x1 = xi_in[g.plane_w + o], x2 = xi_in[2 * g.plane_w + o];
        const float q1 = __fdiv_rn(fmaf(tau, g1, x0), denom);
        const float q2 = __fdiv_rn(fmaf(tau, g2, x1), denom);
        const float q3 = __fdiv_rn(fmaf(tau, g3, x2), denom);
        const float e1 = x0 - q1, e2 = x1 - q2, e3 = x2 - q3;
        d = e1 * e1;
        d = fmaf(e2, e2, d);
        d = fmaf(e3, e3, d);
        xi_out[o] = q1;
        xi_out[g.plane_w + o] = q2;
        xi_out[2 * g.plane_w + o] = q3;
    }
    if (dq) block_max_to(d, dq);
}

// update_kernel (:168-218): g <- g - lambda div xi.
__global__ void __launch_bounds__(kPlainThreads) tv_update_kernel(Geometry g, float *__restrict__ gio,
                                                                  const float *__restrict__ xi, float lam)
{
    const PlainIndex p = plain_index(g, 0, g.ns);
    if (!p.valid) return;
    const LineInfo li = load_line(g, p.line);
    const int64_t o = p.line * g.nstride_w + p.n;
    gio[o] = fmaf(-lam, tv_div_at(g, xi, o, p.n, li), gio[o]);
}

// Whether every forward difference of g is 0 or between 2^-60 and 2^60 in size (*unsafe is set
// where one is not): the quotients by lambda then come from its reciprocal (div4_rn).
__global__ void __launch_bounds__(kPlainThreads) tv_range_kernel(Geometry g, const float *__restrict__ gin,
                                                                 int *__restrict__ unsafe)
{
    const PlainIndex p = plain_index(g, 0, g.ns);
    if (!p.valid) return;
    const LineInfo li = load_line(g, p.line);
    const int64_t o = p.line * g.nstride_w + p.n;
    const float g0 = gin[o];
    float d1 = 0.0f, d2 = 0.0f, d3 = 0.0f;
    if (p.n + 1 < g.ns) d1 = gin[o + 1] - g0;
    if (li.flags & kHasNextRow) d2 = gin[o + g.nstride_w] - g0;
    if (li.next_col >= 0) d3 = gin[(int64_t)li.next_col * g.nstride_w + p.n] - g0;
    if (!none_below_2m60(d1, d2, d3) || !(fabsf(d1) <= 0x1p60f) || !(fabsf(d2) <= 0x1p60f) ||
        !(fabsf(d3) <= 0x1p60f))
        *unsafe = 1;
}

// Tiled fused iteration.  A block owns a tile of 8 rows x 128 slices and marches
// over the columns [ca, cb) of its work item (x = first row, y = first slice,
// z/w = column range).  Warp w < 8 owns row r0 + w and each of its lanes four
// consecutive slices, so every condition on rows and columns is the same in a
// whole warp and shared memory is read 16 bytes at a time; warp 8 computes what
// the tile needs of v = div xi on row r0 + 8 and at slice n0 + 128.  Shared
// memory holds a ring of three column planes of xi (rows r0-1 .. r0+8, slices
// n0-4 .. n0+131, the three components), each one TMA box, and two planes of v,
// from which a warp reads the row below; v of a lane's own voxels at the planes c
// and c+1, and g at c, c+1 and on the row below, stay in its registers (g is
// loaded a plane ahead).  One barrier per plane.  The operations per voxel are
// those of tv_div_at and tv_grad_kernel, in the same order and with the same
// rounding: two slices at a time with the paired instructions, quotients by one
// divisor from its reciprocal where the remainders are exact (for lambda and the
// differences of g that is known before the first iteration).  Box rows outside the plane's column come from other columns or are
// zero-filled; their values are never used.
// HBM traffic per voxel and iteration: xi in and out, g in (28 bytes; three planes
// of precomputed differences of g / lambda in place of g cost 36).  At 512 x 512 x
// 512 (radius 246) an iteration takes 0.61 ms (4.5 TB/s; 0.79 ms with one slice and
// four rows per thread, scalar arithmetic and the difference planes): 4.0 warp
// instructions per voxel at 59 % of the issue slots.  Two blocks of 96 registers
// per multiprocessor: with three (72 registers) it spills, 0.75 ms.
struct TvTile {
    static constexpr int TR = 8, TN = 128, SLOTS = 3;
    static constexpr int XR = TR + 2, XS = TN + 8;  // xi box: rows r0-1 .., row stride (slice n at n - n0 + 4)
    static constexpr int VR = TR + 1, VS = TN + 4;  // v plane: rows r0 .., row stride (slice n at n - n0)
    static constexpr int XC = XR * XS;              // one xi component
    static constexpr int XI_PLANE = 3 * XC;
    static constexpr int XI_SLOT = (XI_PLANE + 31) / 32 * 32;  // 128-byte aligned slots
    static constexpr int V_PLANE = VR * VS;
    static constexpr uint32_t BOX_BYTES = 4u * XI_PLANE;
    static constexpr int OFF_BAR = 4 * (SLOTS * XI_SLOT + 2 * V_PLANE);  // bytes: mbarriers, abort flag
    static constexpr int SMEM_BYTES = OFF_BAR + SLOTS * 8 + 8 + 128;     // + alignment slack
};
constexpr int kTvThreads = 32 * (TvTile::TR + 1);
constexpr int kTvBlocks = 2;  // per multiprocessor

// column table entry: x = first line, y/z = row range of the column (the Potts kernel's table)
__device__ __forceinline__ bool tv_row_in(int4 ci, int row) { return row >= ci.y && row < ci.z; }

// Four values as two pairs.
struct Quad {
    float2 a, b;
};
__device__ __forceinline__ Quad quad(float4 v) { return Quad{f2(v.x, v.y), f2(v.z, v.w)}; }
__device__ __forceinline__ Quad lds4(const float *p) { return quad(*reinterpret_cast<const float4 *>(p)); }
__device__ __forceinline__ Quad zero4() { return Quad{f2(0.0f), f2(0.0f)}; }
__device__ __forceinline__ Quad add4(Quad x, Quad y) { return Quad{add2(x.a, y.a), add2(x.b, y.b)}; }
__device__ __forceinline__ Quad sub4(Quad x, Quad y) { return Quad{sub2(x.a, y.a), sub2(x.b, y.b)}; }
// x with the elements j where m has no bit j set to 0
__device__ __forceinline__ Quad keep4(Quad x, unsigned m)
{
    return Quad{f2(m & 1u ? x.a.x : 0.0f, m & 2u ? x.a.y : 0.0f), f2(m & 4u ? x.b.x : 0.0f, m & 8u ? x.b.y : 0.0f)};
}
// x / b, correctly rounded, from the correctly rounded reciprocal r of b (in_range: 2^-20 <= |b| <=
// 2^20 and x is 0 or between 2^-60 and 2^60 in size, see shrink_rn)
__device__ __forceinline__ Quad div4_rn(Quad x, float b, float r, bool in_range)
{
    if (in_range) return Quad{quot2_rn(x.a, f2(-b), f2(r)), quot2_rn(x.b, f2(-b), f2(r))};
    return Quad{f2(__fdiv_rn(x.a.x, b), __fdiv_rn(x.a.y, b)), f2(__fdiv_rn(x.b.x, b), __fdiv_rn(x.b.y, b))};
}

__device__ __forceinline__ float rcp_1ulp(float b)  // 1 / b, b normal
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
    return r;
}

// xi <- (xi + tau G) / (1 + tau |G|) for four voxels; returns |dxi|^2 of each.  With 0 <= tau <= 1
// (tau_in_range), |G|^2 <= 2^40 (which a NaN is not) and no tiny numerators the root and the quotients
// are those of shrink_rn: |G|^2 below 2^-80 gives a denominator of 1 whatever its root, so it is raised
// to that.  Else the IEEE operations run (the same bits).
__device__ __forceinline__ uint32_t below_key(float2 a)  // none_below_2m60's key of two values
{
    const uint32_t x = __float_as_uint(a.x), y = __float_as_uint(a.y);
    return min(x + x - 1u, y + y - 1u);
}
__device__ __forceinline__ Quad tv_step(Quad (&x)[3], const Quad (&G)[3], float tau, bool tau_in_range)
{
    const float2 t = f2(tau);
    float2 s[2], a[2][3], q[2][3], d[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const float2 g0 = h ? G[0].b : G[0].a, g1 = h ? G[1].b : G[1].a, g2 = h ? G[2].b : G[2].a;
        s[h] = fma2(g2, g2, fma2(g1, g1, mul2(g0, g0)));
        a[h][0] = fma2(t, g0, h ? x[0].b : x[0].a);
        a[h][1] = fma2(t, g1, h ? x[1].b : x[1].a);
        a[h][2] = fma2(t, g2, h ? x[2].b : x[2].a);
    }
    const uint32_t key = min(min(min(below_key(a[0][0]), below_key(a[0][1])), min(below_key(a[0][2]), below_key(a[1][0]))),
                             min(below_key(a[1][1]), below_key(a[1][2])));
    const float2 sum = add2(s[0], s[1]);  // not below any of the four; a NaN or infinite one makes it so
    if (tau_in_range && sum.x + sum.y <= 0x1p40f && key >= (67u << 24) - 1u) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float2 mz;
            const float2 l = root2_rn(f2(fmaxf(s[h].x, 0x1p-80f), fmaxf(s[h].y, 0x1p-80f)), mz);
            const float2 md = fma2(f2(-tau), l, f2(-1.0f));  // -(1 + tau |G|)
            const float2 r = rcp2_step(md, f2(rcp_1ulp(-md.x), rcp_1ulp(-md.y)));
#pragma unroll
            for (int k = 0; k < 3; ++k) q[h][k] = quot2_rn(a[h][k], md, r);
        }
    } else {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float dx = fmaf(tau, __fsqrt_rn(s[h].x), 1.0f), dy = fmaf(tau, __fsqrt_rn(s[h].y), 1.0f);
#pragma unroll
            for (int k = 0; k < 3; ++k) q[h][k] = f2(__fdiv_rn(a[h][k].x, dx), __fdiv_rn(a[h][k].y, dy));
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const float2 e0 = sub2(h ? x[0].b : x[0].a, q[h][0]), e1 = sub2(h ? x[1].b : x[1].a, q[h][1]),
                     e2 = sub2(h ? x[2].b : x[2].a, q[h][2]);
        d[h] = fma2(e2, e2, fma2(e1, e1, mul2(e0, e0)));
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) x[k] = Quad{q[0][k], q[1][k]};
    return Quad{d[0], d[1]};
}

// rlam = RN(1 / lam); lam_in_range: 2^-20 <= |lam| <= 2^20; tau_in_range: 0 <= tau <= 1.  kVecG: g is 16-byte aligned.  Every
// wait on a load is bounded; a block whose wait gives up sets *err, drains its loads in flight
// (bounded) and stops.
template <bool kVecG>
__global__ void __launch_bounds__(kTvThreads, kTvBlocks)
    tv_tiled_kernel(Geometry g, const int4 *__restrict__ cols, int col_begin, int col_end,
                    const int4 *__restrict__ work, const __grid_constant__ CUtensorMap xi_map,
                    const float *__restrict__ gin, float *__restrict__ xi_out, float lam, float rlam, int lam_in_range,
                    const int *__restrict__ unsafe, float tau, int tau_in_range, float *dq, int *err)
{
    using T = TvTile;
    extern __shared__ __align__(128) uint8_t tv_raw[];
    // align to 128 bytes by pointer arithmetic on the shared array itself
    uint8_t *const base = tv_raw + ((128u - (smem_addr(tv_raw) & 127u)) & 127u);
    float *const smf = reinterpret_cast<float *>(base);
    uint64_t *const bar = reinterpret_cast<uint64_t *>(base + T::OFF_BAR);
    volatile int *const abort = reinterpret_cast<volatile int *>(base + T::OFF_BAR + T::SLOTS * 8);
    auto sx = [&](int sl) { return smf + sl * T::XI_SLOT; };
    auto sv = [&](int sl) { return smf + T::SLOTS * T::XI_SLOT + sl * T::V_PLANE; };
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    const int4 wk = work[blockIdx.x];
    const int r0 = wk.x, n0 = wk.y, ca = wk.z, cb = wk.w;
    const int row = r0 + w, nq = n0 + 4 * lane;
    const bool rcp_lam = lam_in_range && __ldg(unsafe) == 0;
    auto col_at = [&](int c) { return (c >= col_begin && c < col_end) ? __ldg(cols + c) : make_int4(0, 0, 0, 0); };
    // bit j: slice nq + j is in the field, has a next slice.  Values of other slices are computed but
    // reach no voxel: v at the first slice past the end is read only under fwd.
    unsigned in = 0, fwd = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        in |= (nq + j < g.ns ? 1u : 0u) << j;
        fwd |= (nq + j + 1 < g.ns ? 1u : 0u) << j;
    }
    // clears the elements without a next slice: in a tile that ends before the field does there are
    // none, and with whole quads of slices only a last element can be one
    const bool inner = n0 + T::TN < g.ns, quads = (g.ns & 3) == 0;
    auto mask_fwd = [&](Quad &x) {
        if (inner) return;
        if (quads)
            x.b.y = fwd & 8u ? x.b.y : 0.0f;
        else
            x = keep4(x, fwd);
    };

    if (t == 0) {
        for (int k = 0; k < T::SLOTS; ++k) mbar_init(bar + k, 1);
        *abort = 0;
        mbar_fence_init();
        tma_prefetch_desc(&xi_map);
    }
    __syncthreads();
    uint32_t phase = 0, pending = 0;  // per slot: parity of the next wait, load in flight (thread 0's view)
    auto issue = [&](int c, int slot) {  // plane c's xi box; thread 0 only
        const int4 ci = col_at(c);
        mbar_arrive_expect_tx(bar + slot, T::BOX_BYTES);
        tma_load_3d(sx(slot), &xi_map, bar + slot, n0 - 4, ci.x - ci.y + r0 - 1, 0);
        pending |= 1u << slot;
    };
    auto wait_slot = [&](int slot) {  // warp-uniform; a wait that gives up sets *abort
        if (mbar_wait_warp(bar + slot, (phase >> slot) & 1u, abort)) {
            phase ^= 1u << slot;
            pending &= ~(1u << slot);
        }
    };
    // offset of the lane's first voxel on the plane with entry ci
    auto offset = [&](int4 ci) { return ((int64_t)ci.x + (row - ci.y)) * g.nstride_w + nq; };
    // the lane's g at offset o (0 where there is none) and its slice n0+128 (lane 31)
    auto load_g = [&](bool there, int64_t o) {
        if (w == T::TR || !there || in == 0u) return zero4();
        const float *p = gin + o;
        if constexpr (kVecG) return quad(__ldg(reinterpret_cast<const float4 *>(p)));
        return Quad{f2(__ldg(p), __ldg(p + 1)), f2(__ldg(p + 2), __ldg(p + 3))};
    };
    const bool edge_lane = lane == 31 && nq + 4 < g.ns && w < T::TR;
    auto load_edge = [&](bool there, int64_t o) { return edge_lane && there ? __ldg(gin + o + 4) : 0.0f; };
    // v = div xi of the lane's voxels on the plane with entry ci (xi box X), previous plane cp (xi box
    // Xp), next cn; stored to V (warp 8: also slice n0+128 of the tile's rows)
    auto divergence = [&](int4 ci, int4 cp, int4 cn, const float *X, const float *Xp, float *V) {
        const float *s0 = X, *s1 = X + T::XC, *s2 = X + 2 * T::XC, *s2p = Xp + 2 * T::XC;
        Quad d = zero4();
        if (tv_row_in(ci, row)) {  // warp-uniform, as all conditions on rows and columns
            const int b = (w + 1) * T::XS + 4 * lane + 4;
            Quad a0 = lds4(s0 + b);
            float prev = __shfl_up_sync(0xffffffffu, a0.b.y, 1);
            if (lane == 0) prev = n0 > 0 ? s0[b - 1] : 0.0f;
            const Quad a0m{f2(prev, a0.a.x), f2(a0.a.y, a0.b.x)};
            mask_fwd(a0);
            d = add4(sub4(d, a0m), a0);
            if (row > ci.y) d = sub4(d, lds4(s1 + b - T::XS));
            if (row + 1 < ci.z) d = add4(d, lds4(s1 + b));
            if (tv_row_in(cp, row)) d = sub4(d, lds4(s2p + b));
            if (tv_row_in(cn, row)) d = add4(d, lds4(s2 + b));
        }
        *reinterpret_cast<float4 *>(V + w * T::VS + 4 * lane) = make_float4(d.a.x, d.a.y, d.b.x, d.b.y);
        if (w == T::TR && lane < T::TR) {  // slice n0+TN of row r0 + lane
            const int rw = r0 + lane, ne = n0 + T::TN, b = (lane + 1) * T::XS + T::TN + 4;
            float e = 0.0f;
            if (tv_row_in(ci, rw) && ne < g.ns) {
                e -= s0[b - 1];
                if (ne + 1 < g.ns) e += s0[b];
                if (rw > ci.y) e -= s1[b - T::XS];
                if (rw + 1 < ci.z) e += s1[b];
                if (tv_row_in(cp, rw)) e -= s2p[b];
                if (tv_row_in(cn, rw)) e += s2[b];
            }
            V[lane * T::VS + T::TN] = e;
        }
        return d;
    };

    // planes ca-1, ca, ca+1 into slots 0, 1, 2 (plane c sits in slot (c - ca + 1) mod 3; plane c+2 is
    // issued when plane c-1 is done with)
    if (t == 0)
        for (int k = 0; k < T::SLOTS; ++k)
            if (ca - 1 + k <= cb) issue(ca - 1 + k, k);
    int4 ci = col_at(ca), cn = col_at(ca + 1);
    int64_t oc = offset(ci), on = offset(cn);
    Quad gc = load_g(tv_row_in(ci, row), oc), gn = load_g(tv_row_in(cn, row), on);
    Quad gd = load_g(tv_row_in(ci, row + 1), oc + g.nstride_w);
    float ge = load_edge(tv_row_in(ci, row), oc), gne = load_edge(tv_row_in(cn, row), on);
    wait_slot(0);
    wait_slot(1);
    Quad v = divergence(ci, col_at(ca - 1), cn, sx(1), sx(0), sv(0));
    __syncthreads();
    if (t == 0 && ca + 2 <= cb) issue(ca + 2, 0);
    float dmax = 0.0f;
    int sc = 1, sn = 2;  // slots of planes c, c+1
    int vc = 0;          // v slot of plane c
#pragma unroll 1
    for (int c = ca; c < cb; ++c) {
        const int4 c2 = col_at(c + 2);
        // g of the next two planes, in flight during this one
        const int64_t o2 = offset(c2);
        const bool there2 = c + 2 <= cb && tv_row_in(c2, row);
        const Quad g2 = load_g(there2, o2), gd1 = load_g(tv_row_in(cn, row + 1), on + g.nstride_w);
        const float g2e = load_edge(there2, o2);
        wait_slot(sn);  // plane c+1
        const Quad vn = divergence(cn, ci, c2, sx(sn), sx(sc), sv(vc ^ 1));
        // the next slice's v and g
        float vr = __shfl_down_sync(0xffffffffu, v.a.x, 1), gr = __shfl_down_sync(0xffffffffu, gc.a.x, 1);
        if (w < T::TR && tv_row_in(ci, row) && in != 0u) {
            const float *Vc = sv(vc) + w * T::VS;
            const float *x0 = sx(sc) + (w + 1) * T::XS + 4 * lane + 4;
            Quad x[3] = {lds4(x0), lds4(x0 + T::XC), lds4(x0 + 2 * T::XC)};
            if (lane == 31) vr = Vc[T::TN], gr = ge;
            Quad G[3] = {sub4(sub4(Quad{f2(v.a.y, v.b.x), f2(v.b.y, vr)}, v),
                              div4_rn(sub4(Quad{f2(gc.a.y, gc.b.x), f2(gc.b.y, gr)}, gc), lam, rlam, rcp_lam)),
                         zero4(), zero4()};
            mask_fwd(G[0]);
            if (row + 1 < ci.z)
                G[1] = sub4(sub4(lds4(Vc + T::VS + 4 * lane), v), div4_rn(sub4(gd, gc), lam, rlam, rcp_lam));
            if (tv_row_in(cn, row)) G[2] = sub4(sub4(vn, v), div4_rn(sub4(gn, gc), lam, rlam, rcp_lam));
            const Quad d = tv_step(x, G, tau, tau_in_range != 0);
            float *o = xi_out + oc;
            if (in == 0xfu) {
                dmax = fmaxf(fmaxf(dmax, fmaxf(d.a.x, d.a.y)), fmaxf(d.b.x, d.b.y));
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    *reinterpret_cast<float4 *>(o + k * g.plane_w) = make_float4(x[k].a.x, x[k].a.y, x[k].b.x, x[k].b.y);
            } else {
                const float dd[4] = {d.a.x, d.a.y, d.b.x, d.b.y};
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if ((in >> j) & 1u) {
                        dmax = fmaxf(dmax, dd[j]);
#pragma unroll
                        for (int k = 0; k < 3; ++k) {
                            const float2 h = j < 2 ? x[k].a : x[k].b;
                            o[k * g.plane_w + j] = j & 1 ? h.y : h.x;
                        }
                    }
            }
        }
        // past this barrier every warp is done with plane c's xi slot and v slot
        if (sync_aborted(abort)) break;
        if (t == 0 && c + 3 <= cb) issue(c + 3, sc);
        v = vn;
        gc = gn, ge = gne, gn = g2, gne = g2e, gd = gd1;
        ci = cn, cn = c2;
        oc = on, on = o2;
        const int s_free = sc;
        sc = sn;
        sn = 3 - s_free - sn;
        vc ^= 1;
    }
    if (t == 0 && *abort) {
        // loads still in flight must land before the block's shared memory goes away
        for (int k = 0; k < T::SLOTS; ++k)
            if ((pending >> k) & 1u) mbar_wait_bounded(bar + k, (phase >> k) & 1u, kDrainTries);
        atomicExch(err, 1);
    }
    if (dq) block_max_to(dmax, dq);
}

}  // namespace potts
