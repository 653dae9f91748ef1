// sph_coop.cuh — cooperative neighbour gathers: what the plain FP64 form (sph_fp64.cu) and
// the FP32-compensated form (sph_fp32.cuh) share, and the building blocks of the former.
//
// GB300 has two FP64 lanes a SM and cycle (1/64 of FP32), so the gathers of the FP64 form are
// bound by their FP64 instructions and, on small scenes, by how few SMs those run on.  Two
// things follow, and both live here:
//   * kCoopLanes lanes of a warp share one particle.  They first select its neighbours with
//     FP32 and integer work alone (a conservative distance test on cell-relative positions,
//     coop_select), packing them into a list in shared memory; then each lane takes every
//     kCoopLanes-th entry of the list, so the FP64 pair terms run on full warps and no
//     rejected candidate costs an FP64 instruction.
//   * each of an SM's four schedulers has its own FP64 unit, which one warp can keep busy:
//     the work has to be even over 608 of them.  The grid is what the SMs hold at once, and
//     its warps draw the scene's particles from a queue, four at a time; after eight draws a
//     warp updates its 32 particles, one a lane.  (Warps with a fixed share of 32 particles
//     left the FP64 units idle for a third of the time, shares of 8 ran the update on a
//     quarter of a warp.)  No warp waits for another.
//   * a particle's sums do not depend on the batch, the warp or its other particles: where a
//     scene at rest cancels large terms (pressure and wall forces) the terms are rounded and
//     added in the reference's own order (pair_kernel, add_terms);
//     the other sums are taken by lane, lane t entries t, t + 8, ..., and the lanes' sums
//     added in one fixed order.
#pragma once

#include <algorithm>

#include "sph_physics.cuh"
#include "sph_kernels.h"

namespace sph {

constexpr int kCoopLanes = 8;        // lanes per particle (the 2 m + 1 <= 7 rows of a plane fit them)
constexpr int kCoopGroups = 32 / kCoopLanes;  // particles a warp works on at a time
// Entries of a particle's list: r_cut = 3 dx has about 28 (2D) / 112 (3D) neighbours; a
// particle with more runs its pair terms in several passes (coop_select).
template <int DIM> constexpr int kCoopList = DIM == 2 ? 64 : 144;
// Row length of the pair terms in shared memory (8-byte words; one term a lane).
constexpr int kTermStride = 33;

// ---------------------------------------------------------------- FP64 building blocks
// Gross approximations (about 20 bits) that start the iterations below.
__device__ __forceinline__ double approx_rsqrt(double a) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    return y;
}
__device__ __forceinline__ double approx_rcp(double a) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    return y;
}

// 1 / a to an ulp: one third-order Householder step, 1 / a = y (1 + e + e^2 + ...) with
// e = 1 - a y (three FP64 instructions).
__device__ __forceinline__ double rcp3(double a) {
    const double y = approx_rcp(a);
    const double e = fma(-a, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// sqrt(a) and (INV) 1 / sqrt(a) to an ulp: a^-1/2 = y (1 + e/2 + 3 e^2/8 + ...) with
// e = 1 - a y^2 (five and seven FP64 instructions).  a below 1e-30 (in units of h^2:
// coincident particles) counts as about 0.
template <bool INV>
__device__ __forceinline__ double sqrt3(double a, double& inv) {
    const double y = approx_rsqrt(__hiloint2double(max(__double2hiint(a), 0x39b4484c), __double2loint(a)));
    const double s = a * y;
    const double e = fma(-s, y, 1.0);
    const double p = fma(e, 0.375, 0.5);
    if (INV) inv = fma(y * e, p, y);
    return fma(s * e, p, s);
}

// y = 1 / a from a residual correction, right but for a mantissa of all ones: there 1 / a lies
// just above the middle between a power of two and its successor, which is the value to return,
// and the correction stays at the power.
__device__ __forceinline__ double rcp_of_ones(double a, double y) {
    const bool ones = (__double2loint(a) & (__double2hiint(a) | 0xfff00000)) == -1;
    return __hiloint2double(__double2hiint(y), ones ? 1 : __double2loint(y));
}

// sqrt(a) and 1 / sqrt(a), both rounded to nearest as the IEEE operations round them
// (the second is 1 / (the rounded root)), for a in [2^-900, 2^900]: the values above,
// corrected by their residuals (Markstein, Computation of elementary functions on the IBM
// RISC System/6000, 1990).  Twelve FP64 instructions for the two.
__device__ __forceinline__ double sqrt_rn(double a, double& inv) {
    const double y = approx_rsqrt(a);
    const double s = a * y;
    const double e = fma(-s, y, 1.0);
    const double p = fma(e, 0.375, 0.5);
    const double y1 = fma(y * e, p, y);
    const double s1 = fma(s * e, p, s);
    const double r = fma(fma(-s1, s1, a), 0.5 * y1, s1);
    inv = rcp_of_ones(r, fma(fma(-r, y1, 1.0), y1, y1));
    return r;
}
__device__ __forceinline__ bool sqrt_rn_range(double a) {
    return ((unsigned)__double2hiint(a) >> 20) - 123u < 1800u;
}
// |a| in [2^-300, 2^300] (a^2 and quotients of ordinary values by it stay normal numbers)
__device__ __forceinline__ bool rcp_rn_range(double a) {
    return ((unsigned)__double2hiint(a) >> 20 & 0x7ffu) - 723u < 600u;
}

// 1 / a rounded to nearest, for |a| in [2^-900, 2^900].
__device__ __forceinline__ double rcp_rn(double a) {
    const double y = rcp3(a);
    return rcp_of_ones(a, fma(fma(-a, y, 1.0), y, y));
}

// a / b rounded to nearest, y = 1 / b rounded to nearest (the same residual correction).
__device__ __forceinline__ double div_rn(double a, double b, double y) {
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
}

// max(a, 0) on the sign bit (integer work)
__device__ __forceinline__ double relu(double a) { return __double2hiint(a) < 0 ? 0.0 : a; }

// (double)x by integer work: the conversion takes the FP64 unit as long as an addition.  A
// subnormal is scaled into the normal numbers (exactly) and its exponent set right after.
__device__ __forceinline__ double widen(float x) {
    const int32_t e = __float_as_int(x) & 0x7f800000;
    const int32_t b = __float_as_int(e ? x : __fmul_rn(x, 16777216.f));
    const int32_t bias = e == 0x7f800000 ? 0x70000000 : (e ? 0x38000000 : 0x38000000 - (24 << 20));
    const int32_t top = (b & 0x7fffffff) ? ((b & 0x7fffffff) >> 3) + bias : 0;
    return __hiloint2double((b & (int32_t)0x80000000) | top, b << 29);
}

// x^4 .. x^7 as jl_powi rounds them (finite x).
template <int N>
__device__ __forceinline__ double powi_fixed(double x) {
    const double h = x * x, l = fma(x, x, -h);
    const double hh = h * h;
    const double ll = fma(h, h, -hh) + h * 2.0 * l;
    if (N == 4) return hh + ll;
    if (N == 5) return fma(hh, x, x * ll);
    if (N == 6) return fma(hh, h, fma(h, ll, hh * l));
    const double c = h * x, cl = fma(h, x, -c) + x * l;  // x^3
    return fma(hh, c, fma(c, ll, hh * cl));
}

// ---------------------------------------------------------------- kernels
// F with dW/dr / r = (kg_a / h) F at q2 = q^2 = (r / h)^2 inside the support, finite at
// r = 0: what continuity needs.
template <int KK>
__device__ __forceinline__ double kernel_f(double q2) {
    double inv;
    if (KK == SPH_KERNEL_GAUSSIAN) return exp(-q2);
    if (KK == SPH_KERNEL_CUBIC_SPLINE) {
        const double q = sqrt3<true>(q2, inv);
        const double t = relu(2.0 - q);
        return __double2hiint(q) < 0x3ff00000 ? fma(3.0, q, -4.0) : -(t * t) * inv;  // q < 1
    }
    const double q = sqrt3<false>(q2, inv);
    const double t = relu(2.0 - q);
    const double t2 = t * t;
    if (KK == SPH_KERNEL_WENDLAND_C2) return t2 * t;
    return (t2 * t2) * t * fma(35.0 / 96.0, q, 7.0 / 48.0);
}

// W and dW/dr at q = r / h, bit for bit those of kernel_wdw.
template <int KK>
__device__ __forceinline__ void kernel_wdw_q(double q, const SceneDev& S, double& W, double& dW) {
    const int hi = __double2hiint(q);
    if (KK == SPH_KERNEL_GAUSSIAN) {
        const double e = exp(-(q * q));
        W = hi < 0x40080000 ? S.kw_a * e : 0.0;  // q < 3
        dW = hi < 0x40080000 ? S.kg_a * q * e : 0.0;
        return;
    }
    const bool in = hi < 0x40000000;  // q < 2
    const double t = 2.0 - q;
    if (KK == SPH_KERNEL_CUBIC_SPLINE) {
        const bool core = hi < 0x3ff00000;  // q < 1
        const double t2 = t * t;
        const double w0 = 3.0 * (q * q) * (q - 2.0) + 4.0, w1 = t2 * t;
        const double d0 = S.kg_a * q * (3.0 * q - 4.0), d1 = -S.kg_a * t2;
        W = in ? S.kw_a * (core ? w0 : w1) : 0.0;
        dW = in ? (core ? d0 : d1) : 0.0;
    } else if (KK == SPH_KERNEL_WENDLAND_C2) {
        W = in ? S.kw_a * powi_fixed<4>(t) * (1.0 + 2.0 * q) * 0.0625 : 0.0;
        dW = in ? S.kg_a * q * (t * t * t) : 0.0;
    } else {
        W = in ? div_rn(S.kw_a * powi_fixed<6>(t) * (35.0 * (q * q) + 36.0 * q + 12.0), 768.0, 1.0 / 768.0) : 0.0;
        dW = in ? S.kg_a * (35.0 / 96.0 * (q * q) + 7.0 / 48.0 * q) * powi_fixed<5>(t) : 0.0;
    }
}

// r, W, dW/dr and grad W of a pair, bit for bit those of sqrt, kernel_wdw and grad_vec.
template <int DIM, int KK>
__device__ __forceinline__ void pair_kernel(const double rv[DIM], double d2, const SceneDev& S, double& r, double& W,
                                            double& dW, double grad[DIM]) {
    if (sqrt_rn_range(d2)) {
        double inv;
        r = sqrt_rn(d2, inv);
        kernel_wdw_q<KK>(div_rn(r, S.h, S.inv_h), S, W, dW);
#pragma unroll
        for (int k = 0; k < DIM; ++k) grad[k] = dW * (rv[k] * inv);
    } else {  // coincident particles, lengths near the limits of FP64
        r = sqrt(d2);
        kernel_wdw<KK>(r, S, W, dW);
        grad_vec<DIM>(dW, r, rv, grad);
    }
}

// Whether a selected pair counts: the reference's own test, d^2 <= r_cut^2 as it rounds it
// (and r / h < 3 for the Gaussian, whose value is cut there), taken in FP64 only for pairs
// within 1e-6 of the cut; the others are decided on the upper word of q^2.
template <int DIM, int KK>
__device__ __forceinline__ bool inside_cut(const double rv[DIM], double q2, const SceneDev& S) {
    if (__double2hiint(q2) < S.q2_in_hi) return true;
    const double d2 = norm_sq<DIM>(rv);
    return d2 <= S.rc2 && (KK != SPH_KERNEL_GAUSSIAN || sqrt(d2) / S.h < 3.0);
}
// the same for d2 = norm_sq(r_vec)
template <int KK>
__device__ __forceinline__ bool inside_cut(double d2, const SceneDev& S) {
    if (__double2hiint(d2) < S.d2_in_hi) return true;
    return d2 <= S.rc2;  // kernel_wdw(_q) cuts the Gaussian itself
}

// ---------------------------------------------------------------- selection
// FP32 position of a particle for the selection, in cell units: (x, y, z) relative to its
// cell and the cell's x index (exact: a grid has at most 2^24 cells on an axis).
template <int DIM, typename V>
__device__ __forceinline__ float4 select_pos(const V& x, const SceneDev& S, const int32_t c[3]) {
    float4 p;
    p.x = (float)fma(x.x - S.lo[0], S.inv_cell[0], -(double)c[0]);
    p.y = (float)fma(x.y - S.lo[1], S.inv_cell[1], -(double)c[1]);
    p.z = DIM == 3 ? (float)fma(comp(x, DIM - 1) - S.lo[2], S.inv_cell[2], -(double)c[2]) : 0.f;
    p.w = (float)c[0];
    return p;
}
__device__ __forceinline__ bool select_far(const float4& p) {
    return !(fabsf(p.x) <= 64.f && fabsf(p.y) <= 64.f && fabsf(p.z) <= 64.f);
}

// |r|^2 with a fixed rounding sequence: every kernel of the FP32 form decides a pair alike.
__device__ __forceinline__ float dist2(float rx, float ry, float rz) {
    return __fmaf_rn(rx, rx, __fmaf_rn(ry, ry, __fmul_rn(rz, rz)));
}

// The neighbours of one particle in the cell list (start, pos), selected in FP32 and packed
// into a list in walk order (cells z, y, x) with a relative margin of 1e-4 on r_cut^2
// (cell-relative differences within the stencil carry an FP32 error of some 1e-6 cells): only
// candidates beyond r_cut are left out.  A particle far outside its cell (clamped from
// outside the grid) or with a non-finite position is tested by within(j), in FP64.  The pair
// work pairs(first, cnt) runs at the end, and before when a list of the warp is full: the list
// (kCoopList entries) then holds entries first .. first + cnt - 1 of the whole.  me: the
// particle's select_pos, c its cell, self its index in `pos` (-1: none).  Every lane of the
// warp calls this together; a group without a particle passes on = false.
//
// Rows and cells beyond r_cut are left out with the same margin.  Rows on the y/z grid
// boundary and the first and last x cells may hold particles clamped from outside the grid
// and stay whole, as does the stencil of a particle itself far outside its cell.
template <int DIM, typename Within, typename Pairs>
__device__ __forceinline__ void coop_select(const SceneDev& S, const int32_t* __restrict__ start,
                                            const float4* __restrict__ pos, const int32_t c[3], const float4& me,
                                            int self, bool on, int32_t* list, Within&& within, Pairs&& pairs) {
    const float ex = S.sel_e[0], ey = S.sel_e[1], ez = S.sel_e[2], inv_ex = S.sel_inv_ex;  // cell edges / r_cut
    constexpr float kR2 = 1.0001f;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & (kCoopLanes - 1);
    const int shift = (threadIdx.x & 31) & ~(kCoopLanes - 1);
    const unsigned below = (1u << lane) - 1u;
    const int m = S.reach;
    const int zr = DIM == 3 ? m : 0;
    const float nx = (float)S.n[0];
    const bool far = select_far(me);
    const int planes = DIM == 3 ? (int)__reduce_max_sync(full, (unsigned)zr) : 0;
    int first_entry = 0, cnt = 0;
    for (int dz = -planes; dz <= planes; ++dz) {
        // lane r holds row dy = r - 3 of this plane: its cells form one run [b, b + l1) of the
        // sorted arrays, or two where a periodic axis wraps
        int b = 0, l1 = 0, b2 = 0, l2 = 0;
        const int dy = lane - 3, y = c[1] + dy, z = c[2] + dz;
        if (on && lane < 7 && dy >= -m && dy <= m && y >= 0 && y < S.n[1] &&
            (DIM == 2 || (dz >= -zr && dz <= zr && z >= 0 && z < S.n[2]))) {
            const int row = S.cell_off + (z * S.n[1] + y) * S.n[0];
            int x0 = c[0] - m, x1 = c[0] + m;
            bool keep = true;
            const bool edge = y == 0 || y == S.n[1] - 1 || (DIM == 3 && (z == 0 || z == S.n[2] - 1));
            if (!edge && !far) {
                const float gy = fmaxf(fmaxf((float)dy - me.y, me.y - (float)(dy + 1)), 0.f) * ey;
                float rem = kR2 - gy * gy;
                if (DIM == 3) {
                    const float gz = fmaxf(fmaxf((float)dz - me.z, me.z - (float)(dz + 1)), 0.f) * ez;
                    rem -= gz * gz;
                }
                keep = !(rem < 0.f);
                if (keep && !S.periodic_x) {
                    const float w = sqrtf(rem) * inv_ex;
                    const int a = c[0] + (int)floorf(me.x - w), e = c[0] + (int)floorf(me.x + w);
                    if (x0 > 0 && a > x0) x0 = min(a, S.n[0] - 1);
                    if (x1 < S.n[0] - 1 && e < x1) x1 = max(e, 0);
                }
            }
            if (keep) {
                const int lo = max(x0, 0), hi = min(x1, S.n[0] - 1);
                if (lo <= hi) {
                    b = __ldg(start + row + lo);
                    l1 = __ldg(start + row + hi + 1) - b;
                }
                if (S.periodic_x && (x0 < 0 || x1 >= S.n[0])) {
                    const int wl = x0 < 0 ? x0 + S.n[0] : 0, wh = x0 < 0 ? S.n[0] - 1 : x1 - S.n[0];
                    b2 = __ldg(start + row + wl);
                    l2 = __ldg(start + row + wh + 1) - b2;
                    if (x0 < 0) {  // the wrapped cells come first in x order
                        const int tb = b, tl = l1;
                        b = b2;
                        l1 = l2;
                        b2 = tb;
                        l2 = tl;
                    }
                }
            }
        }
        int end = l1 + l2;  // inclusive scan over the rows: row r holds candidates [end(r-1), end(r))
#pragma unroll
        for (int o = 1; o < kCoopLanes; o <<= 1) {
            const int v = __shfl_up_sync(full, end, o, kCoopLanes);
            if (lane >= o) end += v;
        }
        const int total = __shfl_sync(full, end, kCoopLanes - 1, kCoopLanes);
        int ends[6];
#pragma unroll
        for (int r = 0; r < 6; ++r) ends[r] = __shfl_sync(full, end, r, kCoopLanes);
        const int first = end - l1 - l2;
        const int shifted = b - first;  // candidate t of the plane is particle t + shifted of its row
        const bool wraps = __any_sync(full, l2 != 0);
        const int most = (int)__reduce_max_sync(full, (unsigned)total);
        const int rounds = dz == planes ? max(most, 1) : most;  // the last round runs the pairs
        // two rounds at a time: both candidates' positions are loaded before the first is tested
        for (int t0 = 0; t0 < rounds; t0 += 2 * kCoopLanes) {
            int j[2];
            float dyf[2];
            float4 p[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int t = t0 + h * kCoopLanes + lane;
                int r = 0;
#pragma unroll
                for (int k = 0; k < 6; ++k) r += t >= ends[k];
                int q = t + __shfl_sync(full, shifted, r, kCoopLanes);
                if (wraps) {
                    const int f = __shfl_sync(full, first, r, kCoopLanes), n1 = __shfl_sync(full, l1, r, kCoopLanes);
                    const int jb2 = __shfl_sync(full, b2, r, kCoopLanes);
                    if (t - f >= n1) q = jb2 + (t - f - n1);
                }
                dyf[h] = (float)(r - 3);
                j[h] = t < total ? q : -1;
                p[h] = me;
                if (t < total) p[h] = __ldg(pos + q);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float cx = me.w - p[h].w;
                if (S.periodic_x) cx = cx > 0.5f * nx ? cx - nx : (cx < -0.5f * nx ? cx + nx : cx);
                const float rx = (cx + (me.x - p[h].x)) * ex;
                const float ry = ((me.y - p[h].y) - dyf[h]) * ey;
                const float rz = DIM == 3 ? ((me.z - p[h].z) - (float)dz) * ez : 0.f;
                bool take = j[h] >= 0 && j[h] != self;
                if (take) take = far ? within(j[h]) : dist2(rx, ry, rz) <= kR2;
                const unsigned hit = (__ballot_sync(full, take) >> shift) & 0xffu;
                if (take) list[cnt + __popc(hit & below)] = j[h];
                cnt += __popc(hit);
            }
            const bool last = dz == planes && t0 + 2 * kCoopLanes >= rounds;
            if (last || __any_sync(full, cnt > kCoopList<DIM> - 2 * kCoopLanes)) {
                __syncwarp(full);
                pairs(first_entry, cnt);
                __syncwarp(full);
                first_entry += cnt;
                cnt = 0;
            }
        }
    }
}

// d^2 <= r_cut^2 in FP64, for the selection of particles far outside the grid.
template <int DIM, typename V>
__device__ __forceinline__ bool within_cut(const V& xi, const V& xj, const SceneDev& S) {
    double rv[DIM];
    make_rvec<DIM>(xi, xj, S, rv);
    return norm_sq<DIM>(rv) <= S.rc2;
}

// The next step's cell key of a particle that moved from x0 to x1: its FP32 cell position
// decides it where the particle is clear of the cell boundaries (by 1e-4 cells, far above
// the FP32 error) and of the grid's edge cells, the FP64 hash otherwise; the key is the
// same.  The hash takes six FP64 instructions an axis, this two.
template <int DIM, typename V>
__device__ __forceinline__ int32_t moved_key(int32_t key, const float4& me, const V& x0, const V& x1,
                                             const SceneDev& S) {
    const float u[3] = {me.x + (float)(x1.x - x0.x) * S.inv_cell_f[0], me.y + (float)(x1.y - x0.y) * S.inv_cell_f[1],
                        DIM == 3 ? me.z + (float)(comp(x1, DIM - 1) - comp(x0, DIM - 1)) * S.inv_cell_f[2] : 0.f};
    int32_t c[3];
    decode_cell(key, S, c);
    bool sure = true;
    int32_t k = key, stride = 1;
#pragma unroll
    for (int a = 0; a < DIM; ++a) {
        const float f = floorf(u[a]), frac = u[a] - f;
        sure &= frac > 1e-4f && frac < 1.f - 1e-4f && fabsf(f) <= 1.f && c[a] > 1 && c[a] < S.n[a] - 2;
        k += (int32_t)f * stride;
        stride *= S.n[a];
    }
    return sure ? k : cell_key<DIM>(x1, S);
}

// Adds a round of pair terms (entry e of the list in lane e of the particle's group, e0 <=
// e < e1; kTerms vectors a pair, in `terms` of the warp) to the particle's vector sum, of
// which lane d < DIM holds component d: entry by entry, term by term.
template <int DIM, int kTerms>
__device__ __forceinline__ void add_terms(const double* terms, int lane, int shift, int e0, int e1, double& sum) {
    if (lane < DIM)
        for (int e = e0; e < e1; ++e)
#pragma unroll
            for (int s = 0; s < kTerms; ++s) sum += terms[(s * DIM + lane) * kTermStride + shift + e];
}

// Sum of v over the lanes of a particle, the same tree and bits in every lane.
__device__ __forceinline__ double coop_sum(double v) {
#pragma unroll
    for (int o = 1; o < kCoopLanes; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The grid: two blocks of eight warps on each of the 152 SMs, where a scene has 16 fours or
// more for each of those warps or no more than one; in between one block of six to eight
// warps an SM (a warp with two or three draws would run its update on few lanes, and the
// 16 warps' second draws would be uneven).  A lid-driven cavity of 10,201 particles: K4 36
// us with 16 warps an SM, 27 us with 6; K5 98 and 86 us.
constexpr int kCoopThreads = 256;
constexpr int kCoopBlocks = 2;
struct CoopShape {
    int grid, threads;
};
inline CoopShape coop_shape(int64_t n) {
    const int64_t sms = 152, fours = std::max<int64_t>(1, (n + kCoopGroups - 1) / kCoopGroups);
    if (fours <= sms * 16 || n >= sms * 8 * 32)
        return {(int)std::min(kCoopBlocks * sms, fours), kCoopThreads};
    return {(int)sms, (int)(32 * std::max<int64_t>(6, n / (32 * sms)))};
}

// A warp's part of n particles: body(i, p, on) for its group's particle i (clamped to a
// valid one with on = false past the end), p its place among the warp's next 32; update(i)
// one lane a particle after each 32 and at the end.  *queue counts the draws beyond every
// warp's first: 0 before the launch, a word of the launch's own (SortScratch::queue).
template <typename Body, typename Update>
__device__ __forceinline__ void coop_turns(int n, int32_t* queue, Body&& body, Update&& update) {
    const unsigned full = 0xffffffffu;
    const int fours = (n + kCoopGroups - 1) / kCoopGroups;
    const int W = gridDim.x * (blockDim.x / 32);
    const int lane = threadIdx.x & 31, g = lane / kCoopLanes;
    int next = threadIdx.x / 32 * gridDim.x + blockIdx.x;  // the first draw
    while (next < fours) {
        int mine = fours;  // lane k: the k-th four of this set
        int k = 0;
#pragma unroll 1
        for (; k < kCoopLanes && next < fours; ++k) {
            if (lane == k) mine = next;
            const int i = next * kCoopGroups + g;
            int drawn = 0;
            if (lane == 0) drawn = atomicAdd(queue, 1);
            body(min(i, n - 1), k * kCoopGroups + g, i < n);
            next = W + __shfl_sync(full, drawn, 0);
        }
        __syncwarp();
        const int i = __shfl_sync(full, mine, lane / kCoopGroups) * kCoopGroups + lane % kCoopGroups;
        if (i < n) update(i);
        __syncwarp();
    }
}

}  // namespace sph
