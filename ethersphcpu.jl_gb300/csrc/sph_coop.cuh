// sph_coop.cuh — cooperative neighbour gathers of the plain FP64 form.
//
// GB300 has two FP64 lanes a SM and cycle (1/64 of FP32), so the gathers of this form are
// bound by their FP64 instructions and, on small scenes, by how few SMs those run on.  Two
// things follow, and both live here:
//   * kCoopLanes lanes of a warp share one particle.  They first select its neighbours with
//     FP32 and integer work alone (a conservative distance test on cell-relative positions,
//     coop_select), packing them into a list in shared memory; then each lane takes every
//     kCoopLanes-th entry of the list, so the FP64 pair terms run on full warps and no
//     rejected candidate costs an FP64 instruction.
//   * a particle's sums do not depend on the batch, the block size or the other particles
//     of its warp: where a scene at rest cancels large terms (pressure and wall forces) the
//     terms are rounded and added in the reference's own order (pair_kernel, add_terms);
//     the other sums are taken by lane, lane t entries t, t + 8, ..., and the lanes' sums
//     added in one fixed order.
#pragma once

#include "sph_physics.cuh"
#include "sph_kernels.h"

namespace sph {

constexpr int kCoopLanes = 8;        // lanes per particle (the 2 m + 1 <= 7 rows of a plane fit them)
constexpr int kCoopMaxParticles = 32;  // particles of the largest block (256 threads)
// Entries of a particle's list: r_cut = 3 dx has about 28 (2D) / 112 (3D) neighbours; a
// particle with more runs its pair terms in several passes (coop_select).
template <int DIM> constexpr int kCoopList = DIM == 2 ? 64 : 144;
// Row lengths in shared memory, in 8-byte words: partial sums (a particle's lanes fall on
// different banks) and pair terms (one a lane).
constexpr int kCoopStride = kCoopMaxParticles + 4;
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
    inv = fma(fma(-r, y1, 1.0), y1, y1);
    return r;
}
__device__ __forceinline__ bool sqrt_rn_range(double a) {
    return ((unsigned)__double2hiint(a) >> 20) - 123u < 1800u;
}

// a / b rounded to nearest, y = 1 / b rounded to nearest (the same residual correction).
__device__ __forceinline__ double div_rn(double a, double b, double y) {
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
}

// max(a, 0) on the sign bit (integer work)
__device__ __forceinline__ double relu(double a) { return __double2hiint(a) < 0 ? 0.0 : a; }

// x^4, x^5, x^6 as jl_powi rounds them (finite x).
template <int N>
__device__ __forceinline__ double powi_fixed(double x) {
    const double h = x * x, l = fma(x, x, -h);
    const double hh = h * h;
    const double ll = fma(h, h, -hh) + h * 2.0 * l;
    if (N == 4) return hh + ll;
    if (N == 5) return fma(hh, x, x * ll);
    return fma(hh, h, fma(h, ll, hh * l));
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
    float fu[3];
    cell_units<DIM>(x, S, c, fu);
    return make_float4(fu[0], fu[1], fu[2], (float)c[0]);
}

// The candidates of one particle in the cell list (start, pos), tested in FP32 and packed
// into `list` (shared memory of the particle's lanes) in walk order (cells z, y, x); the
// pair work `flush(cnt)` runs when the list is full and at the end.  me: the particle's
// select_pos, c its cell, self its index in `pos` (-1: none).  Every lane of the warp calls
// this together; a group without a particle passes on = false.
//
// The test keeps a relative margin of 1e-4 on r_cut^2: cell-relative differences within
// the stencil carry an FP32 error of some 1e-6 cells.  A particle clamped into an edge cell
// from further than 64 cells outside the grid, or with a non-finite position, is tested by
// `within(j)` instead (FP64), so only candidates beyond r_cut are left out.
template <int DIM, typename Within, typename Pairs>
__device__ __forceinline__ void coop_select(const SceneDev& S, const int32_t* __restrict__ start,
                                            const float4* __restrict__ pos, const int32_t c[3], const float4 me,
                                            int self, bool on, int32_t* list, Within&& within,
                                            Pairs&& pairs) {
    constexpr int CAP = kCoopList<DIM>;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & (kCoopLanes - 1);
    const int shift = (threadIdx.x & 31) & ~(kCoopLanes - 1);
    const unsigned below = (1u << lane) - 1u;
    const int m = S.reach;
    const int zr = DIM == 3 ? m : 0;
    const float ex = S.sel_e[0], ey = S.sel_e[1], ez = S.sel_e[2];  // cell edges in units of r_cut
    const float r2 = 1.0001f;
    const float nx = (float)S.n[0];
    const bool wide = !(fabsf(me.x) <= 64.f && fabsf(me.y) <= 64.f && fabsf(me.z) <= 64.f);
    const int planes = DIM == 3 ? (int)__reduce_max_sync(full, (unsigned)zr) : 0;
    int first_entry = 0, cnt = 0;
    for (int dz = -planes; dz <= planes; ++dz) {
        // lane r holds row dy = r - 3 of this plane: its cells form one run [b, b + l1) of the
        // sorted arrays, or two where a periodic axis wraps; cells beyond r_cut are skipped as
        // in walk_cells_pruned (rows and cells at the grid's edge stay whole: they may hold
        // clamped particles)
        int b = 0, l1 = 0, b2 = 0, l2 = 0;
        const int dy = lane - 3, y = c[1] + dy, z = c[2] + dz;
        if (on && lane < 7 && dy >= -m && dy <= m && y >= 0 && y < S.n[1] &&
            (DIM == 2 || (dz >= -zr && dz <= zr && z >= 0 && z < S.n[2]))) {
            const int row = S.cell_off + (z * S.n[1] + y) * S.n[0];
            int x0 = c[0] - m, x1 = c[0] + m;
            bool keep = true;
            const bool edge = y == 0 || y == S.n[1] - 1 || (DIM == 3 && (z == 0 || z == S.n[2] - 1));
            if (!edge && !wide) {
                const float gy = fmaxf(fmaxf((float)dy - me.y, me.y - (float)(dy + 1)), 0.f) * ey;
                float rem = r2 - gy * gy;
                if (DIM == 3) {
                    const float gz = fmaxf(fmaxf((float)dz - me.z, me.z - (float)(dz + 1)), 0.f) * ez;
                    rem -= gz * gz;
                }
                keep = !(rem < 0.f);
                if (keep && !S.periodic_x) {
                    const float w = sqrtf(rem) * S.sel_inv_ex;
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
        const bool wraps = __any_sync(full, l2 != 0);
        const int most = (int)__reduce_max_sync(full, (unsigned)total);
        const int rounds = dz == planes ? max(most, 1) : most;  // the last round runs the pairs
        for (int t0 = 0; t0 < rounds; t0 += kCoopLanes) {
            const int t = t0 + lane;
            int r = 0;
#pragma unroll
            for (int k = 0; k < 6; ++k) r += t >= ends[k];
            int j = t - __shfl_sync(full, first, r, kCoopLanes);  // place in the row
            const int jb = __shfl_sync(full, b, r, kCoopLanes);
            if (wraps) {
                const int n1 = __shfl_sync(full, l1, r, kCoopLanes), jb2 = __shfl_sync(full, b2, r, kCoopLanes);
                j = j < n1 ? jb + j : jb2 + (j - n1);
            } else {
                j += jb;
            }
            bool take = t < total;
            if (take) {
                const float4 p = __ldg(pos + j);
                float cx = p.w - me.w;
                if (S.periodic_x) cx = cx > 0.5f * nx ? cx - nx : (cx < -0.5f * nx ? cx + nx : cx);
                const float rx = (cx + (p.x - me.x)) * ex;
                const float ry = ((float)(r - 3) + (p.y - me.y)) * ey;
                float d2 = rx * rx + ry * ry;
                if (DIM == 3) {
                    const float rz = ((float)dz + (p.z - me.z)) * ez;
                    d2 += rz * rz;
                }
                take = j != self && (wide ? within(j) : d2 <= r2);
            }
            const unsigned hit = (__ballot_sync(full, take) >> shift) & 0xffu;
            if (take) list[cnt + __popc(hit & below)] = j;
            cnt += __popc(hit);
            const bool last = dz == planes && t0 + kCoopLanes >= rounds;
            if (last || __any_sync(full, cnt > CAP - kCoopLanes)) {
                __syncwarp(full);
                pairs(first_entry, cnt);
                __syncwarp(full);
                first_entry += cnt;
                cnt = 0;
            }
        }
    }
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

// Particles of a block (blockDim.x / kCoopLanes) for n particles.  Large blocks run the
// per-particle epilogue (about 70 FP64 instructions) on full warps; small ones spread a
// small scene over the SMs.
inline int coop_particles(int64_t n) {
    const int64_t sms = 152;
    if (n >= 6 * sms * 32) return 32;
    if (n >= 4 * sms * 16) return 16;
    return 8;
}

}  // namespace sph
