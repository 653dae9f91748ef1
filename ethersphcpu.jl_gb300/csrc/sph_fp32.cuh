// sph_fp32.cuh — FP32-compensated form of the continuity, momentum and Shepard gathers
//
// Pair arithmetic runs in FP32 on cell-relative positions: every particle carries its
// position relative to its cell, in cell units, and its cell's x index (select_pos), so the
// vector to a neighbour dx cells away is (dx + (x_i - x_j)) edge, formed from numbers of
// magnitude <= 4 with an error of some 1e-7 cells.  Continuity and force sums are
// Kahan-compensated FP32 accumulators; the result (sum - compensation) goes to FP64 before
// the forward-Euler update, which runs in FP64 on the FP64 master position / velocity /
// density / temperature.  The Shepard sums accumulate in FP64 (FP32 kernel values times
// FP64 volumes and masses), in the list's order.
//
// Continuity walks the cells, one thread a particle on large scenes and a lane a neighbour
// row on small ones (the same sums, bit for bit), and records each particle's neighbours
// (NbrList).  Momentum reads that list, on small scenes with eight lanes a particle: lane t
// takes entries t, t + 8, ... with compensated partial sums of its own; its block's first warp merges them
// (TwoSum of the sums, the rounding errors joining the compensations) and updates the
// particles, one thread each, because FP64 instructions, of which a GB300 SM runs 1/64 of
// its FP32 rate, cost a warp the same however many lanes take part.  On large scenes a thread
// takes a particle and forms the same eight sums.  The cells of the walls, and of a particle
// whose list does not fit, are walked with a lane a neighbour row (coop_rows).  No sum depends
// on the variant, the batch or the pruning.
//
// What bounds them: on small scenes the chain of loads and rounds of one particle, on large
// ones the issue of instructions (continuity issues in 71 to 80 of 100 cycles, momentum in 43
// to 57 with 15 warps an SM for its eight sums, waiting on neighbours from L2); the bytes would
// take a sixth of the time.
//
// On a re-initialisation step the momentum gather also forms the Shepard sums over the
// same neighbours and writes the re-initialised density: the update and the
// re-initialisation are one kernel.
//
// Same terms, order of walls after fluid, and solve variants as sph_fp64.cu; the
// formulas follow Continuity.jl, PressureForce.jl, ViscosityForce.jl, WallForce.jl,
// ThermalConduction.jl, SelfAction/*.jl and ReconstructValue.jl.
#pragma once

#include "sph_coop.cuh"

namespace sph {

namespace {

enum { kModeFluidWall = 0, kModeWallPressure = 1, kModeThermal = 2, kModeBuffers = 3 };

struct Kahan {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float x) {
        const float y = x - c;
        const float t = s + y;
        c = (t - s) - y;
        s = t;
    }
};

// x^n for n >= 0 by repeated squaring, without the compensation of jl_powi.
__device__ __forceinline__ double powi_plain(double x, int n) {
    double y = 1.0;
    while (n > 0) {
        if (n & 1) y *= x;
        x *= x;
        n >>= 1;
    }
    return y;
}

// Adds a compensated sum (s, c) to another: the sums by an error-free TwoSum whose rounding
// error joins the compensations.
__device__ __forceinline__ void merge(Kahan& k, float s2, float c2) {
    const float t = k.s + s2;
    const float bp = t - k.s;
    const float e = (k.s - (t - bp)) + (s2 - bp);
    k.s = t;
    k.c = (k.c + c2) - e;
}

// 1 / sqrt(a) and a / b by the hardware's approximations, subnormal arguments taken as zero
// (q^2 and the divisors below are ordinary numbers).
__device__ __forceinline__ float rsqrt_ftz(float a) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(a));
    return y;
}
__device__ __forceinline__ float div_ftz(float a, float b) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
    return __fmul_rn(a, y);
}

// F with dW/dr / r = (kg_a / h) F (finite at r = 0) and w with W = kw_a w at q = r / h;
// inv_q = 1 / q (0 at q = 0).  Every product and sum is rounded as written (no contraction
// left to the compiler), so each kernel that forms a pair gets the same bits.
template <int KK>
__device__ __forceinline__ void kernel_fw(float q, float inv_q, float& F, float& w) {
    if (KK == SPH_KERNEL_GAUSSIAN) {
        const float e = q < 3.f ? __expf(-__fmul_rn(q, q)) : 0.f;
        F = e;
        w = e;
    } else if (KK == SPH_KERNEL_CUBIC_SPLINE) {
        const float t = fmaxf(__fsub_rn(2.f, q), 0.f);
        const float t2 = __fmul_rn(t, t);
        const bool in = q < 1.f;
        F = in ? __fmaf_rn(3.f, q, -4.f) : -__fmul_rn(t2, inv_q);
        w = in ? __fmaf_rn(__fmul_rn(3.f, __fmul_rn(q, q)), __fsub_rn(q, 2.f), 4.f) : __fmul_rn(t2, t);
    } else if (KK == SPH_KERNEL_WENDLAND_C2) {
        const float t = fmaxf(__fsub_rn(2.f, q), 0.f);
        const float t2 = __fmul_rn(t, t);
        F = __fmul_rn(t2, t);
        w = __fmul_rn(__fmul_rn(t2, t2), __fmaf_rn(0.125f, q, 0.0625f));
    } else {
        const float t = fmaxf(__fsub_rn(2.f, q), 0.f);
        const float t2 = __fmul_rn(t, t);
        const float t5 = __fmul_rn(__fmul_rn(t2, t2), t);
        F = __fmul_rn(t5, __fmaf_rn(35.f / 96.f, q, 7.f / 48.f));
        w = __fmul_rn(__fmul_rn(t5, t), __fmaf_rn(__fmaf_rn(35.f / 768.f, q, 36.f / 768.f), q, 12.f / 768.f));
    }
}
template <int KK>
__device__ __forceinline__ float kernel_w_f(float q) {
    float F, w;
    kernel_fw<KK>(q, 1.f, F, w);
    return w;
}

constexpr int kSumStride = 36;  // row of lane sums in shared memory (a warp's lanes fall on different banks)

// A pair with r_vec (metres) and the neighbour's index in e.
template <int DIM, int KK>
struct PairF {
    float r[3], d2, F, w;
    int j;
    __device__ __forceinline__ PairF(const float4& e, const SceneDev& S) {
        r[0] = e.x;
        r[1] = e.y;
        r[2] = DIM == 3 ? e.z : 0.f;
        j = __float_as_int(e.w);
        d2 = dist2(r[0], r[1], r[2]);
        const float q2 = __fmul_rn(d2, S.inv_hh_f);
        const float inv_q = q2 > 1e-30f ? rsqrt_ftz(q2) : 0.f;  // a coincident neighbour has q = 0
        kernel_fw<KK>(__fmul_rn(q2, inv_q), inv_q, F, w);
    }
};

constexpr int kRowEntries = 16;  // neighbours of a row that k_continuity_rows_f32 keeps in shared memory

// List entry of neighbour j of i in the cell (dx, dy, dz) away: (j - i) << 9 | (dz + 3) << 6 |
// (dy + 3) << 3 | (dx + 3).
__device__ __forceinline__ float code_offset(int32_t code, int shift) {  // the offset + 3 as a float
    return __int_as_float(0x4b000000 | (code >> shift & 7)) - (8388608.f + 3.f);
}
// r_vec of the listed pair as run_walk forms it, and the neighbour's index.
template <int DIM>
__device__ __forceinline__ float4 listed(int32_t code, const float4& me, const float4& p, int j, const SceneDev& S) {
    const float rx = ((me.x - p.x) - code_offset(code, 0)) * S.cell_f[0];
    const float ry = ((me.y - p.y) - code_offset(code, 3)) * S.cell_f[1];
    const float rz = DIM == 3 ? ((me.z - p.z) - code_offset(code, 6)) * S.cell_f[2] : 0.f;
    return make_float4(rx, ry, rz, __int_as_float(j));
}

// -------------------------------------------------------------------- K4 (FP32)
// The cells of neighbour row (dy, dz) of a particle, as one run [b, e) of the sorted arrays
// or two where a periodic axis wraps, in x order; cells beyond r_cut are left out (prune) with
// the margin rc2_prune and the exceptions of coop_select.
template <int DIM>
__device__ __forceinline__ void row_runs(const SceneDev& S, const int32_t* __restrict__ start, const int32_t c[3],
                                         const float4& me, bool prune, int dy, int dz, int& b, int& e, int& b2,
                                         int& e2) {
    b = e = b2 = e2 = 0;
    const int m = S.reach, y = c[1] + dy, z = c[2] + dz;
    if (dy < -m || dy > m || y < 0 || y >= S.n[1]) return;
    if (DIM == 3 ? (dz < -m || dz > m || z < 0 || z >= S.n[2]) : dz > 0) return;
    int x0 = c[0] - m, x1 = c[0] + m;
    if (prune && y != 0 && y != S.n[1] - 1 && (DIM == 2 || (z != 0 && z != S.n[2] - 1))) {
        const float gy = fmaxf(fmaxf((float)dy - me.y, me.y - (float)(dy + 1)), 0.f) * S.cell_f[1];
        float rem = S.rc2_prune - gy * gy;
        if (DIM == 3) {
            const float gz = fmaxf(fmaxf((float)dz - me.z, me.z - (float)(dz + 1)), 0.f) * S.cell_f[2];
            rem -= gz * gz;
        }
        if (rem < 0.f) return;
        if (!S.periodic_x) {
            const float w = sqrtf(rem) * S.inv_cell_fx;
            const int a = c[0] + (int)floorf(me.x - w), q = c[0] + (int)floorf(me.x + w);
            if (x0 > 0 && a > x0) x0 = min(a, S.n[0] - 1);
            if (x1 < S.n[0] - 1 && q < x1) x1 = max(q, 0);
        }
    }
    const int32_t* s = start + S.cell_off + (z * S.n[1] + y) * S.n[0];
    const int lo = max(x0, 0), hi = min(x1, S.n[0] - 1);
    if (lo <= hi) {
        b = __ldg(s + lo);
        e = __ldg(s + hi + 1);
    }
    if (S.periodic_x && (x0 < 0 || x1 >= S.n[0])) {
        b2 = __ldg(s + (x0 < 0 ? x0 + S.n[0] : 0));
        e2 = __ldg(s + (x0 < 0 ? S.n[0] : x1 - S.n[0] + 1));
        if (x0 < 0) {  // the wrapped cells come first in x order
            const int tb = b, te = e;
            b = b2;
            e = e2;
            b2 = tb;
            e2 = te;
        }
        if (b >= e) {  // the first run is empty only where both are
            b = b2;
            e = e2;
            b2 = e2 = 0;
        }
    }
}

// One run of candidates of particle i: those within r_cut are passed to f(j, r, dx + 3, data)
// with r = x_i - x_j; data = load(j), loaded with the position before the candidate in front
// of it is tested.
template <int DIM, typename Load, typename F>
__device__ __forceinline__ void run_walk(const SceneDev& S, const float4* __restrict__ pos, int i, const float4& me,
                                         int j, int e, float dyf, float dzf, Load&& load, F&& f) {
    if (j >= e) return;
    const float nx = (float)S.n[0];
    float4 p = __ldg(pos + j);
    auto data = load(j);
    for (;;) {
        const int jn = j + 1;
        float4 pn = p;
        auto dn = data;
        if (jn < e) {
            pn = __ldg(pos + jn);
            dn = load(jn);
        }
        float cx = me.w - p.w;
        if (S.periodic_x) cx = cx > 0.5f * nx ? cx - nx : (cx < -0.5f * nx ? cx + nx : cx);
        const float rx = ((me.x - p.x) + cx) * S.cell_f[0];
        const float ry = ((me.y - p.y) - dyf) * S.cell_f[1];
        const float rz = DIM == 3 ? ((me.z - p.z) - dzf) * S.cell_f[2] : 0.f;
        if (dist2(rx, ry, rz) <= S.rc2_f && j != i)
            f(j, make_float4(rx, ry, rz, __int_as_float(j)), __float_as_int((8388608.f + 3.f) - cx) & 7, data);
        if (jn >= e) return;
        j = jn;
        p = pn;
        data = dn;
    }
}

// The continuity terms of a run into `sum`, each neighbour listed by emit(code).
template <int DIM, int KK, typename Emit>
__device__ __forceinline__ void run_pairs(const SceneDev& S, const SortedState& st, int i, const float4& me,
                                          const float4& vi, int j, int e, float dyf, float dzf, int tag, Kahan& sum,
                                          Emit&& emit) {
    run_walk<DIM>(S, st.fa, i, me, j, e, dyf, dzf, [&](int q) { return __ldg(st.fb + q); },
                  [&](int q, const float4& r, int dx3, const float4& v) {
                      emit((int32_t)((uint32_t)(q - i) << 9) | tag | dx3);
                      const PairF<DIM, KK> p(r, S);
                      float dot = __fmaf_rn(__fsub_rn(vi.x, v.x), r.x, __fmul_rn(__fsub_rn(vi.y, v.y), r.y));
                      if (DIM == 3) dot = __fmaf_rn(__fsub_rn(vi.z, v.z), r.z, dot);
                      sum.add(__fmul_rn(__fmul_rn(v.w, p.F), dot));
                  });
}

// Whether every neighbour of particle i fits a list entry (23 bits of j - i).
template <int DIM>
__device__ __forceinline__ bool entries_fit(const SceneDev& S, const int32_t* __restrict__ start, const int32_t c[3],
                                            int i) {
    const int m = S.reach;
    const int zl = DIM == 3 ? max(c[2] - m, 0) : 0, zh = DIM == 3 ? min(c[2] + m, S.n[2] - 1) : 0;
    const int32_t* s = start + S.cell_off;
    const int lo = __ldg(s + (zl * S.n[1] + max(c[1] - m, 0)) * S.n[0]);
    const int hi = __ldg(s + (zh * S.n[1] + min(c[1] + m, S.n[1] - 1) + 1) * S.n[0]);
    return i - lo < kListDelta && hi - i < kListDelta;
}

// The density update and equation of state of particle i with its continuity sum.
template <int DIM, int KK>
__device__ __forceinline__ void continuity_update(const SceneDev& S, const SortedState& st, const BufferState& bf,
                                                  int i, float2 sum) {
    double dr = (double)sum.x - (double)sum.y;
    if (bf.n) {  // inlet/outlet buffer neighbours, FP64
        using V = typename VecT<DIM>::T;
        int32_t c[3];
        decode_cell(st.cell[i], S, c);
        dr += buffer_drho<DIM, KK>(S, bf, c, ((const V*)st.x)[i], ((const V*)st.v)[i]);
    }
    // Tait equation of state (UpdatePressure.jl:8-16) in FP64 with one reciprocal and plain
    // powers: the values feed FP32 pair terms (P) or FP64 sums (vol), where last-bit
    // differences from the reference's rounding do not show.
    const double m_i = st.m[i];
    const double rho = fma(dr, S.dt, st.rho[i]);
    const double inv_rho = rcp_rn_range(rho) ? rcp3(rho) : 1.0 / rho;
    const double rr = rho * S.inv_rho0;
    const double p = fma(S.b, powi_plain(rr, S.gamma) - 1.0, S.p0);
    const double cs =
        S.c0 * ((S.gamma & 1) ? powi_plain(rr, (S.gamma - 1) >> 1) : sqrt(powi_plain(rr, S.gamma - 1)));
    const double P = p * inv_rho * inv_rho;
    st.rhoc[i] = rho;
    st.p[i] = p;
    st.c[i] = cs;
    st.P[i] = P;
    st.vol[i] = m_i * inv_rho;
    *reinterpret_cast<float2*>(st.fc + i) = make_float2((float)rho, (float)P);
}

// Large scenes: one thread a particle.  A row's terms are one compensated sum and the rows'
// sums are merged in order; k_continuity_rows_f32 forms the same sums with a lane a row.  The
// next row's cell starts and the next candidate's data are loaded ahead.  22.2 -> 19.7 us on a
// 65,536-particle cavity, 170 -> 148 on a million particles (and momentum reads the list it
// records), 418 -> 349 on a 432,000-particle 3D dam break.
template <int DIM, int KK, int BLOCKS>
__global__ void __launch_bounds__(128, BLOCKS) k_continuity_f32(const SceneDev* __restrict__ scenes, SortedState st,
                                                        SortScratch sc, int32_t cap, BufferState bf, NbrList nl,
                                                        WallState wl) {
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cap || i >= *sc.n_live) return;
    const SceneDev& S = scenes[st.scene[i]];
    if (!scene_runs(S, sc.scene_step[st.scene[i]])) return;
    const float4 me = st.fa[i], vi = st.fb[i];
    int32_t c[3];
    decode_cell(st.cell[i], S, c);
    const int zr = DIM == 3 ? S.reach : 0;
    const bool prune = S.prune && !select_far(me);
    const bool fits = nl.e && entries_fit<DIM>(S, sc.start, c, i);
    const int room = fits ? nl.kmax : 0;
    int32_t* entry = nl.e + i;
    int cnt = 0;
    Kahan total;
    auto emit = [&](int32_t code) {
        if (cnt < room) {
            *entry = code;
            entry += nl.stride;
        }
        ++cnt;
    };
    int b, e, b2, e2;
    row_runs<DIM>(S, sc.start, c, me, prune, -S.reach, -zr, b, e, b2, e2);
#pragma unroll 1
    for (int dz = -zr; dz <= zr; ++dz) {
#pragma unroll 1
        for (int dy = -S.reach; dy <= S.reach; ++dy) {
            int nb, ne, nb2, ne2;  // the next row's runs, loaded before this row is walked
            const bool turn = dy == S.reach;
            row_runs<DIM>(S, sc.start, c, me, prune, turn ? -S.reach : dy + 1, turn ? (DIM == 3 ? dz + 1 : 4) : dz, nb,
                          ne, nb2, ne2);
            Kahan row;
            const int tag = (dz + 3) << 6 | (dy + 3) << 3;
#pragma unroll 1
            while (b < e) {
                run_pairs<DIM, KK>(S, st, i, me, vi, b, e, (float)dy, (float)dz, tag, row, emit);
                b = b2;
                e = e2;
                b2 = e2 = 0;
            }
            merge(total, row.s, row.c);
            b = nb;
            e = ne;
            b2 = nb2;
            e2 = ne2;
        }
    }
    const bool walk = !(fits && cnt <= room);
    if (nl.e) nl.n[i] = walk ? kListWalk : cnt;
    if (walk || (wl.n > 0 && wl.near[st.cell[i]])) sc.walked[atomicAdd(sc.n_walked, 1)] = i;
    continuity_update<DIM, KK>(S, st, bf, i, make_float2(total.s, total.c));
}

// Small scenes: eight lanes a particle, lane r the row dy = r - 3 of each plane, so the chain
// of loads a particle waits for is a row's instead of the whole stencil's (21.5 -> 7.4 us on a
// 5,000-particle dam break, 30.2 -> 10.5 on a 15,000-particle channel).  A block of 256
// threads takes 32 particles; its first warp updates them.  Where a thread a particle takes the
// momentum gather (threads), the particles it walks the cells for are listed as in
// k_continuity_f32.
template <int DIM, int KK>
__global__ void __launch_bounds__(256) k_continuity_rows_f32(const SceneDev* __restrict__ scenes, SortedState st,
                                                             SortScratch sc, int32_t cap, BufferState bf, NbrList nl,
                                                             WallState wl, bool threads) {
    pdl_wait();
    if (!threads) pdl_trigger();
    const unsigned full = 0xffffffffu;
    __shared__ int32_t rows[kRowEntries * 256];
    __shared__ float2 sums[32];
    const int g = threadIdx.x / kCoopLanes, lane = threadIdx.x % kCoopLanes;
    const int i0 = blockIdx.x * (blockDim.x / kCoopLanes);
    const int n = min(cap, *sc.n_live);
    if (i0 >= n) return;  // the whole block
    {
        const int i = min(i0 + g, n - 1);
        const SceneDev& S = scenes[st.scene[i]];
        const bool on = i0 + g < n && scene_runs(S, sc.scene_step[st.scene[i]]);
        const float4 me = st.fa[i], vi = st.fb[i];
        int32_t c[3];
        decode_cell(st.cell[i], S, c);
        const bool prune = S.prune && !select_far(me);
        bool fits = on && nl.e && entries_fit<DIM>(S, sc.start, c, i);
        int32_t* mine = rows + threadIdx.x;
        int count = 0;
        Kahan total;
        const int planes = DIM == 3 ? (int)__reduce_max_sync(full, (unsigned)S.reach) : 0;
        for (int dz = -planes; dz <= planes; ++dz) {
            const int dy = lane - 3;
            int b = 0, e = 0, b2 = 0, e2 = 0, cnt = 0;
            if (on && lane < 7) row_runs<DIM>(S, sc.start, c, me, prune, dy, dz, b, e, b2, e2);
            const int first = b, first_end = e, second = b2, second_end = e2;
            Kahan row;
            const int tag = (dz + 3) << 6 | lane << 3;
#pragma unroll 1
            while (b < e) {
                run_pairs<DIM, KK>(S, st, i, me, vi, b, e, (float)dy, (float)dz, tag, row, [&](int32_t code) {
                    if (cnt < kRowEntries) mine[cnt * 256] = code;
                    ++cnt;
                });
                b = b2;
                e = e2;
                b2 = e2 = 0;
            }
            __syncwarp(full);
#pragma unroll
            for (int r = 0; r < 7; ++r) {  // the rows' sums in order, in every lane
                const float s = __shfl_sync(full, row.s, r, kCoopLanes), k = __shfl_sync(full, row.c, r, kCoopLanes);
                merge(total, s, k);
            }
            int end = cnt;  // the places of the rows' entries in the list
#pragma unroll
            for (int o = 1; o < kCoopLanes; o <<= 1) {
                const int v = __shfl_up_sync(full, end, o, kCoopLanes);
                if (lane >= o) end += v;
            }
            const int all = __shfl_sync(full, end, kCoopLanes - 1, kCoopLanes);
            fits &= count + all <= nl.kmax;
            if (fits) {
                int32_t* entry = nl.e + (int64_t)(count + end - cnt) * nl.stride + i;
                if (cnt <= kRowEntries) {
                    for (int q = 0; q < cnt; ++q, entry += nl.stride) *entry = mine[q * 256];
                } else {  // a long row (wide cells, or a spacing far below r_cut): walked again
                    auto list_run = [&](int j, int e) {
                        run_walk<DIM>(S, st.fa, i, me, j, e, (float)dy, (float)dz, [](int) { return 0; },
                                      [&](int q, const float4&, int dx3, int) {
                                          *entry = (int32_t)((uint32_t)(q - i) << 9) | tag | dx3;
                                          entry += nl.stride;
                                      });
                    };
                    list_run(first, first_end);
                    list_run(second, second_end);
                }
            }
            count += all;
        }
        if (lane == 0) {
            sums[g] = make_float2(total.s, total.c);
            if (on && nl.e) nl.n[i] = fits ? count : kListWalk;
            if (threads && on && (!fits || (wl.n > 0 && wl.near[st.cell[i]])))
                sc.walked[atomicAdd(sc.n_walked, 1)] = i;
        }
    }
    __syncthreads();
    const int i = i0 + threadIdx.x;
    if (threadIdx.x >= blockDim.x / kCoopLanes || i >= n) return;
    const SceneDev& S = scenes[st.scene[i]];
    if (!scene_runs(S, sc.scene_step[st.scene[i]])) return;
    continuity_update<DIM, KK>(S, st, bf, i, sums[threadIdx.x]);
}

// -------------------------------------------------------------------- K5 (FP32)
// A particle's own FP32 values in the momentum terms.
struct SelfF {
    float4 x, v, f;  // select_pos; (velocity, m kg_a / h); (rho, P, T, kappa)
    float inv_cp2;   // 2 / cp
    float tens;      // 0.01 kw_a / W(gap_i)
    double gap;      // read when the gaps differ
};
// The sums of a particle or of one of its lanes.
template <int DIM, bool HEAT>
struct SumsF {
    Kahan dv[DIM], dT;
    __device__ __forceinline__ void add(const float t[DIM + 1]) {
#pragma unroll
        for (int k = 0; k < DIM; ++k) dv[k].add(t[k]);
        if (HEAT) dT.add(t[DIM]);
    }
    __device__ __forceinline__ void merge_in(const SumsF& o) {
#pragma unroll
        for (int k = 0; k < DIM; ++k) merge(dv[k], o.dv[k].s, o.dv[k].c);
        if (HEAT) merge(dT, o.dT.s, o.dT.c);
    }
};

template <int DIM, int KK, bool HEAT>
__device__ __forceinline__ SelfF self_f(const SceneDev& S, const SortedState& st, int i) {
    SelfF a;
    a.x = st.fa[i];
    a.v = st.fb[i];
    a.f = st.fc[i];
    a.inv_cp2 = HEAT ? 2.f / (float)st.cp[i] : 0.f;
    a.gap = 0.0;
    a.tens = S.tens_f;
    if (!S.uniform_gap) {
        a.gap = st.gap[i];
        a.tens = 0.01f / kernel_w_f<KK>((float)a.gap * S.inv_h_f);
    }
    return a;
}

// Terms of a fluid pair: acceleration t[0 .. DIM-1] and heating t[DIM]; returns w (W / kw_a).
// Pressure with its tensile part (PressureForce.jl:14-19), viscosity (ViscosityForce.jl:15-23;
// mu_i + mu_j = nu0 (rho_i + rho_j)), heat (ThermalConduction.jl:15-21).
template <int DIM, int KK, bool HEAT>
__device__ __forceinline__ float pair_terms(const SceneDev& S, const SortedState& st, const SelfF& a, const float4& r,
                                            const float4& vj, const float4& fj, float t[DIM + 1]) {
    const PairF<DIM, KK> p(r, S);
    float prho2 = __fadd_rn(a.f.y, fj.y);
    const float tens =
        S.uniform_gap ? S.tens_f : 0.01f / kernel_w_f<KK>((float)(0.5 * (a.gap + st.gap[p.j])) * S.inv_h_f);
    prho2 = __fmaf_rn(__fmul_rn(fabsf(prho2), p.w), tens, prho2);
    const float mF = __fmul_rn(vj.w, p.F);
    const float dh = __fadd_rn(p.d2, S.hh001_f);
    const float mFd = __fmul_rn(mF, p.d2);
    const float gp = -__fmul_rn(mF, prho2);
    const float gv = div_ftz(__fmul_rn(mFd, S.nu4_f), __fmul_rn(__fadd_rn(a.f.x, fj.x), dh));
    t[0] = __fmaf_rn(gp, p.r[0], __fmul_rn(gv, __fsub_rn(a.v.x, vj.x)));
    t[1] = __fmaf_rn(gp, p.r[1], __fmul_rn(gv, __fsub_rn(a.v.y, vj.y)));
    if (DIM == 3) t[DIM - 1] = __fmaf_rn(gp, p.r[2], __fmul_rn(gv, __fsub_rn(a.v.z, vj.z)));
    if (HEAT) {
        const float keq = div_ftz(__fmul_rn(2.f, __fmul_rn(a.f.w, fj.w)), __fadd_rn(a.f.w, fj.w));
        const float h = div_ftz(__fmul_rn(mFd, keq), __fmul_rn(__fmul_rn(a.f.x, fj.x), dh));
        t[DIM] = __fmul_rn(__fmul_rn(h, __fsub_rn(a.f.z, fj.z)), a.inv_cp2);
    }
    return p.w;
}

// A neighbour's terms of the Shepard sums (ReconstructValue.jl:28-50), FP64; w = W / kw_a.
__device__ __forceinline__ void shepard_terms(const SceneDev& S, float w, double vol, double m, double& sw, double& sws) {
    const double W = widen(__fmul_rn(S.kw_a_f, w));
    sw = fma(W, vol, sw);
    sws = fma(W, m, sws);
}

// Terms of a wall pair: the compulsive force (WallForce.jl:15-28), background pressure
// (PressureForce.jl:29-33), viscosity (ViscosityForce.jl:34-44), heat (ThermalConduction.jl:
// 31-35).
template <int DIM, int KK, int MODE>
__device__ __forceinline__ void wall_terms(const SceneDev& S, const WallState& wl, const SelfF& a, float c_i,
                                           const float4& r, float t[DIM + 1]) {
    constexpr bool HEAT = MODE == kModeThermal;
    const PairF<DIM, KK> p(r, S);
    const float4 wn = wl.fb[p.j], wv = wl.fc[p.j];  // (normal, gap), (velocity, T)
    const float gw = wn.w;
    const float v0 = __fsub_rn(a.v.x, wv.x), v1 = __fsub_rn(a.v.y, wv.y), v2 = DIM == 3 ? __fsub_rn(a.v.z, wv.z) : 0.f;
    float vert = __fmaf_rn(v0, wn.x, __fmul_rn(v1, wn.y)), psi = __fmaf_rn(p.r[0], wn.x, __fmul_rn(p.r[1], wn.y));
    if (DIM == 3) {
        vert = __fmaf_rn(v2, wn.z, vert);
        psi = __fmaf_rn(p.r[2], wn.z, psi);
    }
    psi = fabsf(psi);
    float wf = 0.f;
    const float along = sqrtf(fmaxf(__fmaf_rn(-psi, psi, p.d2), 0.f));
    const float q = psi / gw;
    if (!(q > 1.f || along > gw)) {
        const float pxi = fabsf(__fmul_rn(__fadd_rn(1.f, cospif(along / gw)), 0.5f));
        const float beta = vert > 0.f ? 0.f : c_i;
        wf = __fmul_rn(__fmul_rn(__fmul_rn(__fmaf_rn(beta, fabsf(vert), __fmul_rn(0.01f, __fmul_rn(c_i, c_i))), S.inv_h_f),
                                 fabsf(__fsub_rn(1.f, q))),
                       __fmul_rn(rsqrtf(q), pxi));
    }
    const float mF = __fmul_rn(a.v.w, p.F);
    float gp = 0.f;
    if (MODE == kModeWallPressure || HEAT) {
        const float pw = __fadd_rn(a.f.y, S.P_bg_f);
        gp = -__fmul_rn(__fmaf_rn(__fmul_rn(fabsf(pw), p.w), a.tens, pw), mF);
    }
    const float mFd = __fmul_rn(mF, p.d2);
    const float den = __fmul_rn(a.f.x, __fadd_rn(p.d2, S.hh001_f));
    const float gv = div_ftz(__fmul_rn(__fmul_rn(0.5f, S.nu4_f), mFd), den);
    const float along_n = __fmaf_rn(-gv, vert, wf);
    t[0] = __fmaf_rn(along_n, wn.x, __fmaf_rn(gp, p.r[0], __fmul_rn(gv, v0)));
    t[1] = __fmaf_rn(along_n, wn.y, __fmaf_rn(gp, p.r[1], __fmul_rn(gv, v1)));
    if (DIM == 3) t[DIM - 1] = __fmaf_rn(along_n, wn.z, __fmaf_rn(gp, p.r[2], __fmul_rn(gv, v2)));
    if (HEAT) {
        t[DIM] = 0.f;
        if (wl.kind[p.j] == SPH_WALL_THERMOSTATIC) {
            const float k = __fmul_rn(__fmul_rn(S.inv_cp_f, __fadd_rn(a.f.w, wl.fk[p.j])), S.inv_rho0_f);
            t[DIM] = __fmul_rn(div_ftz(__fmul_rn(k, mFd), den), __fsub_rn(a.f.z, wv.w));
        }
    }
}

// The cell walks of the momentum gather: the walls, and the fluid of a particle whose list did
// not fit (`walk`).  The eight lanes of a group walk for its particle i, lane r the rows
// dy = r - 3 of every plane, and merge their sums in order: every lane of the group ends with
// `fluid` and `wall` whole.  shepard(w, j) takes a fluid neighbour's Shepard terms.  All lanes
// of the warp call this together.
template <int DIM, int KK, int MODE, typename Shepard>
__device__ __forceinline__ void coop_rows(const SceneDev& S, const SortedState& st, const WallState& wl,
                                          const int32_t* __restrict__ start, int i, const SelfF& a, bool walk,
                                          bool walls, SumsF<DIM, MODE == kModeThermal>& fluid,
                                          SumsF<DIM, MODE == kModeThermal>& wall, Shepard&& shepard) {
    constexpr bool HEAT = MODE == kModeThermal;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & (kCoopLanes - 1), dy = lane - 3;
    int32_t c[3];
    decode_cell(st.cell[i], S, c);
    const bool prune = S.prune && !select_far(a.x);
    const float c_i = (float)st.c[i];
    const int planes = DIM == 3 ? (int)__reduce_max_sync(full, walk || walls ? (unsigned)S.reach : 0u) : 0;
    const bool any_walk = __any_sync(full, walk), any_walls = __any_sync(full, walls);
    auto rows = [&](const int32_t* starts, const float4* pos, int self, int dz, auto&& term) {
        int b, e, b2, e2;
        row_runs<DIM>(S, starts, c, a.x, prune, dy, dz, b, e, b2, e2);
#pragma unroll 1
        while (b < e) {
            run_walk<DIM>(S, pos, self, a.x, b, e, (float)dy, (float)dz, [](int) { return 0; },
                          [&](int j, const float4& r, int, int) { term(j, r); });
            b = b2;
            e = e2;
            b2 = e2 = 0;
        }
    };
#pragma unroll 1
    for (int dz = -planes; dz <= planes; ++dz) {
        if (any_walk && walk && lane < 7)
            rows(start, st.fa, i, dz, [&](int j, const float4& r) {
                float t[DIM + 1];
                shepard(pair_terms<DIM, KK, HEAT>(S, st, a, r, st.fb[j], st.fc[j], t), j);
                fluid.add(t);
            });
        if (any_walls && walls && lane < 7)
            rows(wl.start, wl.fa, -1, dz, [&](int, const float4& r) {
                float t[DIM + 1];
                wall_terms<DIM, KK, MODE>(S, wl, a, c_i, r, t);
                wall.add(t);
            });
    }
    __syncwarp(full);
    auto merged = [&](Kahan& k) {
        Kahan m;
#pragma unroll
        for (int r = 0; r < 7; ++r)
            merge(m, __shfl_sync(full, k.s, r, kCoopLanes), __shfl_sync(full, k.c, r, kCoopLanes));
        k = m;
    };
    auto merge_all = [&](SumsF<DIM, HEAT>& s) {
#pragma unroll
        for (int k = 0; k < DIM; ++k) merged(s.dv[k]);
        if (HEAT) merged(s.dT);
    };
    if (any_walk) merge_all(fluid);
    if (any_walls) merge_all(wall);
}

// The update of particle i with its sums: FP64 forward Euler on the masters
// (UpdateTemperature/Velocity/Position.jl), the re-initialised density with the particle's
// own W(0) term (SHEP; ReconstructValue.jl:51-55), the out-of-domain check and the next
// step's cell arrival.
template <int DIM, int KK, int MODE, bool SHEP>
__device__ __forceinline__ void momentum_update(const SceneDev& S, const SortedState& st, const NextState& nx,
                                                const SortScratch& sc, const BufferState& bf, const BufferScratch& bs,
                                                const BufferRules& br, int i, int64_t step,
                                                const SumsF<DIM, MODE == kModeThermal>& sum, double sw, double sws) {
    using V = typename VecT<DIM>::T;
    constexpr bool HEAT = MODE == kModeThermal;
    double dvd[DIM];
#pragma unroll
    for (int k = 0; k < DIM; ++k) dvd[k] = (double)sum.dv[k].s - (double)sum.dv[k].c;
    const double dTd = HEAT ? (double)sum.dT.s - (double)sum.dT.c : 0.0;
    const V x0 = ((const V*)st.x)[i];
    const V v0 = ((const V*)st.v)[i];
    const double rho_d = st.rhoc[i];
    if (MODE == kModeBuffers && bf.n) {  // inlet/outlet buffer neighbours, FP64
        const double gap_d = st.gap[i];
        int32_t c[3];
        decode_cell(st.cell[i], S, c);
        buffer_dv<DIM, KK>(S, bf, c, x0, v0, rho_d, st.P[i], gap_d, kernel_w<KK>(gap_d, S), S.nu0 * rho_d, dvd);
    }
    const double dt = S.dt;
    double body[DIM];
    if (HEAT) {
        const double Tn = fma(dt, dTd, st.T[i]);
#pragma unroll
        for (int k = 0; k < DIM; ++k) body[k] = S.bous[k] * (Tn - S.t0);
        nx.T[i] = Tn;
    } else {
        if (nx.T) nx.T[i] = st.T[i];
#pragma unroll
        for (int k = 0; k < DIM; ++k) body[k] = S.g[k];
    }
    double vn[DIM], xn[DIM];
    vn[0] = v0.x; vn[1] = v0.y;
    xn[0] = x0.x; xn[1] = x0.y;
    if (DIM == 3) {
        vn[DIM - 1] = comp(v0, DIM - 1);
        xn[DIM - 1] = comp(x0, DIM - 1);
    }
#pragma unroll
    for (int k = 0; k < DIM; ++k) {
        vn[k] += body[k] * dt;
        vn[k] += dvd[k] * dt;
        xn[k] += vn[k] * dt - dvd[k] * S.half_dtdt;  // dv dt^2 / 2
    }
    if (S.periodic_x) {
        if (xn[0] >= S.wrap_hi) xn[0] -= S.period;
        else if (xn[0] < S.lo[0]) xn[0] += S.period;
    }
    V xo, vo;
    xo.x = xn[0]; xo.y = xn[1];
    vo.x = vn[0]; vo.y = vn[1];
    if constexpr (DIM == 3) {
        xo.z = xn[2]; xo.w = 0.0;
        vo.z = vn[2]; vo.w = 0.0;
    }
    ((V*)nx.x)[i] = xo;
    ((V*)nx.v)[i] = vo;
    if constexpr (SHEP) {  // with the particle's own W(0) term (ReconstructValue.jl:51-55)
        nx.rho[i] = (sws + S.k0 * st.m[i]) / (sw + S.k0 * st.vol[i]);
    } else {
        nx.rho[i] = rho_d;
    }

    bool finite = bits_finite(rho_d);
#pragma unroll
    for (int k = 0; k < DIM; ++k) finite &= bits_finite(xn[k]) & bits_finite(vn[k]);
    if (!finite && S.nan_check) atomicOr(sc.status, kStatusNonFinite);
    bool dead = false;
    if (S.check_enabled && is_step(step, S.check_interval)) {
#pragma unroll
        for (int k = 0; k < DIM; ++k) dead |= (xn[k] > S.check_hi[k]) | (xn[k] < S.check_lo[k]);
    }
    if (dead) {
        sc.key[i] = kDeadKey;
    } else if (MODE == kModeBuffers && bs.npend && beyond_plane<DIM>(br.out_n, br.out_d, xn)) {
        // outlet_out_calculation_domain_check: leaves the fluid, joins the outlet
        sc.key[i] = kDeadKey;
        const int32_t k = atomicAdd(bs.npend, 1);
        if (k < bs.cap) bs.pend[k] = i;
        else atomicOr(sc.status, kStatusBufferOverflow);
    } else {
        cell_arrival(sc, i, moved_key<DIM>(st.cell[i], st.fa[i], x0, xo, S));
    }
}

// A particle takes part in a momentum launch (SHEP: of re-initialisation steps) when its
// scene runs and its step is of the launch's kind; `sel`: with SHEP, every running scene;
// without, the re-initialising scenes are left to the SHEP launch of the same step (a batch
// whose scenes re-initialise at different steps runs both): every particle goes through the
// kernel of its own scene's step kind, so a scene's result does not depend on its batch.
template <bool SHEP>
__device__ __forceinline__ bool takes_part(const SceneDev& S, int64_t step, int sel) {
    const bool runs = scene_runs(S, step);
    if (SHEP) return runs && (sel || is_step(step, S.reinit_interval));
    return runs && !(sel && is_step(step, S.reinit_interval));
}

// Large scenes, the cell walks: eight lanes for each particle that continuity listed as
// walked (near a wall, or without a list; in any order), their sums into sc.walk_sums for
// k_momentum_f32.  Walked by that kernel's own threads, a wall cost every lane of a warp with
// one particle near it, and half the time of a 3D dam break's momentum gather.
template <int DIM, int KK, int MODE, bool SHEP>
__global__ void __launch_bounds__(256, DIM == 3 ? 3 : 4)
    k_walks_f32(const SceneDev* __restrict__ scenes, SortedState st, WallState wl, SortScratch sc, NbrList nl, int sel) {
    pdl_wait();
    pdl_trigger();  // k_momentum_f32 takes its lists meanwhile: it needs the walks' sums last
    constexpr bool HEAT = MODE == kModeThermal;
    constexpr int kSums = DIM + (HEAT ? 1 : 0);
    const int n = *sc.n_walked, lane = threadIdx.x % kCoopLanes;
    const int stride = gridDim.x * (blockDim.x / kCoopLanes);
    for (int q0 = (blockIdx.x * blockDim.x + (threadIdx.x & ~31)) / kCoopLanes; q0 < n; q0 += stride) {
        const int q = q0 + (threadIdx.x & 31) / kCoopLanes;
        const int i = sc.walked[min(q, n - 1)];
        const SceneDev& S = scenes[st.scene[i]];
        const bool on = q < n && takes_part<SHEP>(S, sc.scene_step[st.scene[i]], sel);
        const bool walk = on && (!nl.e || nl.n[i] == kListWalk), walls = on && wl.n > 0 && wl.near[st.cell[i]];
        SumsF<DIM, HEAT> fluid, wall;
        double sw = 0.0, sws = 0.0;
        coop_rows<DIM, KK, MODE>(S, st, wl, sc.start, i, self_f<DIM, KK, HEAT>(S, st, i), walk, walls, fluid, wall,
                                 [&](float wk, int j) { if constexpr (SHEP) shepard_terms(S, wk, st.vol[j], st.m[j], sw, sws); });
        if constexpr (SHEP) {
            sw = coop_sum(sw);
            sws = coop_sum(sws);
        }
        if (on && lane == 0) {
            float2* out = sc.walk_sums + (int64_t)i * (2 * kSums + 2);
#pragma unroll
            for (int k = 0; k < DIM; ++k) {
                out[k] = make_float2(fluid.dv[k].s, fluid.dv[k].c);
                out[kSums + k] = make_float2(wall.dv[k].s, wall.dv[k].c);
            }
            if (HEAT) {
                out[DIM] = make_float2(fluid.dT.s, fluid.dT.c);
                out[kSums + DIM] = make_float2(wall.dT.s, wall.dT.c);
            }
            if constexpr (SHEP) {
                reinterpret_cast<double*>(out)[2 * kSums] = sw;
                reinterpret_cast<double*>(out)[2 * kSums + 1] = sws;
            }
        }
    }
}

// Large scenes: one thread a particle.  Eight sums take the entries of the list in turns, as
// the lanes of k_momentum_lanes_f32 do, so both give the same bits; a warp's threads read the
// same entry of 32 consecutive particles, whose neighbours lie side by side.  It runs beside
// k_walks_f32, which starts it once continuity's results are visible, and waits for it where it
// needs the walks' sums and before it writes anything (every thread waits: the grid must not
// end before the walks).  Both together against one after the other: 17.0 against 24.1 us on
// a 65,536-particle cavity (54 -> 47 us a step), 216 against 228 on a million particles,
// 315 against 330 on a 432,000-particle 3D dam break (before the eight sums: 25.7, 254, 488).
// The Shepard sums are one FP64 sum each, in the list's order: 285 us with them at a million
// particles, 409 on the 3D dam break (eight sums each, in a second pass over the list: 385 and
// 633; before: 330 and 533).  A neighbour's volume and mass are loaded with its other values
// (415 us in 3D against 457), and its kernel value is widened without the FP64 unit, which the
// sums keep busy (285 against 315 us).
template <int DIM, int KK, int MODE, bool SHEP>
__global__ void __launch_bounds__(128, 4)
    k_momentum_f32(const SceneDev* __restrict__ scenes, SortedState st, NextState nx, WallState wl, SortScratch sc,
                   int32_t cap, BufferState bf, BufferScratch bs, BufferRules br, NbrList nl, int sel) {
    constexpr bool HEAT = MODE == kModeThermal;
    constexpr int kSums = DIM + (HEAT ? 1 : 0);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cap || i >= *sc.n_live) {
        pdl_wait();
        return;
    }
    const SceneDev& S = scenes[st.scene[i]];
    const int64_t step = sc.scene_step[st.scene[i]];
    if (!takes_part<SHEP>(S, step, sel)) {
        pdl_wait();
        if (!SHEP && !scene_runs(S, step)) carry_frozen<DIM>(i, S, st, nx, sc);
        return;
    }
    const SelfF a = self_f<DIM, KK, HEAT>(S, st, i);
    const int count = nl.e ? nl.n[i] : kListWalk;
    SumsF<DIM, HEAT> acc[kCoopLanes];
    double sw = 0.0, sws = 0.0;  // Shepard sums, in the list's order
    if (count != kListWalk) {
        // the next eight entries are loaded before the current eight are processed
        const int32_t* entry = nl.e + i;
        const int64_t stride = nl.stride;
        int32_t next[kCoopLanes];
#pragma unroll
        for (int u = 0; u < kCoopLanes; ++u) next[u] = u < count ? __ldg(entry + u * stride) : 0;
#pragma unroll 1
        for (int k = 0; k < count; k += kCoopLanes) {
            int32_t code[kCoopLanes];
#pragma unroll
            for (int u = 0; u < kCoopLanes; ++u) {
                code[u] = next[u];
                next[u] = k + kCoopLanes + u < count ? __ldg(entry + (k + kCoopLanes + u) * stride) : 0;
            }
#pragma unroll
            for (int u = 0; u < kCoopLanes; ++u) {
                const int j = i + (code[u] >> 9);
                const float4 r = listed<DIM>(code[u], a.x, __ldg(st.fa + j), j, S);
                double vol = 0.0, m = 0.0;
                if constexpr (SHEP) {
                    vol = __ldg(st.vol + j);
                    m = __ldg(st.m + j);
                }
                float t[DIM + 1];
                const float w = pair_terms<DIM, KK, HEAT>(S, st, a, r, __ldg(st.fb + j), __ldg(st.fc + j), t);
                if (k + u < count) {
                    acc[u].add(t);
                    if constexpr (SHEP) shepard_terms(S, w, vol, m, sw, sws);
                }
            }
        }
    }
#pragma unroll
    for (int u = 1; u < kCoopLanes; ++u) acc[0].merge_in(acc[u]);
    pdl_wait();
    if (count == kListWalk || (wl.n > 0 && wl.near[st.cell[i]])) {  // the cell walks (k_walks_f32)
        const float2* in = sc.walk_sums + (int64_t)i * (2 * kSums + 2);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int k = 0; k < DIM; ++k) merge(acc[0].dv[k], in[h * kSums + k].x, in[h * kSums + k].y);
            if (HEAT) merge(acc[0].dT, in[h * kSums + DIM].x, in[h * kSums + DIM].y);
        }
        if (SHEP && count == kListWalk) {
            sw = reinterpret_cast<const double*>(in)[2 * kSums];
            sws = reinterpret_cast<const double*>(in)[2 * kSums + 1];
        }
    }
    momentum_update<DIM, KK, MODE, SHEP>(S, st, nx, sc, bf, bs, br, i, step, acc[0], sw, sws);
}

// Small scenes: eight lanes a particle, lane t the
// entries t, t + 8, ... of its list, or a neighbour row of the walls (and of the fluid, for a
// particle whose list did not fit).  A block of 256 threads takes 32 particles; its first
// warp merges the lanes' sums and updates the particles (30.6 -> 9.1 us on a 5,000-particle dam
// break, 23.9 -> 11.3 on a 15,000-particle channel; a million particles would take 473 us, a
// thread each 216).  Continuity starts it early: the
// chain of loads to a particle's scene and own values is then over when the lists are there
// (a step of a 5,000-particle dam break 23.5 -> 22.7 us).
template <int DIM, int KK, int MODE, bool SHEP>
__global__ void __launch_bounds__(256, DIM == 3 ? 3 : 4)
    k_momentum_lanes_f32(const SceneDev* __restrict__ scenes, SortedState st, NextState nx, WallState wl,
                         SortScratch sc, int32_t cap, BufferState bf, BufferScratch bs, BufferRules br, NbrList nl,
                         int sel) {
    constexpr bool HEAT = MODE == kModeThermal;
    constexpr int kSums = DIM + (HEAT ? 1 : 0), kParts = kCoopLanes + 1;
    const unsigned full = 0xffffffffu;
    __shared__ float2 sums[kSums * kParts * kSumStride];
    __shared__ double shep[SHEP ? 64 : 1];
    const int g = threadIdx.x / kCoopLanes, lane = threadIdx.x % kCoopLanes;
    const int i0 = blockIdx.x * (blockDim.x / kCoopLanes);
    const int n = min(cap, *sc.n_live);
    if (i0 >= n) {  // the whole block
        pdl_wait();
        return;
    }
    {
        // what continuity does not write is loaded before the wait
        const int i = min(i0 + g, n - 1);
        const SceneDev& S = scenes[st.scene[i]];
        const bool on = i0 + g < n && takes_part<SHEP>(S, sc.scene_step[st.scene[i]], sel);
        const bool walls = on && wl.n > 0 && wl.near[st.cell[i]];
        SelfF a = self_f<DIM, KK, HEAT>(S, st, i);
        pdl_wait();
        a.f = st.fc[i];
        SumsF<DIM, HEAT> sum;
        double sw = 0.0, sws = 0.0;  // Shepard sums of a walked particle, by lane
        const int count = on ? (nl.e ? nl.n[i] : kListWalk) : 0;
        auto shepard = [&](float w, int j) { if constexpr (SHEP) shepard_terms(S, w, st.vol[j], st.m[j], sw, sws); };
        if (count != kListWalk && lane < count) {
            // the entry two rounds ahead and the neighbour one round ahead are loaded before the
            // current pair is processed
            const int32_t* entry = nl.e + i + lane * nl.stride;
            const int64_t ahead = kCoopLanes * nl.stride;
            int32_t code = __ldg(entry), next = 0;
            if (lane + kCoopLanes < count) next = __ldg(entry += ahead);
            int j = i + (code >> 9);
            float4 p = __ldg(st.fa + j), v = __ldg(st.fb + j), f = __ldg(st.fc + j);
            for (int k = lane;;) {
                const bool more = k + kCoopLanes < count;
                const float4 r = listed<DIM>(code, a.x, p, j, S);
                const float4 vj = v, fj = f;
                if (more) {
                    code = next;
                    j = i + (code >> 9);
                    p = __ldg(st.fa + j);
                    v = __ldg(st.fb + j);
                    f = __ldg(st.fc + j);
                    if (k + 2 * kCoopLanes < count) next = __ldg(entry += ahead);
                }
                float t[DIM + 1];
                pair_terms<DIM, KK, HEAT>(S, st, a, r, vj, fj, t);
                sum.add(t);
                if (!more) break;
                k += kCoopLanes;
            }
        }
        __syncwarp(full);
        const bool walk = count == kListWalk;
        SumsF<DIM, HEAT> wall;
        if (__any_sync(full, walk || walls)) {
            SumsF<DIM, HEAT> fluid;
            coop_rows<DIM, KK, MODE>(S, st, wl, sc.start, i, a, walk, walls, fluid, wall, shepard);
            if (walk && lane == 0) sum = fluid;
        }
        if constexpr (SHEP) {
            // in the list's order, as a thread of k_momentum_f32 adds them: the lanes form eight
            // kernel values, lane 0 adds W vol and lane 1 W m
            const int entries = walk ? 0 : count;
            const int most = (int)__reduce_max_sync(full, (unsigned)entries);
            double s = 0.0;
            for (int k0 = 0; k0 < most; k0 += kCoopLanes) {
                const int k = k0 + lane;
                const int32_t code = k < entries ? __ldg(nl.e + i + k * nl.stride) : 0;
                const int j = i + (code >> 9);
                const PairF<DIM, KK> p(listed<DIM>(code, a.x, __ldg(st.fa + j), j, S), S);
                const double W = widen(__fmul_rn(S.kw_a_f, p.w)), vol = st.vol[j], m = st.m[j];
#pragma unroll
                for (int e = 0; e < kCoopLanes; ++e) {
                    const double We = __shfl_sync(full, W, e, kCoopLanes), ve = __shfl_sync(full, vol, e, kCoopLanes),
                                 me = __shfl_sync(full, m, e, kCoopLanes);
                    if (k0 + e < entries) s = fma(We, lane == 1 ? me : ve, s);
                }
            }
            const double lw = __shfl_sync(full, s, 0, kCoopLanes), lws = __shfl_sync(full, s, 1, kCoopLanes);
            sw = coop_sum(sw);
            sws = coop_sum(sws);
            if (!walk) {
                sw = lw;
                sws = lws;
            }
        }
#pragma unroll
        for (int k = 0; k < DIM; ++k) sums[(k * kParts + lane) * kSumStride + g] = make_float2(sum.dv[k].s, sum.dv[k].c);
        if (HEAT) sums[(DIM * kParts + lane) * kSumStride + g] = make_float2(sum.dT.s, sum.dT.c);
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < DIM; ++k)
                sums[(k * kParts + kCoopLanes) * kSumStride + g] = make_float2(wall.dv[k].s, wall.dv[k].c);
            if (HEAT) sums[(DIM * kParts + kCoopLanes) * kSumStride + g] = make_float2(wall.dT.s, wall.dT.c);
            if constexpr (SHEP) {
                shep[g] = sw;
                shep[32 + g] = sws;
            }
        }
    }
    __syncthreads();
    const int i = i0 + threadIdx.x;
    if (threadIdx.x >= blockDim.x / kCoopLanes || i >= n) return;
    const SceneDev& S = scenes[st.scene[i]];
    const int64_t step = sc.scene_step[st.scene[i]];
    if (!takes_part<SHEP>(S, step, sel)) {
        if (!SHEP && !scene_runs(S, step)) carry_frozen<DIM>(i, S, st, nx, sc);
        return;
    }
    auto merged = [&](int k) {
        const float2* q = sums + k * kParts * kSumStride + threadIdx.x;
        Kahan t;
        t.s = q[0].x;
        t.c = q[0].y;
#pragma unroll
        for (int l = 1; l < kParts; ++l) merge(t, q[l * kSumStride].x, q[l * kSumStride].y);
        return t;
    };
    SumsF<DIM, HEAT> sum;
#pragma unroll
    for (int k = 0; k < DIM; ++k) sum.dv[k] = merged(k);
    if (HEAT) sum.dT = merged(DIM);
    momentum_update<DIM, KK, MODE, SHEP>(S, st, nx, sc, bf, bs, br, i, step, sum, SHEP ? shep[threadIdx.x] : 0.0,
                                         SHEP ? shep[32 + threadIdx.x] : 0.0);
}

// -------------------------------------------------------------------- launchers
// Continuity takes a lane a row up to two waves of its blocks of 32 particles (four resident an
// SM) and a thread a particle beyond.  The chain of a thread takes the same time however few
// particles there are, the rows the longer the more waves they come in: 2D cavities of 10,000,
// 29,900, 39,600 and 50,200 particles take 9, 17, 22 and 26 us in rows and 18, 20, 20 and 22 us
// in threads, 3D dam breaks of 9,700, 38,700 and 53,200 particles 24, 67 and 113 us against 73,
// 77 and 77.
constexpr int64_t kRowsUpTo = 2 * 152 * 4 * 32;
// Continuity's thread kernel takes 72 registers, seven blocks of 128 an SM; held to 56 (2D: nine
// blocks) or 64 (3D: eight) it spills a little and is the faster one where that saves a wave:
// cavities of 144,400 and 1,048,576 particles 36 -> 26 and 163 -> 147 us, 3D dam breaks of 432,000
// particles 359 -> 348.  With as many waves either way it is not: a step of 202,500 particles
// 101.2 us against 102.0, of 250,000 in 3D 466 against 469.  Ten (nine) blocks: 158 (352).
// (Without the bound of seven the compiler takes more registers: 360,000 particles 72 us, not 62.)
constexpr int kSpread = 7;
template <int DIM>
constexpr int kPacked = DIM == 3 ? 8 : 9;
template <int DIM>
bool continuity_packed(int64_t blocks) {
    auto waves = [&](int64_t an_sm) { return (blocks + 152 * an_sm - 1) / (152 * an_sm); };
    return waves(kPacked<DIM>) < waves(kSpread);
}
// Momentum takes eight lanes a particle while their blocks of 32 particles are all resident at
// once (four an SM in 2D, three in 3D), a thread a particle beyond: cavities of 10,000, 15,100
// and 19,900 particles 12.2, 13.5 and 18.9 us in lanes and 13.1, 12.9 and 13.4 us in threads, 3D
// dam breaks of 9,700, 15,000 and 21,900 particles 31, 43 and 53 us against 33, 35 and 36.
template <int DIM>
constexpr int64_t kMomentumLanesUpTo = 152 * 32 * (DIM == 3 ? 3 : 4);
template <int DIM>
bool momentum_lanes(const LaunchCtx& L) {
    return L.lanes[1] < 0 ? L.cap <= kMomentumLanesUpTo<DIM> : L.lanes[1] != 0;
}

template <int DIM, int KK, int MODE>
void launch_momentum(const LaunchCtx& L) {
    const int sel = L.shepard ? L.force_reinit : L.skip_reinit;
    if (momentum_lanes<DIM>(L)) {
        auto kernel = L.shepard ? k_momentum_lanes_f32<DIM, KK, MODE, true> : k_momentum_lanes_f32<DIM, KK, MODE, false>;
        launch_dep(kernel, (L.cap + 31) / 32, 256, L.stream, L.scenes, L.st, L.nx, L.wl, L.sc, L.cap, L.bf, L.bs, L.br,
                   L.nl, sel);
        return;
    }
    auto walks = L.shepard ? k_walks_f32<DIM, KK, MODE, true> : k_walks_f32<DIM, KK, MODE, false>;
    launch_dep(walks, 152 * 3, 256, L.stream, L.scenes, L.st, L.wl, L.sc, L.nl, sel);
    auto kernel = L.shepard ? k_momentum_f32<DIM, KK, MODE, true> : k_momentum_f32<DIM, KK, MODE, false>;
    launch_dep(kernel, (L.cap + 127) / 128, 128, L.stream, L.scenes, L.st, L.nx, L.wl, L.sc, L.cap, L.bf, L.bs, L.br,
               L.nl, sel);
}

template <int DIM, int KK>
void launch_kk(int stage, const LaunchCtx& L) {
    if (stage == 0) {
        if (L.lanes[0] < 0 ? L.cap <= kRowsUpTo : L.lanes[0])
            launch_dep(k_continuity_rows_f32<DIM, KK>, (L.cap + 31) / 32, 256, L.stream, L.scenes, L.st, L.sc, L.cap,
                       L.bf, L.nl, L.wl, !momentum_lanes<DIM>(L));
        else
            launch_dep(continuity_packed<DIM>((L.cap + 127) / 128) ? k_continuity_f32<DIM, KK, kPacked<DIM>>
                                                                   : k_continuity_f32<DIM, KK, kSpread>,
                       (L.cap + 127) / 128, 128, L.stream, L.scenes, L.st, L.sc, L.cap, L.bf, L.nl, L.wl);
        return;
    }
    switch (L.mode) {
        case kModeFluidWall: launch_momentum<DIM, KK, kModeFluidWall>(L); break;
        case kModeWallPressure: launch_momentum<DIM, KK, kModeWallPressure>(L); break;
        case kModeBuffers: launch_momentum<DIM, KK, kModeBuffers>(L); break;
        default: launch_momentum<DIM, KK, kModeThermal>(L);
    }
}

template <int DIM>
void dispatch(int stage, const LaunchCtx& L) {
    switch (L.kernel) {
        case SPH_KERNEL_CUBIC_SPLINE: launch_kk<DIM, SPH_KERNEL_CUBIC_SPLINE>(stage, L); break;
        case SPH_KERNEL_GAUSSIAN: launch_kk<DIM, SPH_KERNEL_GAUSSIAN>(stage, L); break;
        case SPH_KERNEL_WENDLAND_C2: launch_kk<DIM, SPH_KERNEL_WENDLAND_C2>(stage, L); break;
        default: launch_kk<DIM, SPH_KERNEL_WENDLAND_C4>(stage, L); break;
    }
}

}  // namespace

}  // namespace sph
