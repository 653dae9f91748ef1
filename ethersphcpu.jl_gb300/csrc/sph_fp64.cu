// sph_fp64.cu — plain FP64 gather kernels of the WCSPH step (compiled -fmad=false: the
// per-particle updates keep the reference's unfused operations; the pair terms write their
// fused multiply-adds out).
//
// K4 continuity + updateDensity! + updatePressure!   (Continuity.jl:8-17,
//    UpdateDensity.jl:8-12, UpdatePressure.jl:8-16)
// K5 momentum (pressure, viscosity, compulsive wall, heat) + updateTemperature! +
//    updateVelocity! + updatePosition!, fused with the out-of-domain check and the
//    cell hash of the next step's sort   (PressureForce.jl, ViscosityForce.jl,
//    WallForce.jl, ThermalConduction.jl, SelfAction/*.jl, FluidWallSolve.jl:37-81)
// On a re-initialisation step K5 also forms the Shepard sums of reconstructScalar!
//    (ReconstructValue.jl:22-57) over the same fluid neighbours at the same start-of-step
//    positions, and writes the re-initialised density: the update and the
//    re-initialisation are one kernel (FluidWallSolve.jl:64-72).
//
// Eight lanes share one fluid particle (sph_coop.cuh): FP32 selection of its neighbours
// into shared memory, FP64 pair terms over that list, and one lane that updates the
// particle.  No atomics on the physics, a fixed order of every sum: results are
// deterministic and do not depend on the batch.
//
// What bounds them: FP64 instructions (2 lanes a SM and cycle).
//   * K4 and the viscosity and heat terms of K5 are factored so that a pair divides once or
//     not at all: r by one Householder step on rsqrt, dW/r as the kernel's own polynomial
//     (no normalisation of r_vec), constants outside the sums, m/rho formed once a particle,
//     one reciprocal for the quotients of viscosity and heat.
//   * pressure and wall forces cancel to a 1e-9 th of themselves in a fluid at rest, so their
//     terms keep the reference's operations, rounding and order of addition; what changes
//     is their cost: root and reciprocal share one iteration, division by h and W(gap) is a
//     multiplication with a residual step, and rejected candidates cost no FP64 at all.
// Measured (us, K4 / K5; before: a thread a particle walking the cells, every candidate's
// distance in FP64): dam breaks of 800 and 5,000 particles 117 / 253 -> 11 / 34 and 125 / 254 ->
// 17 / 49, cavities of 10,201 and 65,536 particles 133 / 311 -> 27 / 86 and 340 / 1023 -> 97 /
// 394, a 3D dam break of 52,000 particles 1636 / 3403 -> 306 / 1300.
#include "sph_coop.cuh"

namespace sph {

// Solve variants: which wall terms and which body force.
enum { kModeFluidWall = 0, kModeWallPressure = 1, kModeThermal = 2, kModeBuffers = 3 };

// Geometry of the pair (i, j): r_vec and q^2 = |r_vec|^2 / h^2.
template <int DIM, typename V>
__device__ __forceinline__ double pair_q2(const V& xi, const V& xj, const SceneDev& S, double rv[DIM]) {
    make_rvec<DIM>(xi, xj, S, rv);
    double d2 = fma(rv[0], rv[0], rv[1] * rv[1]);
    if (DIM == 3) d2 = fma(rv[DIM - 1], rv[DIM - 1], d2);
    return d2 * S.inv_hh;
}

template <int DIM, typename V>
__device__ __forceinline__ void vec_diff(const V& a, const V& b, double d[DIM]) {
    d[0] = a.x - b.x;
    d[1] = a.y - b.y;
    if (DIM == 3) d[DIM - 1] = comp(a, DIM - 1) - comp(b, DIM - 1);
}

template <int DIM>
__device__ __forceinline__ double dot_fma(const double a[DIM], const double b[DIM]) {
    double s = fma(a[0], b[0], a[1] * b[1]);
    if (DIM == 3) s = fma(a[DIM - 1], b[DIM - 1], s);
    return s;
}

template <int DIM, int KK>
__global__ void __launch_bounds__(kCoopThreads, kCoopBlocks)
    k_continuity_fp64(const SceneDev* __restrict__ scenes, SortedState st, SortScratch sc, int32_t cap, BufferState bf) {
    pdl_wait();
    pdl_trigger();
    using V = typename VecT<DIM>::T;
    constexpr int kWarps = kCoopThreads / 32;
    __shared__ int32_t lists[kWarps * kCoopGroups * kCoopList<DIM>];
    __shared__ double drho_all[kCoopThreads];
    const int lane = threadIdx.x % kCoopLanes;
    const V* __restrict__ x = (const V*)st.x;
    const V* __restrict__ v = (const V*)st.v;
    const double* __restrict__ m = st.m;
    int32_t* list = lists + threadIdx.x / kCoopLanes * kCoopList<DIM>;
    double* drhos = drho_all + (threadIdx.x & ~31);
    auto gather = [&](int i, int place, bool valid) {
        const SceneDev& S = scenes[st.scene[i]];
        const bool on = valid && scene_runs(S, sc.scene_step[st.scene[i]]);
        const V xi = x[i];
        const V vi = v[i];
        int32_t c[3];
        decode_cell(st.cell[i], S, c);
        double drho = 0.0;
        coop_select<DIM>(
            S, sc.start, st.fa, c, st.fa[i], i, on, list, [&](int j) { return within_cut<DIM>(xi, x[j], S); },
            [&](int first, int cnt) {
                int k = (lane - first) & (kCoopLanes - 1);
                if (k >= cnt) return;
                V xn = x[list[k]], vn = v[list[k]];
                double mn = m[list[k]];
                for (; k < cnt; k += kCoopLanes) {
                    const V xj = xn;
                    const V vj = vn;
                    const double m_j = mn;
                    if (k + kCoopLanes < cnt) {  // the next pair's data
                        const int j = list[k + kCoopLanes];
                        xn = x[j];
                        vn = v[j];
                        mn = m[j];
                    }
                    double rv[DIM], vv[DIM];
                    const double q2 = pair_q2<DIM>(xi, xj, S, rv);
                    if (!inside_cut<DIM, KK>(rv, q2, S)) continue;
                    vec_diff<DIM>(vi, vj, vv);
                    drho = fma(m_j * kernel_f<KK>(q2), dot_fma<DIM>(rv, vv), drho);
                }
            });
        drho *= S.kg_h;
        if (on && bf.n) {  // inlet/outlet buffer neighbours (FluidInletOutletWallSolve.jl:59-72)
            const V* __restrict__ bx = (const V*)bf.x;
            const V* __restrict__ bv = (const V*)bf.v;
            walk_cells<DIM>(S, bf.start, c, [&](int jb, int je) {
                for (int b = jb + lane; b < je; b += kCoopLanes) {
                    double rv[DIM], vv[DIM];
                    const double q2 = pair_q2<DIM>(xi, bx[b], S, rv);
                    if (!(q2 <= S.q2_max) || !inside_cut<DIM, KK>(rv, q2, S)) continue;
                    vec_diff<DIM>(vi, bv[b], vv);
                    drho = fma(bf.m[b] * kernel_f<KK>(q2) * S.kg_h, dot_fma<DIM>(rv, vv), drho);
                }
            });
        }
        drho = coop_sum(drho);
        if (lane == 0) drhos[place] = drho;
    };
    auto update = [&](int i) {
        const SceneDev& S = scenes[st.scene[i]];
        if (!scene_runs(S, sc.scene_step[st.scene[i]])) return;
        const double drho = drhos[threadIdx.x & 31];
        const double m_i = m[i];
        double rho = st.rho[i];
        rho += drho * S.dt;  // written to rhoc, so the kernel can be re-run on the same input
        // updatePressure! (UpdatePressure.jl:8-16), every operation rounded as written there
        const bool ordinary = rcp_rn_range(rho) && rho > 0.0;
        const double rr = ordinary ? div_rn(rho, S.rho0, S.inv_rho0) : rho / S.rho0;
        double pw, cw;  // rr^gamma, rr^(gamma - 1)
        if (S.gamma == 7 && ordinary) {
            pw = powi_fixed<7>(rr);
            cw = powi_fixed<6>(rr);
        } else {
            pw = jl_powi(rr, S.gamma);
            cw = jl_powi(rr, S.gamma - 1);
        }
        double inv;
        const double p = S.b * (pw - 1.0) + S.p0;
        st.rhoc[i] = rho;
        st.p[i] = p;
        st.c[i] = S.c0 * (sqrt_rn_range(cw) ? sqrt_rn(cw, inv) : sqrt(cw));
        if (ordinary) {
            const double r2 = rho * rho;
            st.P[i] = div_rn(p, r2, rcp_rn(r2));
            st.vol[i] = div_rn(m_i, rho, rcp_rn(rho));
        } else {
            st.P[i] = p / (rho * rho);
            st.vol[i] = m_i / rho;
        }
    };
    coop_turns(min(cap, *sc.n_live), sc.queue + kQueueContinuity, gather, update);
}

// SHEP: the momentum gather of density re-initialisation steps, for the particles of the
// scenes whose step re-initialises (every running scene when `sel` is set).  Without SHEP,
// `sel` set leaves those particles to the SHEP launch of the same step (a batch whose
// scenes re-initialise at different steps runs both).  Continuity starts this kernel early: the
// selection of a warp's first particles needs positions only, so it runs where continuity
// leaves room and the wait comes after it (a step of an 800-particle dam break 51.9 -> 49.5
// us, of 5,000 particles 70.8 -> 66.2, of a 10,201-particle cavity 120.6 -> 117.8).
template <int DIM, int KK, int MODE, bool SHEP>
__global__ void __launch_bounds__(kCoopThreads, kCoopBlocks)
    k_momentum_fp64(const SceneDev* __restrict__ scenes, SortedState st, NextState nx, WallState wl, SortScratch sc,
                    int32_t cap, BufferState bf, BufferScratch bs, BufferRules br, int sel) {
    using V = typename VecT<DIM>::T;
    constexpr bool HEAT = MODE == kModeThermal;
    constexpr int kSums = (HEAT ? 2 : 0) + (SHEP ? 2 : 0);  // sums taken by lane
    constexpr int kWarps = kCoopThreads / 32;
    __shared__ int32_t lists[kWarps * kCoopGroups * kCoopList<DIM>];
    __shared__ double terms_all[kWarps * 3 * DIM * kTermStride];
    __shared__ double vecs_all[kWarps * DIM * 32], sums_all[kWarps * (kSums ? kSums : 1) * 32];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % kCoopLanes;
    double* terms = terms_all + warp * 3 * DIM * kTermStride;
    double* vecs = vecs_all + warp * DIM * 32;
    double* sums = sums_all + warp * (kSums ? kSums : 1) * 32;
    const V* __restrict__ x = (const V*)st.x;
    const V* __restrict__ v = (const V*)st.v;
    auto takes = [&](const SceneDev& S, int64_t step) {  // the particle's sums are formed by this launch
        const bool runs = scene_runs(S, step);
        if (SHEP) return runs && (sel || is_step(step, S.reinit_interval));
        return runs && !(sel && is_step(step, S.reinit_interval));
    };
    const int shift = (threadIdx.x & 31) - lane;
    double* mine = terms + (threadIdx.x & 31);  // this lane's place in a row of terms
    int32_t* list = lists + threadIdx.x / kCoopLanes * kCoopList<DIM>;
    bool ready = false;  // continuity's results are visible
    auto gather = [&](int i, int place, bool valid) {
        const SceneDev& S = scenes[st.scene[i]];
        const bool on = valid && takes(S, sc.scene_step[st.scene[i]]);
        const V xi = x[i];
        const V vi = v[i];
        double rho_i = 0.0, P_i = 0.0;
        if (ready) {
            rho_i = st.rhoc[i];
            P_i = st.P[i];
        }
        const double gap_i = st.gap[i];
        // W((gap_i + gap_j)/2) of the tensile term: with uniform gaps a constant of the scene
        const bool uniform = S.uniform_gap != 0;
        double T_i = 0.0, kap_i = 0.0;
        if (HEAT) {
            T_i = st.T[i];
            kap_i = st.kappa[i];
        }
        int32_t c[3];
        decode_cell(st.cell[i], S, c);
        const float4 me = st.fa[i];
        double dv = 0.0;  // lane d < DIM: component d of the acceleration
        double aT = 0.0, wT = 0.0, sw = 0.0, sws = 0.0;

        // rounds of a list pass: the entries' places are those of the whole list (first + k),
        // so a lane's entries do not depend on where the passes are cut
        auto rounds = [&](int first, int cnt, auto&& body) {
            const int r0 = first / kCoopLanes, r1 = (first + cnt + kCoopLanes - 1) / kCoopLanes;
            const int most = (int)__reduce_max_sync(0xffffffffu, (unsigned)(r1 - r0));
            for (int r = 0; r < most; ++r) {
                const int at = (r0 + r) * kCoopLanes - first;  // entry of lane 0
                body(at + lane, max(0, -at), min(kCoopLanes, cnt - at));
            }
        };

        // ---- fluid neighbours: pressureForce! + viscosityForce! (+ thermalConduction!),
        // PressureForce.jl:14-19, ViscosityForce.jl:15-23, ThermalConduction.jl:15-21.  With
        // mu = nu0 rho the viscosity factor is 4 nu0 m_j r dW / ((rho_i + rho_j) (r^2 + 0.01 h^2));
        // heat is taken as aT = sum m_j/rho_j kappa_j r dW / ((kappa_i + kappa_j) (r^2 + 0.01 h^2)) T_ij
        coop_select<DIM>(
            S, sc.start, st.fa, c, me, i, on, list, [&](int j) { return within_cut<DIM>(xi, x[j], S); },
            [&](int first, int cnt) {
                if (!ready) {
                    pdl_wait();
                    ready = true;
                    rho_i = st.rhoc[i];
                    P_i = st.P[i];
                }
                rounds(first, cnt, [&](int k, int e0, int e1) {
                    double tp[DIM], tv[DIM];
#pragma unroll
                    for (int d = 0; d < DIM; ++d) tp[d] = tv[d] = 0.0;
                    if (k >= 0 && k < cnt) {
                        const int j = list[k];
                        const V xj = x[j];
                        const V vj = v[j];
                        const double m_j = st.m[j], rho_j = st.rhoc[j], P_j = st.P[j];
                        double vol_j = 0.0, kap_j = 0.0, T_j = 0.0;
                        if (HEAT || SHEP) vol_j = st.vol[j];
                        if (HEAT) {
                            kap_j = st.kappa[j];
                            T_j = st.T[j];
                        }
                        double rv[DIM];
                        make_rvec<DIM>(xi, xj, S, rv);
                        const double d2 = norm_sq<DIM>(rv);
                        if (inside_cut<KK>(d2, S)) {
                            double r, W, dW, grad[DIM], vv[DIM];
                            pair_kernel<DIM, KK>(rv, d2, S, r, W, dW, grad);
                            if (SHEP) {
                                sw = fma(W, vol_j, sw);
                                sws = fma(W, m_j, sws);
                            }
                            double prho2 = P_i + P_j;
                            const double tens = fabs(prho2) * 0.01 * W;
                            prho2 += uniform ? div_rn(tens, S.wg, S.inv_wg)
                                             : tens / kernel_w<KK>((gap_i + st.gap[j]) / 2.0, S);
                            const double fp = -m_j * prho2;
                            vec_diff<DIM>(vi, vj, vv);
                            const double sum_rho = rho_i + rho_j;
                            const double rdW = r * dW;
                            const double den = sum_rho * (d2 + S.hh001);
                            double fv;
                            if (HEAT) {
                                const double sum_kap = kap_i + kap_j;
                                const double R = rcp3(den * sum_kap);
                                fv = m_j * (S.nu4 * rdW) * (R * sum_kap);
                                aT = fma(rdW * vol_j * (R * sum_rho * kap_j), T_i - T_j, aT);
                            } else {
                                fv = m_j * (S.nu4 * rdW) * rcp3(den);
                            }
#pragma unroll
                            for (int d = 0; d < DIM; ++d) {
                                tp[d] = fp * grad[d];
                                tv[d] = fv * vv[d];
                            }
                        }
                    }
#pragma unroll
                    for (int d = 0; d < DIM; ++d) {
                        mine[d * kTermStride] = tp[d];
                        mine[(DIM + d) * kTermStride] = tv[d];
                    }
                    __syncwarp();
                    add_terms<DIM, 2>(terms, lane, shift, e0, e1, dv);
                    __syncwarp();
                });
            });

        // ---- inlet/outlet buffer neighbours: pressureForce! + viscosityForce! with the
        // buffer particle's frozen density and pressure (FluidInletOutletWallSolve.jl:125-158)
        if (MODE == kModeBuffers) {
            const V* __restrict__ bx = (const V*)bf.x;
            const V* __restrict__ bv = (const V*)bf.v;
            double db[DIM];  // every lane of the particle continues the whole sum (few particles do)
#pragma unroll
            for (int d = 0; d < DIM; ++d) db[d] = __shfl_sync(0xffffffffu, dv, d, kCoopLanes);
            if (on && bf.n) {
                walk_cells<DIM>(S, bf.start, c, [&](int jb, int je) {
                    for (int b = jb; b < je; ++b) {
                        double rv[DIM], vv[DIM];
                        make_rvec<DIM>(xi, bx[b], S, rv);
                        const double d2 = norm_sq<DIM>(rv);
                        if (!(d2 <= S.rc2)) continue;
                        double r, W, dW, grad[DIM];
                        pair_kernel<DIM, KK>(rv, d2, S, r, W, dW, grad);
                        vec_diff<DIM>(vi, bv[b], vv);
                        const double rho_b = bf.rho[b], m_b = bf.m[b], gap_b = bf.gap[b];
                        double prho2 = P_i + bf.p[b] / (rho_b * rho_b);
                        prho2 += fabs(prho2) * 0.01 * W / kernel_w<KK>(gap_b == gap_i ? gap_i : (gap_i + gap_b) / 2.0, S);
                        const double fv = S.nu4 * (r * dW) / ((rho_i + rho_b) * (d2 + S.hh001));
#pragma unroll
                        for (int k = 0; k < DIM; ++k) db[k] += -m_b * prho2 * grad[k];
#pragma unroll
                        for (int k = 0; k < DIM; ++k) db[k] += m_b * fv * vv[k];
                    }
                });
            }
#pragma unroll
            for (int d = 0; d < DIM; ++d)
                if (lane == d) dv = db[d];
        }

        // ---- walls: wallForce! (+ background pressureForce!) + viscosityForce! (+ heat),
        // only where a wall cell is within reach of the particle's cell
        const bool walls = on && wl.n > 0 && wl.near[st.cell[i]];
        const bool near = __any_sync(0xffffffffu, walls);
        if (near) {
            const V* __restrict__ wx = (const V*)wl.x;
            const V* __restrict__ wn = (const V*)wl.nrm;
            const V* __restrict__ wv = (const V*)wl.v;
            const double c_i = st.c[i];
            const double m_i = st.m[i];
            const double Pw = P_i + S.P_bg;
            const double Wg_i = uniform ? S.wg : kernel_w<KK>(gap_i, S);
            const double nu_rho = 2.0 * S.nu0 / rho_i;  // 8 mu_i / (2 rho_i)^2
            coop_select<DIM>(
                S, wl.start, wl.fa, c, me, -1, walls, list, [&](int j) { return within_cut<DIM>(xi, wx[j], S); },
                [&](int first, int cnt) {
                    rounds(first, cnt, [&](int k, int e0, int e1) {
                        double tw[DIM], tp[DIM], tv[DIM];
#pragma unroll
                        for (int d = 0; d < DIM; ++d) tw[d] = tp[d] = tv[d] = 0.0;
                        if (k >= 0 && k < cnt) {
                            const int j = list[k];
                            const V nw = wn[j];
                            double rv[DIM];
                            make_rvec<DIM>(xi, wx[j], S, rv);
                            const double d2 = norm_sq<DIM>(rv);
                            if (inside_cut<KK>(d2, S)) {
                                double r, W, dW, grad[DIM], vv[DIM], nn[DIM];
                                pair_kernel<DIM, KK>(rv, d2, S, r, W, dW, grad);
                                vec_diff<DIM>(vi, wv[j], vv);
                                nn[0] = nw.x;
                                nn[1] = nw.y;
                                if (DIM == 3) nn[DIM - 1] = comp(nw, DIM - 1);
                                const double vert = dotd<DIM>(vv, nn);
                                {  // WallForce.jl:15-28 (Rogers & Dalrymple 2008)
                                    const double gw = wl.gap[j];
                                    const double psi = fabs(dotd<DIM>(rv, nn));
                                    double t = r * r - psi * psi;
                                    t = t < 0.0 ? 0.0 : t;  // NaN stays
                                    const double far = gw * (1.0 + 1e-9);
                                    if (!(psi > far || t > far * far)) {
                                        const double xi_ = sqrt(t);
                                        const double q = psi / gw;
                                        if (!(q > 1.0 || xi_ > gw)) {
                                            const double pxi = fabs((1.0 + cos(CUDART_PI * xi_ / gw)) / 2.0);
                                            const double beta = vert > 0.0 ? 0.0 : 1.0;
                                            const double rpsi = (0.01 * (c_i * c_i) + beta * c_i * fabs(vert)) / S.h *
                                                                fabs(1.0 - q) / sqrt(q);
                                            const double wf = rpsi * pxi;
#pragma unroll
                                            for (int d = 0; d < DIM; ++d) tw[d] = wf * nn[d];
                                        }
                                    }
                                }
                                if (MODE == kModeWallPressure || HEAT) {  // PressureForce.jl:29-33
                                    const double tens = fabs(Pw) * 0.01 * W;
                                    const double prho2 = Pw + (uniform ? div_rn(tens, S.wg, S.inv_wg) : tens / Wg_i);
#pragma unroll
                                    for (int d = 0; d < DIM; ++d) tp[d] = -m_i * prho2 * grad[d];
                                }
                                // ViscosityForce.jl:34-44
                                const double rdW = r * dW * rcp3(d2 + S.hh001);
                                const double fv = m_i * (nu_rho * rdW);
#pragma unroll
                                for (int d = 0; d < DIM; ++d) tv[d] = fv * fma(-vert, nn[d], vv[d]);
                                if (HEAT && wl.kind[j] == SPH_WALL_THERMOSTATIC)  // ThermalConduction.jl:31-35
                                    wT = fma((kap_i + wl.kappa[j]) * rdW, T_i - wl.T[j], wT);
                            }
                        }
#pragma unroll
                        for (int d = 0; d < DIM; ++d) {
                            mine[d * kTermStride] = tw[d];
                            mine[(DIM + d) * kTermStride] = tp[d];
                            mine[(2 * DIM + d) * kTermStride] = tv[d];
                        }
                        __syncwarp();
                        add_terms<DIM, 3>(terms, lane, shift, e0, e1, dv);
                        __syncwarp();
                    });
                });
        }
        if (lane < DIM) vecs[lane * 32 + place] = dv;
        if (HEAT) {
            aT = coop_sum(aT);
            if (near) wT = coop_sum(wT);
        }
        if (SHEP) {
            sw = coop_sum(sw);
            sws = coop_sum(sws);
        }
        if (lane == 0) {
            if (HEAT) {
                sums[place] = aT;
                sums[32 + place] = wT;
            }
            if constexpr (SHEP) {
                sums[(kSums - 2) * 32 + place] = sw;
                sums[(kSums - 1) * 32 + place] = sws;
            }
        }
    };

    // ---- the update, one lane a particle
    auto update = [&](int i) {
        const SceneDev& S = scenes[st.scene[i]];
        const int64_t step = sc.scene_step[st.scene[i]];
        if (!takes(S, step)) {
            if (!SHEP && !scene_runs(S, step)) carry_frozen<DIM>(i, S, st, nx, sc);
            return;
        }
        const V xi = x[i];
        const V vi = v[i];
        const double rho_i = st.rhoc[i];
        const double m_i = st.m[i];
        double dv[DIM];
#pragma unroll
        for (int k = 0; k < DIM; ++k) dv[k] = vecs[k * 32 + (threadIdx.x & 31)];
        double T_i = 0.0, dT = 0.0;
        if (HEAT) {
            T_i = st.T[i];
            const double fluid = sums[threadIdx.x & 31], wall = sums[32 + (threadIdx.x & 31)];
            const double cp_i = st.cp[i];
            dT = (4.0 * st.kappa[i] * fluid + S.inv_cp_d * S.inv_rho0 * m_i * cp_i * wall) / (cp_i * rho_i);
        }

        // ---- updateTemperature!, updateVelocity!, updatePosition!
        const double dt = S.dt;
        double body[DIM];
        if (MODE == kModeThermal) {
            T_i += dt * dT;
#pragma unroll
            for (int k = 0; k < DIM; ++k) body[k] = S.bous[k] * (T_i - S.t0);
            nx.T[i] = T_i;
        } else {
            if (nx.T) nx.T[i] = st.T[i];  // thermal particles in a solve without heat terms
#pragma unroll
            for (int k = 0; k < DIM; ++k) body[k] = S.g[k];
        }
        double vn[DIM], xn[DIM];
        vn[0] = vi.x;
        vn[1] = vi.y;
        xn[0] = xi.x;
        xn[1] = xi.y;
        if (DIM == 3) {
            vn[DIM - 1] = comp(vi, DIM - 1);
            xn[DIM - 1] = comp(xi, DIM - 1);
        }
#pragma unroll
        for (int k = 0; k < DIM; ++k) vn[k] += body[k] * dt;
#pragma unroll
        for (int k = 0; k < DIM; ++k) vn[k] += dv[k] * dt;
#pragma unroll
        for (int k = 0; k < DIM; ++k) xn[k] += vn[k] * dt - dv[k] * S.dtdt / 2.0;
        if (S.periodic_x) {
            if (xn[0] >= S.wrap_hi) xn[0] -= S.period;
            else if (xn[0] < S.lo[0]) xn[0] += S.period;
        }
        V xo, vo;
        xo.x = xn[0];
        xo.y = xn[1];
        vo.x = vn[0];
        vo.y = vn[1];
        if constexpr (DIM == 3) {
            xo.z = xn[2];
            xo.w = 0.0;
            vo.z = vn[2];
            vo.w = 0.0;
        }
        ((V*)nx.x)[i] = xo;
        ((V*)nx.v)[i] = vo;
        if constexpr (SHEP) {  // the particle's own W(0) term, then the Shepard quotient
            const double sw = sums[(kSums - 2) * 32 + (threadIdx.x & 31)] + S.k0 * m_i / rho_i;
            const double sws = sums[(kSums - 1) * 32 + (threadIdx.x & 31)] + S.k0 * m_i;
            nx.rho[i] = sws / sw;
        } else {
            nx.rho[i] = rho_i;
        }

        // ---- non-finite state, out-of-domain check, next step's cell hash
        bool finite = bits_finite(rho_i);
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
            cell_arrival(sc, i, moved_key<DIM>(st.cell[i], st.fa[i], xi, xo, S));
        }
    };
    coop_turns(min(cap, *sc.n_live), sc.queue + (SHEP ? kQueueShepard : kQueueMomentum), gather, update);
    pdl_wait();
}

// ---------------------------------------------------------------- launchers
namespace {
template <int DIM, int KK>
void launch_k4(const LaunchCtx& L) {
    const CoopShape shape = coop_shape(L.cap);
    launch_dep(k_continuity_fp64<DIM, KK>, shape.grid, shape.threads, L.stream, L.scenes, L.st, L.sc, L.cap, L.bf);
}
template <int DIM, int KK, int MODE>
void launch_k5(const LaunchCtx& L) {
    const CoopShape shape = coop_shape(L.cap);
    if (L.shepard)
        launch_dep(k_momentum_fp64<DIM, KK, MODE, true>, shape.grid, shape.threads, L.stream, L.scenes, L.st, L.nx, L.wl,
                   L.sc, L.cap, L.bf, L.bs, L.br, L.force_reinit);
    else
        launch_dep(k_momentum_fp64<DIM, KK, MODE, false>, shape.grid, shape.threads, L.stream, L.scenes, L.st, L.nx, L.wl,
                   L.sc, L.cap, L.bf, L.bs, L.br, L.skip_reinit);
}

template <int DIM>
void dispatch_kk(int kk, int stage, int mode, const LaunchCtx& L) {
#define SPH_KK_CASE(KKV)                                                        \
    case KKV:                                                                   \
        if (stage == 0) launch_k4<DIM, KKV>(L);                                 \
        else if (mode == kModeFluidWall) launch_k5<DIM, KKV, kModeFluidWall>(L); \
        else if (mode == kModeWallPressure) launch_k5<DIM, KKV, kModeWallPressure>(L); \
        else if (mode == kModeBuffers) launch_k5<DIM, KKV, kModeBuffers>(L);    \
        else launch_k5<DIM, KKV, kModeThermal>(L);                              \
        break;
    switch (kk) {
        SPH_KK_CASE(SPH_KERNEL_CUBIC_SPLINE)
        SPH_KK_CASE(SPH_KERNEL_GAUSSIAN)
        SPH_KK_CASE(SPH_KERNEL_WENDLAND_C2)
        SPH_KK_CASE(SPH_KERNEL_WENDLAND_C4)
    }
#undef SPH_KK_CASE
}
}  // namespace

void launch_physics_fp64(int stage, const LaunchCtx& L) {
    if (L.dim == 2) dispatch_kk<2>(L.kernel, stage, L.mode, L);
    else dispatch_kk<3>(L.kernel, stage, L.mode, L);
}

}  // namespace sph
