// sph_diag.cu — diagnostics of the per-step cell list: the cell key of every sorted
// particle, and the fluid neighbours each particle's gathers accept.
//
// They expose what the reference's neighbour search produces inside a step
// (CellListMap.update!/neighborlist! + findNeighbours!, FluidWallSolve.jl:21-35,
// Neighbour.jl:88-128) so that it can be compared particle by particle with a CPU
// restatement: the key is the one the step's sort uses, and the neighbours are found by the
// functions with which the gathers of the handle's form find them (FP64: coop_select and
// inside_cut, as k_momentum_fp64; FP32-compensated: row_runs and run_walk, as
// k_continuity_f32 records its list).
#include "sph_fp32.cuh"

namespace sph {

namespace {

template <int DIM>
__global__ void k_cell_keys(const SceneDev* __restrict__ scenes, SortedState st, int32_t b, int32_t e,
                            int32_t* __restrict__ keys) {
    using V = typename VecT<DIM>::T;
    const int i = b + (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= e) return;
    const SceneDev& S = scenes[st.scene[i]];
    keys[i - b] = cell_key<DIM>(((const V*)st.x)[i], S) - S.cell_off;
}

// counts != null: the number of accepted neighbours of sorted particle i; ids != null:
// their ids (upload indices) from ids[rows[i - b]] on, in walk order.
template <int DIM>
__global__ void __launch_bounds__(kCoopThreads)
    k_neighbours_fp64(const SceneDev* __restrict__ scenes, SortedState st, const int32_t* start, int32_t b, int32_t e,
                      int32_t* __restrict__ counts, const int64_t* __restrict__ rows, int32_t* __restrict__ ids) {
    using V = typename VecT<DIM>::T;
    constexpr int kGroups = kCoopThreads / kCoopLanes;
    __shared__ int32_t lists[kGroups * kCoopList<DIM>];
    const int lane = threadIdx.x % kCoopLanes, group = threadIdx.x / kCoopLanes;
    const int place = b + (int)blockIdx.x * kGroups + group;
    const bool on = place < e;
    const int i = min(place, e - 1);
    const SceneDev& S = scenes[st.scene[i]];
    const V* __restrict__ x = (const V*)st.x;
    const V xi = x[i];
    int32_t c[3];
    decode_cell(st.cell[i], S, c);
    int32_t* list = lists + group * kCoopList<DIM>;
    int32_t* out = ids ? ids + rows[i - b] : nullptr;
    int32_t n = 0;
    coop_select<DIM>(
        S, start, st.fa, c, st.fa[i], i, on, list, [&](int j) { return within_cut<DIM>(xi, x[j], S); },
        [&](int, int cnt) {
            const int most = (int)__reduce_max_sync(0xffffffffu, (unsigned)cnt);
            for (int k0 = 0; k0 < most; k0 += kCoopLanes) {
                const int j = k0 + lane < cnt ? list[k0 + lane] : i;
                double rv[DIM];
                make_rvec<DIM>(xi, x[j], S, rv);
                const bool in = k0 + lane < cnt && inside_cut<SPH_KERNEL_CUBIC_SPLINE>(norm_sq<DIM>(rv), S);
                const unsigned hit = (__ballot_sync(0xffffffffu, in) >> ((threadIdx.x & 31) - lane)) & 0xffu;
                if (in && out) out[n + __popc(hit & ((1u << lane) - 1u))] = st.id[j];
                n += __popc(hit);
            }
        });
    if (on && lane == 0 && counts) counts[i - b] = n;
}

template <int DIM>
__global__ void __launch_bounds__(128)
    k_neighbours_f32(const SceneDev* __restrict__ scenes, SortedState st, const int32_t* start, int32_t b, int32_t e,
                     int32_t* __restrict__ counts, const int64_t* __restrict__ rows, int32_t* __restrict__ ids) {
    const int i = b + (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= e) return;
    const SceneDev& S = scenes[st.scene[i]];
    const float4 me = st.fa[i];
    int32_t c[3];
    decode_cell(st.cell[i], S, c);
    const bool prune = S.prune && !select_far(me);
    const int zr = DIM == 3 ? S.reach : 0;
    int32_t* out = ids ? ids + rows[i - b] : nullptr;
    int32_t n = 0;
    for (int dz = -zr; dz <= zr; ++dz)
        for (int dy = -S.reach; dy <= S.reach; ++dy) {
            int first, end, first2, end2;
            row_runs<DIM>(S, start, c, me, prune, dy, dz, first, end, first2, end2);
            auto run = [&](int j, int je) {
                run_walk<DIM>(S, st.fa, i, me, j, je, (float)dy, (float)dz, [](int) { return 0; },
                              [&](int q, const float4&, int, int) {
                                  if (out) out[n] = st.id[q];
                                  ++n;
                              });
            };
            run(first, end);
            run(first2, end2);
        }
    if (counts) counts[i - b] = n;
}

}  // namespace

void launch_cell_keys(const LaunchCtx& L, int32_t b, int32_t e, int32_t* keys) {
    const int n = e - b, block = 128, grid = (n + block - 1) / block;
    if (n <= 0) return;
    if (L.dim == 2) k_cell_keys<2><<<grid, block, 0, L.stream>>>(L.scenes, L.st, b, e, keys);
    else k_cell_keys<3><<<grid, block, 0, L.stream>>>(L.scenes, L.st, b, e, keys);
}

void launch_neighbours(const LaunchCtx& L, int32_t b, int32_t e, int32_t* counts, const int64_t* rows,
                       int32_t* ids) {
    const int n = e - b;
    if (n <= 0) return;
    if (L.precision == SPH_PRECISION_FP32_COMPENSATED) {
        auto kernel = L.dim == 2 ? k_neighbours_f32<2> : k_neighbours_f32<3>;
        kernel<<<(n + 127) / 128, 128, 0, L.stream>>>(L.scenes, L.st, L.sc.start, b, e, counts, rows, ids);
    } else {
        constexpr int kGroups = kCoopThreads / kCoopLanes;
        auto kernel = L.dim == 2 ? k_neighbours_fp64<2> : k_neighbours_fp64<3>;
        kernel<<<(n + kGroups - 1) / kGroups, kCoopThreads, 0, L.stream>>>(L.scenes, L.st, L.sc.start, b, e, counts,
                                                                          rows, ids);
    }
}

}  // namespace sph
