// Grouped kernels of the one-element-per-thread classes of a batch: one persistent launch
// per stage of a class, whose blocks walk the members' virtual blocks.
#include "batch_items.cuh"

namespace hgg {

namespace {

// one element per thread, a warp per tile, kLaneWarps tiles per virtual block
template <typename KT, int P, int DIM, int NIN, bool FIN>
__global__ void __launch_bounds__(32 * kLaneWarps)
    grouped_tensor_lane(const TensorLaneItem<KT> *items, const int *n_items, const int64_t *total, const int *parity,
                        const int *remaining) {
    chain_wait();
    const int n = *n_items;
    const int64_t nb = *total;
    for (int64_t vb = blockIdx.x; vb < nb; vb += gridDim.x) {
        const int i = find_item(total, n, vb);
        const int slot = items[i].slot;
        __syncthreads();
        if (remaining[slot] <= 0) continue;
        __shared__ TensorLaneItem<KT> s_it;
        const TensorLaneItem<KT> &it = item_to_shared(items, i, s_it);
        const int64_t tile = (vb - it.block0) * kLaneWarps + (threadIdx.x >> 5);
        if (tile < it.g.n_tiles) tensor_lane_body<KT, P, DIM, NIN, FIN>(it.io[parity[slot]], it.g, tile);
    }
}

// simplices and the wave, one element per thread: a chunk of a member per virtual block
template <typename KT, typename CT, typename ST, int DIM, int NFL, int NB>
__global__ void __launch_bounds__(LaneShape<KT, CT, DIM, NFL, NB, true>::THREADS)
    grouped_wave_lane(const LaneItem<KT> *items, const int *n_items, const int64_t *total, const int *parity,
                      const int *remaining) {
    chain_wait();
    const int n = *n_items;
    const int64_t nb = *total;
    for (int64_t vb = blockIdx.x; vb < nb; vb += gridDim.x) {
        const int i = find_item(total, n, vb);
        const int slot = items[i].slot;
        __syncthreads();
        if (remaining[slot] <= 0) continue;
        __shared__ LaneItem<KT> s_it;
        const LaneItem<KT> &it = item_to_shared(items, i, s_it);
        wave_lane_body<KT, CT, ST, DIM, NFL, NB>(it.io[parity[slot]], it.g, vb - it.block0);
    }
}

template <typename KT, typename CT, int DIM, int NFL, int NB, int NIN>
__global__ void __launch_bounds__(LaneShape<KT, CT, DIM, NFL, NB, false>::THREADS)
    grouped_advection_lane(const LaneItem<KT> *items, const int *n_items, const int64_t *total, const int *parity,
                           const int *remaining) {
    chain_wait();
    const int n = *n_items;
    const int64_t nb = *total;
    for (int64_t vb = blockIdx.x; vb < nb; vb += gridDim.x) {
        const int i = find_item(total, n, vb);
        const int slot = items[i].slot;
        __syncthreads();
        if (remaining[slot] <= 0) continue;
        __shared__ LaneItem<KT> s_it;
        const LaneItem<KT> &it = item_to_shared(items, i, s_it);
        advection_lane_body<KT, CT, DIM, NFL, NB, NIN>(it.io[parity[slot]], it.g, vb - it.block0);
    }
}

template <typename Kern, typename Item>
void launch(const LaneClassStage &c, Kern kern, const Item *items, int threads, int smem) {
    if (smem > 48 * 1024 - (int)sizeof(Item))
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (c.occupancy) {
        int n = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, smem) == cudaSuccess) *c.occupancy = n;
        return;
    }
    launch_chained(true, kern, c.grid, threads, smem, c.stream, items, c.n, c.total, c.parity, c.remaining);
}

template <typename KT>
void launch_tensor(const LaneClassStage &c) {
    tensor_lane_dispatch(c.dim, c.order, [&](auto p, auto d) {
        lane_stage_shape(c.nin, c.fin, [&](auto nin, auto fin) {
            launch(c,
                   grouped_tensor_lane<KT, decltype(p)::value, decltype(d)::value, decltype(nin)::value,
                                       decltype(fin)::value>,
                   static_cast<const TensorLaneItem<KT> *>(c.items), 32 * kLaneWarps, 0);
        });
    });
}

template <typename KT, int DIM, int NFL, int WAVE>
void launch_lane(const LaneClassStage &c) {
    const auto *items = static_cast<const LaneItem<KT> *>(c.items);
    dense_dispatch<DIM, NFL, WAVE>(c.nB, [&](auto nbc) {
        constexpr int NB = decltype(nbc)::value;
        using CT = DenseCT<KT, NB>;
        if constexpr (lane_size(DIM, NFL, WAVE, NB)) {
            using SH = LaneShape<KT, CT, DIM, NFL, NB, WAVE>;
            if constexpr (WAVE) {
                if (c.stage > 0)
                    launch(c, grouped_wave_lane<KT, CT, CT, DIM, NFL, NB>, items, SH::THREADS,
                           wave_lane_smem<KT, CT, CT, DIM, NFL, NB>(c.group_bytes, SH::TILES));
                else
                    launch(c, grouped_wave_lane<KT, CT, double, DIM, NFL, NB>, items, SH::THREADS,
                           wave_lane_smem<KT, CT, double, DIM, NFL, NB>(c.group_bytes, SH::TILES));
            } else {
                if (c.nin == 0) launch(c, grouped_advection_lane<KT, CT, DIM, NFL, NB, 0>, items, SH::THREADS, c.group_bytes);
                else if (c.nin == 1)
                    launch(c, grouped_advection_lane<KT, CT, DIM, NFL, NB, 1>, items, SH::THREADS, c.group_bytes);
                else launch(c, grouped_advection_lane<KT, CT, DIM, NFL, NB, -1>, items, SH::THREADS, c.group_bytes);
            }
        }
    });
}

template <typename KT>
void launch_any(const LaneClassStage &c) {
    if (c.tensor) return launch_tensor<KT>(c);
    switch (c.shape) {
        case HGG_SHAPE_TRIANGLE: return c.wave ? launch_lane<KT, 2, 3, 1>(c) : launch_lane<KT, 2, 3, 0>(c);
        case HGG_SHAPE_TETRAHEDRON: return c.wave ? launch_lane<KT, 3, 4, 1>(c) : launch_lane<KT, 3, 4, 0>(c);
        case HGG_SHAPE_SQUARE: return launch_lane<KT, 2, 4, 1>(c);
        case HGG_SHAPE_CUBE: return launch_lane<KT, 3, 6, 1>(c);
    }
}

}  // namespace

void launch_class_lane(const LaneClassStage &c) {
    if (c.mixed) launch_any<float>(c);
    else launch_any<double>(c);
}

}  // namespace hgg
