// Stage launches of the one-element-per-thread kernels of simplices and the wave.
#include <type_traits>

#include "handle.cuh"

namespace hgg {

namespace {

// most: of a block of the kernel on any mesh.  The limit is the process's, so it is set to
// that: a smaller mesh's launch on another thread does not lower it.
template <typename Kern, typename KT>
void launch(hgg_handle *h, Kern kern, const StageIOT<KT> &io, int threads, int smem, int most) {
    if (most > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    launch_chained(h->overlap, kern, (unsigned)h->lgeo.n_chunks, threads, smem, h->stream, io, h->lgeo);
}

template <typename KT, int DIM, int NFL, int WAVE>
int launch_lane(hgg_handle *h, const StageIOT<KT> &io) {
    bool done = false;
    dense_dispatch<DIM, NFL, WAVE>(h->op.nB, [&](auto nbc) {
        constexpr int NB = decltype(nbc)::value;
        using CT = DenseCT<KT, NB>;
        if constexpr (lane_size(DIM, NFL, WAVE, NB)) {
            if constexpr (WAVE) {
                using SH = LaneShape<KT, CT, DIM, NFL, NB, true>;
                const int threads = 32 * SH::RW * h->lane_tiles, bytes = h->lgeo.group_bytes;
                if (io.win)
                    launch(h, wave_lane<KT, CT, CT, DIM, NFL, NB>, io, threads,
                           wave_lane_smem<KT, CT, CT, DIM, NFL, NB>(bytes, h->lane_tiles),
                           wave_lane_smem<KT, CT, CT, DIM, NFL, NB>(bytes, SH::TILES));
                else
                    launch(h, wave_lane<KT, CT, double, DIM, NFL, NB>, io, threads,
                           wave_lane_smem<KT, CT, double, DIM, NFL, NB>(bytes, h->lane_tiles),
                           wave_lane_smem<KT, CT, double, DIM, NFL, NB>(bytes, SH::TILES));
            } else {
                const int threads = 32 * LaneShape<KT, CT, DIM, NFL, NB, false>::RW * h->lane_tiles;
                const int bytes = h->lgeo.group_bytes;  // the same on every mesh
                if (io.nin == 0) launch(h, advection_lane<KT, CT, DIM, NFL, NB, 0>, io, threads, bytes, bytes);
                else if (io.nin == 1) launch(h, advection_lane<KT, CT, DIM, NFL, NB, 1>, io, threads, bytes, bytes);
                else launch(h, advection_lane<KT, CT, DIM, NFL, NB, -1>, io, threads, bytes, bytes);
            }
            done = true;
        }
    });
    return done ? 0 : fail(h, HGG_ERR_UNSUPPORTED, "lane kernel: no kernel for this basis size");
}

template <typename KT>
int launch_lane_any(hgg_handle *h, const StageIOT<KT> &io) {
    const bool wave = h->op.physics != HGG_PHYSICS_ADVECTION;
    switch (h->op.shape) {
        case HGG_SHAPE_TRIANGLE: return wave ? launch_lane<KT, 2, 3, 1>(h, io) : launch_lane<KT, 2, 3, 0>(h, io);
        case HGG_SHAPE_TETRAHEDRON: return wave ? launch_lane<KT, 3, 4, 1>(h, io) : launch_lane<KT, 3, 4, 0>(h, io);
        case HGG_SHAPE_SQUARE:
            if (wave) return launch_lane<KT, 2, 4, 1>(h, io);
            break;
        case HGG_SHAPE_CUBE:
            if (wave) return launch_lane<KT, 3, 6, 1>(h, io);
            break;
    }
    return fail(h, HGG_ERR_UNSUPPORTED, "lane kernel: shape");
}

}  // namespace

int launch_stage_lane(hgg_handle *h, const StageIOT<double> &io) { return launch_lane_any<double>(h, io); }
int launch_stage_lane(hgg_handle *h, const StageIOT<float> &io) { return launch_lane_any<float>(h, io); }

}  // namespace hgg
