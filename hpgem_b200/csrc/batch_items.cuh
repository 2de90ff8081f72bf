// What the grouped kernels of a batch read per member, and the launch of the classes of
// one-element-per-thread kernels (batch_lane.cu).
#pragma once

#include <cstdint>

#include "handle.cuh"

namespace hgg {

// item whose virtual blocks contain vb: binary search of the items' first blocks,
// which the class table keeps as one compact array after the block total (total[1 + m]
// = item m's block0, ascending, total[1] = 0), so the probes stay in a few cache lines
// instead of touching one item record each
__device__ __forceinline__ int find_item(const int64_t *total, int n, int64_t vb) {
    const int64_t *block0 = total + 1;
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (block0[mid] <= vb) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// The item of the virtual block in shared memory: the stage bodies read its fields
// (pointers, coefficients, sizes) many times, which from shared memory costs what the
// one-problem kernels pay for their parameters, not an L1 load each.  Ends with a
// barrier; the caller's loop begins with one, so the previous block is done with it.
template <typename Item>
__device__ __forceinline__ const Item &item_to_shared(const Item *items, int i, Item &s_item) {
    static_assert(sizeof(Item) % 16 == 0, "items are copied in 16-byte chunks");
    const int4 *src = reinterpret_cast<const int4 *>(items + i);
    int4 *dst = reinterpret_cast<int4 *>(&s_item);
    for (int k = threadIdx.x; k < (int)(sizeof(Item) / 16); k += blockDim.x) dst[k] = src[k];
    __syncthreads();
    return s_item;
}

template <typename KT>
struct alignas(16) TensorLaneItem {
    StageIOT<KT> io[2];
    TensorLaneGeom g;
    int64_t block0;  // first virtual block of kLaneWarps tiles
    int slot;
};
template <typename KT>
struct alignas(16) LaneItem {
    StageIOT<KT> io[2];
    LaneGeom g;
    int64_t block0;  // first virtual block (= chunk)
    int slot;
};

// elements: a warp per tile, kLaneWarps tiles per virtual block (sum-factorised lanes)
constexpr int kLaneWarps = 4;

// One stage of a class of lane kernels.
struct LaneClassStage {
    bool tensor, mixed;
    int dim, order, shape;
    bool wave;
    int nB, stage, nin;
    bool fin;         // the tableau's last stage
    int group_bytes;  // of a group's table
    const void *items;
    const int *n;
    const int64_t *total;
    const int *parity, *remaining;
    unsigned grid;
    cudaStream_t stream;
    int *occupancy;   // set: nothing is launched, the kernel's resident blocks per SM are stored
};
void launch_class_lane(const LaneClassStage &c);

}  // namespace hgg
