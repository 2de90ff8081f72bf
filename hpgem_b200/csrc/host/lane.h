// Set-up of the one-element-per-thread stage kernels (tensor_lane.cuh): the meshes
// they take and the operators their threads share.
#pragma once

#include <cstddef>
#include <cstdint>
#include <vector>

#include "operators.h"

#ifdef __CUDACC__
#define HGG_HOST_DEVICE __host__ __device__
#else
#define HGG_HOST_DEVICE
#endif

namespace hgg {

// Sum-factorised advection with one geometry for all elements: per axis the folded 1D
// matrix and the inflow face.  Sized for the largest one: two axes at p = 5.
struct TensorLaneGeom {
    double E[72];        // [DIM][NP][NP] volume and outflow of each axis
    double L[12];        // [DIM][NP] -sigma times the inflow side's lift
    // the same unfolded, for the FP32 form, which keeps the general kernel's order of operations
    float D1[36];        // [NP][NP]
    float lift[2][6];    // [side][NP]
    float ahat[3];
    float sigma[3][2];   // of each axis and side
    int32_t outflow[3];  // bit `side`: the element's own trace enters that face's flux
    int32_t side[3];     // inflow side of the axis (0: -1, 1: +1), -1: no inflow face
    int32_t n_tiles;
    const int32_t *nbr;  // [n_tiles][DIM][32] the inflow face's neighbour (device)
};

// orders with a kernel: every coefficient of an element fits a thread's registers
inline bool tensor_lane_order(int dim, int p) { return (dim == 2 && p >= 1 && p <= 5) || (dim == 3 && p >= 1 && p <= 2); }

// How much rounding of the vertex coordinates can change an element's geometry.  The cells
// of a structured mesh are equal up to that, and only up to that may an element step with
// another one's values: each entry is compared with its own bound, which on flat cells is
// far below the largest entry's rounding.
class GeometryRounding {
  public:
    GeometryRounding(const hgg_problem_desc &desc, const HostOperators &op);
    // bounds for element e: of its elem_geo, then of its face_geo
    std::vector<double> bounds(int64_t e) const;

  private:
    const hgg_problem_desc &desc;
    const HostOperators &op;
    double eps[3] = {0.0, 0.0, 0.0};  // of a difference of coordinates along each axis
};

// Fills g (but for the device pointer) and nbr when the mesh qualifies: a sum-factorised
// handle of an order with a kernel, whose elements have equal upwind modes and ahat and
// sigma equal up to the coordinates' rounding (all of them then step with the first
// element's values); in the FP32 form, equal as that form rounds them, so that its results
// are the general kernels'.
bool tensor_lane_setup(const hgg_problem_desc &desc, const HostOperators &op, bool fp32, TensorLaneGeom &g,
                       std::vector<int32_t> &nbr);

// ---- simplices and the wave (lane_stage.cuh) -------------------------------------
// Elements with the same operators and geometry (a few groups on a structured mesh) are
// stored together: tiles of 32 elements of one group, up to `chunk_tiles` tiles of a group
// in a chunk, which is one block's work.  slot[e] = 32 tile + lane is element e's place.
struct LaneChunk {
    int32_t tile0, tiles, group, pad;
};
struct LaneMesh {
    int64_t n_slots = 0;
    bool sparse = false;               // more than twice as many padding slots as elements
    std::vector<int32_t> slot;         // [E]
    std::vector<int32_t> nbr;          // [tile][nfl][32] the neighbours' slots (padding: its own)
    std::vector<LaneChunk> chunks;
    std::vector<int64_t> representative;  // [group] its first element
};

// rows of an element's output one thread forms (all variables): the element's nb basis
// rows are split evenly over the fewest warps of at most max_rows rows
HGG_HOST_DEVICE constexpr int lane_warps(int nb, int max_rows) { return (nb + max_rows - 1) / max_rows; }
HGG_HOST_DEVICE constexpr int lane_rows(int nb, int max_rows) {
    return (nb + lane_warps(nb, max_rows) - 1) / lane_warps(nb, max_rows);
}
// the wave: four fields per row, so ten rows are 40 64-bit accumulators; the FP32 form
// keeps every face's two sums as well
HGG_HOST_DEVICE constexpr int lane_wave_rows(bool folded) { return folded ? 10 : 6; }
constexpr int kLaneAdvRows = 28;    // one field per row
// operator rows are padded to 16 bytes
HGG_HOST_DEVICE constexpr int lane_pad(int rows, int elem_bytes) { return elem_bytes == 8 ? (rows + 1) & ~1 : (rows + 3) & ~3; }
// basis functions that do not vanish on a face: the trace space of order p
HGG_HOST_DEVICE constexpr int lane_trace(int dim, int nfl, int p) {
    return dim == 2 ? p + 1 : (nfl == 4 ? (p + 1) * (p + 2) / 2 : (p + 1) * (p + 1));
}

// functions of the complete basis of order p
HGG_HOST_DEVICE constexpr int lane_basis(int dim, int nfl, int p) {
    return nfl == dim + 1 ? (dim == 2 ? (p + 1) * (p + 2) / 2 : (p + 1) * (p + 2) * (p + 3) / 6)
                          : (dim == 2 ? (p + 1) * (p + 1) : (p + 1) * (p + 1) * (p + 1));
}

// What a thread block reads of its group.  The sizes are in elements of the contraction
// type (8 bytes folded, 4 bytes in the FP32 form).
struct LaneTables {
    bool folded = true;              // folded geometry (64-bit handles), else as the FP32 form computes
    int elem_bytes = 8;              // contraction type
    size_t group_bytes = 0;          // bytes of one group's table, a multiple of 16
    int column_words = 0;            // the wave: words of the neighbours' column lists at its end
    std::vector<unsigned char> data;  // [group][group_bytes]
    std::vector<double> geometry;    // plain tables: every element's, [tile][Q][32]
};

// Groups the elements; false when whole tiles of them would take too much padding
// (unstructured meshes, very small ones).
// coefficient_bytes: of all vectors of the handle, per coefficient; spare_bytes: what the
// padding may take per element (and 4 MB).
bool lane_mesh(const hgg_problem_desc &desc, const HostOperators &op, int num_sms, int chunk_tiles_max, bool folded,
               int coefficient_bytes, int spare_bytes, LaneMesh &m);
// Tables of the groups: `folded` as described in lane_stage.cuh, or plain with entries of
// elem_bytes; false when the operators
// do not have the sparsity it relies on (a face couples more functions than its trace
// space has) or a flux form it does not take.
bool lane_wave_tables(const HostOperators &op, const LaneMesh &m, bool folded, int elem_bytes, LaneTables &t);
bool lane_advection_tables(const HostOperators &op, const LaneMesh &m, bool folded, int elem_bytes, LaneTables &t);

}  // namespace hgg
