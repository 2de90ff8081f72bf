// Set-up of the one-element-per-thread stage kernels (tensor_lane.cuh): the meshes
// they take and the operators their threads share.
#pragma once

#include <cstdint>
#include <vector>

#include "operators.h"

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

// Fills g (but for the device pointer) and nbr when the mesh qualifies: a sum-factorised
// handle of an order with a kernel, whose elements agree in ahat, sigma and upwind modes
// to 2^-40 of the largest entry (the cells of a structured mesh differ by the rounding of
// their vertex coordinates; all of them then step with the first element's values).
bool tensor_lane_setup(const HostOperators &op, TensorLaneGeom &g, std::vector<int32_t> &nbr);

}  // namespace hgg
