// Sum-factorised stage kernel with one element per thread (tiled device layout):
// advection on quadrilaterals of order 1..5 and hexahedra of order 1 and 2 whose
// elements all have the same geometry (structured meshes).
//
// What bounds it: a stage moves 16 to 40 bytes per coefficient against 4 p + 10
// FP64 FMAs at most, so large meshes are bound by HBM and meshes that fit the L2
// by latency.  Both want many independent, fully coalesced loads per thread and no
// block-wide synchronisation:
//   * the vectors are stored in tiles of 32 elements, coefficient-major inside a
//     tile (as for the slice kernel), so a warp reads any one coefficient of its 32
//     elements as one 256-byte run, and so it does a neighbour's trace coefficients
//     when the neighbours are consecutive elements;
//   * a thread holds all coefficients of its element in registers (at most 36) and
//     forms its outputs from them: no shared memory, no barrier;
//   * all elements share one geometry, so the volume term ahat_c D1 of an axis and
//     the outflow face's lift sigma l (x) trace fold on the host into one 1D matrix
//     per axis, E_c = ahat_c D1 - sigma l_side (x) e_side, which the stage reads from
//     the kernel's parameters (the FP32 form keeps the general kernel's order of
//     operations instead, so its results do not change by FP32 roundings); per axis one
//     inflow face remains, whose neighbour index is all the geometry an element reads
//     (4 bytes per axis; the general kernels read 112 bytes per element in 3D).
// Measured, us per RK4 step, the one-shot and the pipelined kernel against this one: 32^2
// quadrilaterals at p = 2 17.7 and 20.3 -> 9.5, 150 x 210 at p = 4 56.0 and 65.8 -> 17.8.
#pragma once

#include <cstdint>
#include <type_traits>

#include "dg_kernels.cuh"
#include "host/lane.h"
#include "tensor_slice.cuh"

namespace hgg {

// One warp's work: the 32 elements of `tile`.  NIN: stage vectors in the stage input
// (0, 1, or -1 for a count read from io); FIN: the stage ends with the final update.
template <typename KT, int P, int DIM, int NIN, bool FIN>
__device__ __forceinline__ void tensor_lane_body(const StageIOT<KT> &io, const TensorLaneGeom &g, int64_t tile) {
    using CT = KT;  // contraction type
    constexpr int NP = P + 1, NB = DIM == 2 ? NP * NP : NP * NP * NP, NF = NB / NP;
    const int lane = threadIdx.x & 31;
    const int64_t e = tile * 32 + lane;
    if (e >= io.n_elements) return;
    const int64_t base = tile * (32 * NB) + lane;
    int32_t nb[DIM];
#pragma unroll
    for (int c = 0; c < DIM; ++c) nb[c] = g.side[c] >= 0 ? __ldg(g.nbr + (tile * DIM + c) * 32 + lane) : 0;

    chain_wait();
    // stage input of N coefficients at base + 32 pos(i), formed in FP64 and rounded once;
    // every vector's loads are issued together
    auto input = [&](auto count, auto pos, int64_t from, CT *out) {
        constexpr int N = decltype(count)::value;
        double v[N];
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = load_coef(io.u + from + 32 * pos(i));
        if (NIN != 0) {
            const int nin = NIN > 0 ? NIN : io.nin;
#pragma unroll 1
            for (int j = 0; j < nin; ++j) {
                const double cj = io.cin[j];
                const KT *kj = io.kin[j] + from;
#pragma unroll
                for (int i = 0; i < N; ++i) v[i] += cj * load_coef(kj + 32 * pos(i));
            }
        }
#pragma unroll
        for (int i = 0; i < N; ++i) out[i] = (CT)v[i];
    };
    CT w[NB];
    input(std::integral_constant<int, NB>{}, [](int i) { return i; }, base, w);
    CT tr[DIM][NF];
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
#pragma unroll
        for (int m = 0; m < NF; ++m) tr[c][m] = CT(0);
        if (g.side[c] < 0) continue;
        const int32_t n = nb[c];
        if (n < 0 || n >= io.n_elements) {
            atomicOr(io.status, 1);
            continue;
        }
        // the neighbour's trace on its opposite side: 1D mode 1 seen from our -1 side, 0 from our +1 side
        const int stride = c == 0 ? 1 : (c == 1 ? NP : NP * NP);
        const int64_t from = (int64_t)(n >> 5) * (32 * NB) + (n & 31) + (g.side[c] == 0 ? 32 * stride : 0);
        input(std::integral_constant<int, NF>{},
              [=](int m) {  // the tangential modes, lower axis first
                  const int lo = m % NP, hi = m / NP;
                  return c == 0 ? NP * lo + NP * NP * hi : (c == 1 ? lo + NP * NP * hi : lo + NP * hi);
              },
              from, tr[c]);
    }
    chain_next();
    double fu[FIN ? NB : 1];
    if (FIN) {
#pragma unroll
        for (int i = 0; i < NB; ++i) fu[i] = load_coef(io.u + base + 32 * i);
        for (int j = 0; j < io.nfin; ++j) {
            const double bj = io.bfin[j];
            const KT *kj = io.kfin[j] + base;
#pragma unroll
            for (int i = 0; i < NB; ++i) fu[i] += bj * load_coef(kj + 32 * i);
        }
    }
    // FP32 form: the rounded fluxes of every face
    CT flux[DIM][2][std::is_same_v<CT, float> ? NF : 1];
    if constexpr (std::is_same_v<CT, float>) {
#pragma unroll
        for (int c = 0; c < DIM; ++c)
#pragma unroll
            for (int sd = 0; sd < 2; ++sd) {
                const int stride = c == 0 ? 1 : (c == 1 ? NP : NP * NP);
                const bool in = g.side[c] == sd, out = (g.outflow[c] >> sd) & 1;
#pragma unroll
                for (int m = 0; m < NF; ++m) {
                    const int lo = m % NP, hi = m / NP;
                    const int pos = c == 0 ? NP * lo + NP * NP * hi : (c == 1 ? lo + NP * NP * hi : lo + NP * hi);
                    flux[c][sd][m] = in ? g.sigma[c][sd] * tr[c][m] : (out ? g.sigma[c][sd] * w[pos + sd * stride] : CT(0));
                }
            }
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const int a[3] = {i % NP, (i / NP) % NP, DIM == 3 ? i / (NP * NP) : 0};
        CT r = CT(0);
#pragma unroll
        for (int c = 0; c < DIM; ++c) {
            const int stride = c == 0 ? 1 : (c == 1 ? NP : NP * NP);
            if constexpr (std::is_same_v<CT, double>) {
#pragma unroll
                for (int k = 0; k < NP; ++k) r += g.E[(c * NP + a[c]) * NP + k] * w[i + (k - a[c]) * stride];
                r += g.L[c * NP + a[c]] * tr[c][c == 0 ? a[1] + NP * a[2] : (c == 1 ? a[0] + NP * a[2] : a[0] + NP * a[1])];
            } else {
                CT s = CT(0);
#pragma unroll
                for (int k = 0; k < NP; ++k) s += g.D1[a[c] * NP + k] * w[i + (k - a[c]) * stride];
                r += g.ahat[c] * s;
            }
        }
        if constexpr (std::is_same_v<CT, float>) {
            // the general kernel's order: the faces one after the other, each flux rounded
#pragma unroll
            for (int c = 0; c < DIM; ++c) {
                const int m = c == 0 ? a[1] + NP * a[2] : (c == 1 ? a[0] + NP * a[2] : a[0] + NP * a[1]);
#pragma unroll
                for (int sd = 0; sd < 2; ++sd) r -= g.lift[sd][a[c]] * flux[c][sd][m];
            }
        }
        if (io.kout) io.kout[base + 32 * i] = r;
        if (FIN) io.unew[base + 32 * i] = fu[i] + io.blast * (double)(KT)r;
    }
}

// one problem: a warp per tile
template <typename KT, int P, int DIM, int NIN, bool FIN>
__global__ void __launch_bounds__(128) tensor_lane(const __grid_constant__ StageIOT<KT> io,
                                                   const __grid_constant__ TensorLaneGeom g) {
    const int64_t tile = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (tile < g.n_tiles) tensor_lane_body<KT, P, DIM, NIN, FIN>(io, g, tile);
}

// calls f(NIN, FIN) with the compile-time stage shape of a stage with `nin` vectors in
// its input and (fin) the final update
template <typename F>
void lane_stage_shape(int nin, bool fin, F &&f) {
    using std::integral_constant;
    auto with = [&](auto n) {
        if (fin) f(n, std::true_type{});
        else f(n, std::false_type{});
    };
    if (nin == 0) with(integral_constant<int, 0>{});
    else if (nin == 1) with(integral_constant<int, 1>{});
    else with(integral_constant<int, -1>{});
}

// calls f(P, DIM) for the runtime order and dimension, if they have a kernel
template <typename F>
bool tensor_lane_dispatch(int dim, int order, F &&f) {
    using std::integral_constant;
    using D2 = integral_constant<int, 2>;
    using D3 = integral_constant<int, 3>;
    if (dim == 2) switch (order) {
            case 1: f(integral_constant<int, 1>{}, D2{}); return true;
            case 2: f(integral_constant<int, 2>{}, D2{}); return true;
            case 3: f(integral_constant<int, 3>{}, D2{}); return true;
            case 4: f(integral_constant<int, 4>{}, D2{}); return true;
            case 5: f(integral_constant<int, 5>{}, D2{}); return true;
        }
    if (dim == 3) switch (order) {
            case 1: f(integral_constant<int, 1>{}, D3{}); return true;
            case 2: f(integral_constant<int, 2>{}, D3{}); return true;
        }
    return false;
}

}  // namespace hgg
