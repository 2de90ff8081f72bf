// Stage kernels with one element per thread for simplices (advection) and for the wave
// on any shape, on meshes whose elements fall into few groups with the same operators
// and geometry (structured meshes).
//
// What bounds a stage there: the element's dense operators (tetrahedra at p = 2, wave:
// 1600 FP64 FMAs per element and stage on 40 coefficients), fed from shared memory or L1.
// A kernel whose thread forms one output row reads two values per FMA; this one reads the
// operators once per warp and four FMAs:
//   * the vectors are stored in tiles of 32 elements of one group, coefficient-major
//     inside a tile (LaneMesh), so a warp reads a coefficient of its 32 elements, or of
//     their neighbours across one face, as whole 256-byte runs;
//   * a block works on tiles of one group and copies that group's table into shared
//     memory once; every operator entry is then a broadcast (16 bytes at a time) used for
//     all 32 elements and, in the wave, for two of the four fields;
//   * a thread forms `RB` basis rows of every field (all of them up to 10 rows; larger
//     elements take several warps, each with its rows), so an input value loaded once
//     serves RB rows;
//   * 64-bit handles take tables folded with the group's geometry (lane_wave_tables,
//     lane_advection_tables): physical derivatives for the wave, one own matrix plus the
//     inflow faces' for advection; and a face operator keeps only the columns of the
//     functions that do not vanish on the face (6 of 10 for tetrahedra at p = 2), which
//     also are all that is read of a neighbour.  FP32 handles keep the general kernels'
//     operations in their order (plain tables, every element's own geometry), so their
//     results are the general kernels' bit for bit.
// Measured, us per RK4 step, the general kernel against this one: the upwind wave on
// 32^3 x 5 tetrahedra at p = 2 971 -> 260 (FP64), 831 -> 376 (FP32), the wave on
// 14 x 18 x 12 x 5 at p = 3 297 -> 97 and 239 -> 127, on 128^2 x 2 triangles at p = 4
// 217 -> 62 and 174 -> 86; advection on 192 x 160 x 2 triangles at p = 3 120 -> 18 and
// 78 -> 23, on 16^3 x 5 tetrahedra at p = 3 160 -> 26 and 116 -> 48.
#pragma once

#include <cstdint>
#include <type_traits>

#include "dg_kernels.cuh"
#include "host/lane.h"
#include "tensor_slice.cuh"

namespace hgg {

struct LaneGeom {
    const unsigned char *tables;  // [group][group_bytes]
    const LaneChunk *chunks;      // [n_chunks], one block each
    const int32_t *nbr;           // [tile][NFL][32] neighbour slots
    int64_t n_slots;
    int32_t n_chunks;
    int32_t group_bytes;
    int32_t column_words;         // the wave: last words of a table, the neighbours' trace columns [NFL][NFC] times 32
    // plain tables: [tile][Q][32] every element's geometry in 64 bits (wave: G [DIM][DIM], nu
    // [NFL][DIM]; advection: ahat [DIM], sigma [NFL]): its last bits decide exact ties of the
    // rounding to FP32, so it is not the group's
    const double *geo;
    int32_t neighbour_fp64;       // plain, the wave: n . s of a neighbour summed in FP64 (as the tile kernel does)
                                  // or in the contraction type (as the row kernel does)
};

// order whose basis has NB functions on the shape with NFL faces in DIM dimensions
template <int DIM, int NFL, int NB>
__host__ __device__ constexpr int lane_order() {
    for (int p = 1; p <= 5; ++p)
        if (lane_basis(DIM, NFL, p) == NB) return p;
    return 0;
}

// KT: the stage vectors' type; 64-bit handles take the folded tables, the FP32 form the
// plain ones (with its contraction type CT)
template <typename KT, typename CT, int DIM, int NFL, int NB, bool WAVE>
struct LaneShape {
    static constexpr bool FOLDED = std::is_same_v<KT, double>;
    static constexpr int MAXROWS = WAVE ? lane_wave_rows(FOLDED) : kLaneAdvRows;
    static constexpr int RW = lane_warps(NB, MAXROWS), RB = lane_rows(NB, MAXROWS);
    static constexpr int RBP = lane_pad(RB, sizeof(CT));
    static constexpr int NFC = lane_trace(DIM, NFL, lane_order<DIM, NFL, NB>());
    static constexpr int NC = FOLDED ? NFC : NB;  // columns of a neighbour (the wave)
    static constexpr int SCRATCH = FOLDED || !WAVE ? 0 : (int)sizeof(CT) * 32 * DIM * NB;  // bytes per tile
    static constexpr int TILES = RW >= 4 ? 1 : 4 / RW;  // tiles of a full chunk
    static constexpr int THREADS = 32 * RW * TILES;
};

template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int BYTES>
__device__ __forceinline__ void cp_async(void *dst, const void *src) {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"(BYTES) : "memory");
}
// the group's table into shared memory, by every thread of the block (not committed)
__device__ __forceinline__ void request_table(const LaneGeom &g, const unsigned char *table, unsigned char *dst) {
    for (int i = threadIdx.x; i < g.group_bytes / 16; i += blockDim.x) cp_async<16>(dst + 16 * i, table + 16 * i);
}

// acc[i] += a[i] x, a: RB entries of an operator column in shared memory (a broadcast)
template <int RB, typename CT>
__device__ __forceinline__ void column_load(const CT *a, CT (&o)[RB]) {
    constexpr int N = 16 / sizeof(CT);
    using Vec = std::conditional_t<sizeof(CT) == 8, double2, float4>;
#pragma unroll
    for (int i = 0; i < RB; i += N) {
        const Vec v = *reinterpret_cast<const Vec *>(a + i);
        o[i] = v.x;
        if (i + 1 < RB) o[i + 1] = v.y;
        if constexpr (sizeof(CT) == 4) {
            if (i + 2 < RB) o[i + 2] = v.z;
            if (i + 3 < RB) o[i + 3] = v.w;
        }
    }
}

// Outputs of RB rows of F fields, the fields `step` entries apart: this stage's derivative,
// the next stage's input (u + sum_j b_j k_j + wcoef k, the value the next stage would form
// itself) or the final update.  All fields' loads of one vector are issued together.
template <typename KT, typename CT, int F, int RB>
__device__ __forceinline__ void lane_output(const StageIOT<KT> &io, int64_t idx, int64_t step, int rows,
                                            const CT (&k)[F][RB]) {
    chain_next();
    if (io.kout) {
        KT *out = io.kout + idx;
#pragma unroll
        for (int f = 0; f < F; ++f)
#pragma unroll
            for (int i = 0; i < RB; ++i)
                if (i < rows) out[f * step + 32 * i] = (KT)k[f][i];
    }
    if (!io.wnext && !io.unew) return;
    double r[F][RB];
    const double *u = io.u + idx;
#pragma unroll
    for (int f = 0; f < F; ++f)
#pragma unroll
        for (int i = 0; i < RB; ++i) r[f][i] = i < rows ? load_coef(u + f * step + 32 * i) : 0.0;
#pragma unroll 1
    for (int j = 0; j < io.nfin; ++j) {
        const double bj = io.bfin[j];
        const KT *kj = io.kfin[j] + idx;
#pragma unroll
        for (int f = 0; f < F; ++f)
#pragma unroll
            for (int i = 0; i < RB; ++i)
                if (i < rows) r[f][i] += bj * load_coef(kj + f * step + 32 * i);
    }
    if (io.wnext) {
        CT *out = reinterpret_cast<CT *>(io.wnext) + idx;
        const double c = io.wcoef;
#pragma unroll
        for (int f = 0; f < F; ++f)
#pragma unroll
            for (int i = 0; i < RB; ++i)
                if (i < rows) out[f * step + 32 * i] = (CT)(c != 0.0 ? r[f][i] + c * (double)(KT)k[f][i] : r[f][i]);
    }
    if (io.unew) {
        double *out = io.unew + idx;
#pragma unroll
        for (int f = 0; f < F; ++f)
#pragma unroll
            for (int i = 0; i < RB; ++i)
                if (i < rows) out[f * step + 32 * i] = r[f][i] + io.blast * (double)k[f][i];
    }
}

// ---- the wave ---------------------------------------------------------------------
// An element's data is read by all warps that form its rows, and the loads of a face's 24
// to 60 values per element would take registers the accumulators need: each tile keeps its
// 32 elements' input and a ring of two faces' neighbour traces in shared memory, filled by
// asynchronous copies.  The first two faces are in flight while the volume term is formed,
// face f + 2 while face f + 1 is.  (Read straight from global memory the kernel stalled on
// those loads: 114 us per stage on 32^3 x 5 tetrahedra at p = 2, FP64 pipe 20 % busy.)
constexpr int kLaneRing = 2;

// operations the compiler may not contract
__device__ __forceinline__ float lane_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double lane_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float lane_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double lane_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float lane_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double lane_fma(double a, double b, double c) { return __fma_rn(a, b, c); }

// dynamic shared memory: the group's table, then per tile the elements' input [R][32] and
// the ring of faces [V][NC][32], in elements of the source type; NC columns of a neighbour:
// its trace functions in a folded table, any with a nonzero entry in a plain one
// (plain tables: and a scratch [DIM][NB][32] of the contraction type)
template <typename ST, int DIM, int NB, int NC, int SCRATCH>
__host__ __device__ constexpr int lane_tile_bytes() {
    return (int)sizeof(ST) * 32 * (DIM + 1) * (NB + kLaneRing * NC) + SCRATCH;
}

// ST: type of the stage input's vector (double: the solution; the contraction type: the
// input the previous stage formed).
template <typename KT, typename CT, typename ST, int DIM, int NFL, int NB>
__device__ __forceinline__ void wave_lane_body(const StageIOT<KT> &io, const LaneGeom &g, int64_t block) {
    using SH = LaneShape<KT, CT, DIM, NFL, NB, true>;
    constexpr int RW = SH::RW, RB = SH::RB, RBP = SH::RBP, NFC = SH::NFC, NC = SH::NC, V = DIM + 1, R = V * NB;
    extern __shared__ __align__(16) unsigned char lane_shared[];
    const LaneChunk ch = g.chunks[block];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int local = warp / RW, rw = warp % RW;
    const bool active = local < ch.tiles;
    const int64_t tile = ch.tile0 + (active ? local : 0);
    const ST *src = std::is_same_v<ST, double> && (!io.win || !std::is_same_v<CT, double>)
                        ? reinterpret_cast<const ST *>(io.u)
                        : reinterpret_cast<const ST *>(io.win);
    const unsigned char *table = g.tables + (size_t)ch.group * g.group_bytes;
    ST *own = reinterpret_cast<ST *>(lane_shared + g.group_bytes + local * lane_tile_bytes<ST, DIM, NB, NC, SH::SCRATCH>());
    ST *ring = own + 32 * R;
    // column lists [NFL][NC], at the end of the table (read here from global memory: the copy of the
    // table is still in flight when the neighbours' addresses are formed)
    const int32_t *gcols = reinterpret_cast<const int32_t *>(table + g.group_bytes - 4 * g.column_words);
    int32_t nb[NFL];
#pragma unroll
    for (int f = 0; f < NFL; ++f) nb[f] = __ldg(g.nbr + (tile * NFL + f) * 32 + lane);

    request_table(g, table, lane_shared);
    chain_wait();
    if (active)
        for (int i = rw * 32 + lane; i < (int)sizeof(ST) * 2 * R; i += 32 * RW)
            cp_async<16>(reinterpret_cast<unsigned char *>(own) + 16 * i,
                         reinterpret_cast<const unsigned char *>(src + tile * (32 * R)) + 16 * i);
    cp_async_commit();
    auto request = [&](int f) {  // the neighbours across face f (one commit, empty past the last face)
        if (f < NFL && active) {
            int32_t n = nb[0];
#pragma unroll
            for (int k = 1; k < NFL; ++k) n = f == k ? nb[k] : n;
            if (n < 0 || n >= g.n_slots) {
                atomicOr(io.status, 1);
                n = 0;
            }
            const ST *other = src + (int64_t)(n >> 5) * (32 * R) + (n & 31);
            ST *dst = ring + (f % kLaneRing) * (32 * V * NC) + lane;
            if constexpr (SH::FOLDED) {
                // lane m holds the place of the face's m-th trace function
                const int32_t col = lane < NC ? __ldg(gcols + f * NC + lane) : 0;
#pragma unroll
                for (int m0 = 0; m0 < NC; m0 += RW) {
                    const int m = m0 + rw;
                    const ST *from = other + __shfl_sync(0xffffffffu, col, m & 31);
                    if (m < NC)
#pragma unroll
                        for (int v = 0; v < V; ++v) cp_async<sizeof(ST)>(dst + 32 * (v * NC + m), from + 32 * v * NB);
                }
            } else {
#pragma unroll 4
                for (int q = rw; q < R; q += RW) cp_async<sizeof(ST)>(dst + 32 * q, other + 32 * q);
            }
        }
        cp_async_commit();
    };
    request(0);
    request(1);
    // what the outputs will read, into L2 meanwhile
    if (active && rw == 0 && lane == 0) {
        if (io.wnext || io.unew) {
            if (src != reinterpret_cast<const ST *>(io.u)) prefetch_l2(io.u + tile * (32 * R), 32 * R * sizeof(double));
            for (int j = 0; j < io.nfin; ++j) prefetch_l2(io.kfin[j] + tile * (32 * R), 32 * R * sizeof(KT));
        }
    }
    cp_async_wait<kLaneRing>();
    __syncthreads();  // the table and every tile's own input
    if (!active) return;
    auto tile_sync = [&]() {  // the warps of this tile
        if constexpr (RW == 1) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(local + 1), "n"(32 * RW) : "memory");
    };
    const int rows = min(RB, NB - rw * RB);
    const int64_t out = tile * (32 * R) + lane + 32 * (rw * RB);
    const CT *ops = reinterpret_cast<const CT *>(lane_shared);
    CT *scratch = reinterpret_cast<CT *>(ring + kLaneRing * (32 * V * NC)) + lane;  // plain tables: [DIM][NB][32]
    own += lane;  // (the copies of later faces still go by the ring's start)

    if constexpr (SH::FOLDED) {
        constexpr int OPS = (DIM * NB + 2 * NFL * NFC) * RBP;  // of one row warp
        const double *op = ops + rw * OPS;
        const double *head = ops + RW * OPS;  // per face nu[DIM], c |nu|, invc nu[DIM], c nu / |nu|; invc
        const int32_t *cols = reinterpret_cast<const int32_t *>(head + NFL * (1 + 3 * DIM) + 1);  // [NFL][NFC] own
        double K[V][RB];  // pressure, velocity
#pragma unroll
        for (int i = 0; i < RB; ++i) {
            K[0][i] = 0.0;
#pragma unroll
            for (int d = 0; d < DIM; ++d) K[1 + d][i] = 0.0;
        }
#pragma unroll 2
        for (int j = 0; j < NB; ++j) {
            const double q = own[32 * j];
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                const double s = own[32 * ((d + 1) * NB + j)];
                double o[RB];
                column_load<RB>(op + (j * DIM + d) * RBP, o);
#pragma unroll
                for (int i = 0; i < RB; ++i) {
                    K[0][i] += o[i] * s;
                    K[1 + d][i] += o[i] * q;
                }
            }
        }
        const double invc = head[NFL * (1 + 3 * DIM)];
#pragma unroll
        for (int d = 0; d < DIM; ++d)
#pragma unroll
            for (int i = 0; i < RB; ++i) K[1 + d][i] *= invc;
        op += DIM * NB * RBP;
#pragma unroll 1
        for (int f = 0; f < NFL; ++f) {
            const double *h = head + f * (1 + 3 * DIM);
            const int32_t *cf = cols + f * NFC;
            const ST *other = ring + (f % kLaneRing) * (32 * V * NC) + lane;
            double nu[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d) nu[d] = h[d];
            double B[RB], J[RB];  // lifted jumps of the pressure and of nu . s
#pragma unroll
            for (int i = 0; i < RB; ++i) B[i] = J[i] = 0.0;
            cp_async_wait<kLaneRing - 1>();
            tile_sync();  // face f of every warp of the tile
#pragma unroll 2
            for (int m = 0; m < NFC; ++m) {
                const int js = cf[m];
                const double qs = own[js], qn = other[32 * m];
                double ss = 0.0, sn = 0.0;
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    ss += nu[d] * own[js + 32 * (d + 1) * NB];
                    sn += nu[d] * other[32 * ((d + 1) * NFC + m)];
                }
                double o[RB];
                column_load<RB>(op + (2 * m) * RBP, o);
#pragma unroll
                for (int i = 0; i < RB; ++i) {
                    B[i] += o[i] * qs;
                    J[i] += o[i] * ss;
                }
                column_load<RB>(op + (2 * m + 1) * RBP, o);
#pragma unroll
                for (int i = 0; i < RB; ++i) {
                    B[i] -= o[i] * qn;
                    J[i] -= o[i] * sn;
                }
            }
            op += 2 * NFC * RBP;
            tile_sync();  // the face's buffer is read
            request(f + kLaneRing);
            const double cn = h[DIM];
#pragma unroll
            for (int i = 0; i < RB; ++i) {
                K[0][i] -= J[i] + cn * B[i];
#pragma unroll
                for (int d = 0; d < DIM; ++d) K[1 + d][i] -= h[DIM + 1 + d] * B[i] + h[2 * DIM + 1 + d] * J[i];
            }
        }
        lane_output<KT, CT, V, RB>(io, out, 32 * NB, rows, K);
    } else {
        constexpr int OPS = (DIM * NB + 2 * NFL * NB) * RBP;
        const CT *op = ops + rw * OPS;
        const CT cu = ops[RW * OPS], invc = ops[RW * OPS + 1];
        const double *geo = g.geo + tile * (32 * (DIM * DIM + NFL * DIM)) + lane, *geo_nu = geo + 32 * DIM * DIM;
        CT G[DIM * DIM];
#pragma unroll
        for (int i = 0; i < DIM * DIM; ++i) G[i] = (CT)ldg_f64(geo + 32 * i);
        // t_c = sum_d G_dc s_d, formed once per tile
        for (int j = rw; j < NB; j += RW) {
            CT s[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d) s[d] = (CT)own[32 * ((d + 1) * NB + j)];
#pragma unroll
            for (int c = 0; c < DIM; ++c) {
                CT t = lane_mul(G[c], s[0]);
#pragma unroll
                for (int d = 1; d < DIM; ++d) t = lane_fma(G[d * DIM + c], s[d], t);
                scratch[32 * (c * NB + j)] = t;
            }
        }
        tile_sync();
        CT K[V][RB];
        {
            CT Pc[DIM][RB], A[DIM][RB];
#pragma unroll
            for (int c = 0; c < DIM; ++c)
#pragma unroll
                for (int i = 0; i < RB; ++i) Pc[c][i] = A[c][i] = CT(0);
#pragma unroll 2
            for (int j = 0; j < NB; ++j) {
                const CT q = (CT)own[32 * j];
#pragma unroll
                for (int c = 0; c < DIM; ++c) {
                    const CT t = scratch[32 * (c * NB + j)];
                    CT o[RB];
                    column_load<RB>(op + (j * DIM + c) * RBP, o);
#pragma unroll
                    for (int i = 0; i < RB; ++i) {
                        Pc[c][i] += o[i] * t;
                        A[c][i] += o[i] * q;
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < RB; ++i) {
                K[0][i] = CT(0);
#pragma unroll
                for (int c = 0; c < DIM; ++c) K[0][i] += Pc[c][i];
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    K[1 + d][i] = CT(0);
#pragma unroll
                    for (int c = 0; c < DIM; ++c) K[1 + d][i] += G[d * DIM + c] * A[c][i];
                }
            }
        }
        op += DIM * NB * RBP;
        CT Bf[NFL][RB], Jf[NFL][RB];
#pragma unroll
        for (int f = 0; f < NFL; ++f) {
            ST *other = ring + (f % kLaneRing) * (32 * V * NC) + lane;
            CT nu[DIM];
            double nud[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                nud[d] = ldg_f64(geo_nu + 32 * (f * DIM + d));
                nu[d] = (CT)nud[d];
            }
#pragma unroll
            for (int i = 0; i < RB; ++i) Bf[f][i] = Jf[f][i] = CT(0);
            cp_async_wait<kLaneRing - 1>();
            tile_sync();
            // n . s of both sides, formed once per tile; the neighbour's takes its first component's place
            for (int j = rw; j < NB; j += RW) {
                CT ss = lane_mul(nu[0], (CT)own[32 * (NB + j)]);
#pragma unroll
                for (int d = 1; d < DIM; ++d) ss = lane_fma(nu[d], (CT)own[32 * ((d + 1) * NB + j)], ss);
                scratch[32 * j] = ss;
                CT sn;
                if (g.neighbour_fp64) {
                    double x = 0.0;
#pragma unroll
                    for (int d = 0; d < DIM; ++d) x += nud[d] * (double)(CT)other[32 * ((d + 1) * NB + j)];
                    sn = (CT)x;
                } else {
                    sn = lane_mul(nu[0], (CT)other[32 * (NB + j)]);
#pragma unroll
                    for (int d = 1; d < DIM; ++d) sn = lane_fma(nu[d], (CT)other[32 * ((d + 1) * NB + j)], sn);
                }
                other[32 * (NB + j)] = (ST)sn;
            }
            tile_sync();
#pragma unroll 4
            for (int j = 0; j < NB; ++j) {
                const CT qs = (CT)own[32 * j], ss = scratch[32 * j];
                const CT qn = (CT)other[32 * j], sn = (CT)other[32 * (NB + j)];
                CT os[RB], on[RB];
                column_load<RB>(op + (2 * j) * RBP, os);
                column_load<RB>(op + (2 * j + 1) * RBP, on);
                // (the general kernels' order: the difference of the two products, then its sum)
#pragma unroll
                for (int i = 0; i < RB; ++i) {
                    Jf[f][i] = lane_add(Jf[f][i], lane_fma(os[i], ss, -lane_mul(on[i], sn)));
                    Bf[f][i] = lane_add(Bf[f][i], lane_fma(os[i], qs, -lane_mul(on[i], qn)));
                }
            }
            op += 2 * NB * RBP;
            tile_sync();  // the face's buffer and the scratch are read
            request(f + kLaneRing);
#pragma unroll
            for (int i = 0; i < RB; ++i) {
                K[0][i] -= Jf[f][i];
#pragma unroll
                for (int d = 0; d < DIM; ++d) K[1 + d][i] -= nu[d] * Bf[f][i];
            }
        }
#pragma unroll
        for (int i = 0; i < RB; ++i)
#pragma unroll
            for (int d = 0; d < DIM; ++d) K[1 + d][i] *= invc;
        if (cu != CT(0)) {
#pragma unroll
            for (int f = 0; f < NFL; ++f) {
                double nu[DIM], q = 0.0;
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    nu[d] = ldg_f64(geo_nu + 32 * (f * DIM + d));
                    q += nu[d] * nu[d];
                }
                const CT n = (CT)sqrt(q);
                CT along[DIM];
#pragma unroll
                for (int d = 0; d < DIM; ++d) along[d] = cu * ((CT)nu[d] / n);
#pragma unroll
                for (int i = 0; i < RB; ++i) {
                    K[0][i] -= cu * n * Bf[f][i];
#pragma unroll
                    for (int d = 0; d < DIM; ++d) K[1 + d][i] -= along[d] * Jf[f][i];
                }
            }
        }
        lane_output<KT, CT, V, RB>(io, out, 32 * NB, rows, K);
    }
}

template <typename KT, typename CT, typename ST, int DIM, int NFL, int NB>
__global__ void __launch_bounds__(LaneShape<KT, CT, DIM, NFL, NB, true>::THREADS)
    wave_lane(const __grid_constant__ StageIOT<KT> io, const __grid_constant__ LaneGeom g) {
    wave_lane_body<KT, CT, ST, DIM, NFL, NB>(io, g, blockIdx.x);
}
// dynamic shared memory of a block of `tiles` tiles
template <typename KT, typename CT, typename ST, int DIM, int NFL, int NB>
int wave_lane_smem(int group_bytes, int tiles) {
    using SH = LaneShape<KT, CT, DIM, NFL, NB, true>;
    return group_bytes + tiles * lane_tile_bytes<ST, DIM, NB, SH::NC, SH::SCRATCH>();
}

// ---- advection ----------------------------------------------------------------------
// NIN: stage vectors in the stage input (0, 1, or -1 for a count read from io); they are
// combined on loading, in FP64 and rounded once, so no vector is formed ahead.
// Small elements (REG) hold all their inputs in registers: one round of loads, in flight
// with the table, then arithmetic alone.  Larger ones load up to ten columns at a time.
template <typename KT, typename CT, int DIM, int NFL, int NB, int NIN>
__device__ __forceinline__ void advection_lane_body(const StageIOT<KT> &io, const LaneGeom &g, int64_t block) {
    using SH = LaneShape<KT, CT, DIM, NFL, NB, false>;
    constexpr int RW = SH::RW, RB = SH::RB, RBP = SH::RBP, NFC = SH::NFC;
    constexpr int NC = SH::FOLDED ? NFC : NB;  // columns of a face
    constexpr bool REG = NB <= (SH::FOLDED ? 21 : 15);
    constexpr bool FACES_AHEAD = REG && NFL * NC <= 40;
    constexpr int CH = REG ? (NB > NC ? NB : NC) : 10;  // columns loaded together
    constexpr int OPS = (SH::FOLDED ? NB + NFL * NFC : (DIM + NFL) * NB) * RBP;  // of one row warp
    extern __shared__ __align__(16) unsigned char lane_shared[];
    const LaneChunk ch = g.chunks[block];
    const unsigned char *table = g.tables + (size_t)ch.group * g.group_bytes;
    request_table(g, table, lane_shared);
    cp_async_commit();
    // folded: number of inflow faces, [NFL] face, [NFL][NFC] column; plain: [NFL] upwind mode
    // (read from global memory: the table is in flight)
    const int32_t *head = reinterpret_cast<const int32_t *>(table + sizeof(CT) * RW * OPS);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int local = warp / RW, rw = warp % RW;
    const bool active = local < ch.tiles;
    const int64_t tile = ch.tile0 + (active ? local : 0);
    const int64_t base = tile * (32 * NB) + lane;
    int32_t nb[NFL];
#pragma unroll
    for (int f = 0; f < NFL; ++f) nb[f] = __ldg(g.nbr + (tile * NFL + f) * 32 + lane);
    const double *geo = g.geo + tile * (32 * (DIM + NFL)) + lane;  // plain
    CT ahat[DIM], sigma[NFL];
    if constexpr (!SH::FOLDED) {
#pragma unroll
        for (int c = 0; c < DIM; ++c) ahat[c] = (CT)ldg_f64(geo + 32 * c);
#pragma unroll
        for (int f = 0; f < NFL; ++f) sigma[f] = (CT)ldg_f64(geo + 32 * (DIM + f));
    }
    // the k-th neighbour that enters the stage: the face, or -1
    auto inflow = [&](int k) {
        if constexpr (SH::FOLDED) return k < __ldg(head) ? __ldg(head + 1 + k) : -1;
        else return __ldg(head + k) == 2 ? k : -1;
    };
    auto neighbour = [&](int f) {  // first coefficient of the neighbour across face f
        int32_t n = nb[0];
#pragma unroll
        for (int k = 1; k < NFL; ++k) n = f == k ? nb[k] : n;
        if (n < 0 || n >= g.n_slots) {
            atomicOr(io.status, 1);
            n = 0;
        }
        return (int64_t)(n >> 5) * (32 * NB) + (n & 31);
    };
    // stage input of up to CH coefficients at from + offset(i), i < count
    auto input = [&](int64_t from, int count, auto offset, CT *x) {
        double v[CH];
#pragma unroll
        for (int i = 0; i < CH; ++i) v[i] = i < count ? load_coef(io.u + from + offset(i)) : 0.0;
        if (NIN != 0) {
            const int nin = NIN > 0 ? NIN : io.nin;
#pragma unroll 1
            for (int j = 0; j < nin; ++j) {
                const double cj = io.cin[j];
                const KT *kj = io.kin[j] + from;
#pragma unroll
                for (int i = 0; i < CH; ++i)
                    if (i < count) v[i] += cj * load_coef(kj + offset(i));
            }
        }
#pragma unroll
        for (int i = 0; i < CH; ++i) x[i] = (CT)v[i];
    };
    auto own_input = [&](int j, CT *x) { input(base, min(NB - j, CH), [=](int i) { return 32 * (j + i); }, x); };
    auto face_input = [&](int k, int f, int j, CT *x) {
        const int64_t from = neighbour(f);
        if constexpr (SH::FOLDED) {
            const int32_t *cols = head + 1 + NFL + k * NFC + j;
            input(from, min(NC - j, CH), [=](int i) { return __ldg(cols + i); }, x);
        } else {
            input(from, min(NC - j, CH), [=](int i) { return 32 * (j + i); }, x);
        }
    };
    chain_wait();
    CT xo[CH], xn[FACES_AHEAD ? NFL : 1][CH];
    if (active) {
        own_input(0, xo);
        if constexpr (FACES_AHEAD) {
#pragma unroll
            for (int k = 0; k < NFL; ++k) {
                const int f = inflow(k);
                if (f >= 0) face_input(k, f, 0, xn[k]);
            }
        }
    }
    cp_async_wait<0>();
    __syncthreads();  // the table
    if (!active) return;
    const int rows = min(RB, NB - rw * RB);
    const CT *op = reinterpret_cast<const CT *>(lane_shared) + rw * OPS;
    CT acc[1][RB];
#pragma unroll
    for (int i = 0; i < RB; ++i) acc[0][i] = CT(0);
    // out += the operator's columns j .. j + CH (of n) times x; stride: entries between columns
    auto columns = [&](const CT *a, int stride, int n, const CT *x, CT *out) {
#pragma unroll
        for (int q = 0; q < CH; ++q) {
            if (q >= n) continue;
            CT o[RB];
            column_load<RB>(a + q * stride, o);
#pragma unroll
            for (int i = 0; i < RB; ++i) out[i] += o[i] * x[q];
        }
    };
    if constexpr (SH::FOLDED) {
        columns(op, RBP, NB, xo, acc[0]);
        if constexpr (!REG) {
#pragma unroll 1
            for (int j = CH; j < NB; j += CH) {
                own_input(j, xo);
                columns(op + j * RBP, RBP, NB - j, xo, acc[0]);
            }
        }
        op += NB * RBP;
        if constexpr (FACES_AHEAD) {
#pragma unroll
            for (int k = 0; k < NFL; ++k)
                if (inflow(k) >= 0) columns(op + k * NC * RBP, RBP, NC, xn[k], acc[0]);
        } else {
#pragma unroll 1
            for (int k = 0; k < NFL; ++k) {
                const int f = inflow(k);
                if (f < 0) break;
#pragma unroll 1
                for (int j = 0; j < NC; j += CH) {
                    face_input(k, f, j, xo);
                    columns(op + (k * NC + j) * RBP, RBP, NC - j, xo, acc[0]);
                }
            }
        }
    } else {
        // the row kernel's order of operations: the axes' sums, then the faces' one after the other
        CT s[DIM][RB];
#pragma unroll
        for (int c = 0; c < DIM; ++c) {
#pragma unroll
            for (int i = 0; i < RB; ++i) s[c][i] = CT(0);
            columns(op + c * RBP, DIM * RBP, NB, xo, s[c]);
        }
        if constexpr (!REG) {
#pragma unroll 1
            for (int j = CH; j < NB; j += CH) {
                own_input(j, xo);
#pragma unroll
                for (int c = 0; c < DIM; ++c) columns(op + (j * DIM + c) * RBP, DIM * RBP, NB - j, xo, s[c]);
            }
        }
#pragma unroll
        for (int c = 0; c < DIM; ++c)
#pragma unroll
            for (int i = 0; i < RB; ++i) acc[0][i] += ahat[c] * s[c][i];
        op += DIM * NB * RBP;
        auto flux = [&](int f, const CT *t) {  // each face's rounded, then added
#pragma unroll
            for (int i = 0; i < RB; ++i) acc[0][i] = lane_add(acc[0][i], -lane_mul(sigma[f], t[i]));
        };
#pragma unroll
        for (int f = 0; f < NFL; ++f) {
            const int md = __ldg(head + f);
            if (md != 1 && md != 2) continue;
            CT t[RB];
#pragma unroll
            for (int i = 0; i < RB; ++i) t[i] = CT(0);
            const CT *a = op + f * NB * RBP;
            if constexpr (FACES_AHEAD) {
                if (md == 1) columns(a, RBP, NB, xo, t);
                else columns(a, RBP, NB, xn[f], t);
            } else {
#pragma unroll 1
                for (int j = 0; j < NB; j += CH) {
                    CT x[CH];
                    if (md == 1) own_input(j, x);
                    else face_input(f, f, j, x);
                    columns(a + j * RBP, RBP, NB - j, x, t);
                }
            }
            flux(f, t);
        }
    }
    lane_output<KT, CT, 1, RB>(io, base + 32 * (rw * RB), 0, rows, acc);
}

template <typename KT, typename CT, int DIM, int NFL, int NB, int NIN>
__global__ void __launch_bounds__(LaneShape<KT, CT, DIM, NFL, NB, false>::THREADS)
    advection_lane(const __grid_constant__ StageIOT<KT> io, const __grid_constant__ LaneGeom g) {
    advection_lane_body<KT, CT, DIM, NFL, NB, NIN>(io, g, blockIdx.x);
}

// basis sizes with a lane kernel: the wave up to 36 functions in 2D and 3D, advection on simplices
constexpr bool lane_size(int dim, int nfl, bool wave, int nb) {
    return dim >= 2 && (wave ? nb <= 36 : nfl == dim + 1 && nb <= 56);
}

}  // namespace hgg
