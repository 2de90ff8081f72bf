// Runge-Kutta stage kernel of HpgemAPILinear's stored-matrix form
// (kernel/Base/HpgemAPILinear_Impl.h): per element
//   w_e = u_e + sum_j dt a_ij k_j,e                     (getLinearCombinationOfVectors)
//   k_e = D_e w_e + sum_s N_{e,s} w_{n(e,s)}            (multiplyStiffnessMatrices, :360-434,
//                                                        then solveMassMatrixEquations, :143-156,
//                                                        with M_e^{-1} folded into D and N)
// and in the final stage u_new = u + sum_j dt b_j k_j.  The distinct matrices
// are few on structured meshes, so they stay in L1/L2 while the per-element
// stage vectors stream from HBM.
#pragma once

#include <cstdint>

#include "dg_kernels.cuh"

namespace hgg {

// Status word bits set here: 1 a neighbour index out of range, 4 a matrix
// index out of range (2 is the bounded-wait bit of the persistent kernels).
struct LinearGeom {
    const double *table;      // [n_mats][R][R] transposed: table[m][j][i] = (matrix m)_{ij}
    const double *table_rm;   // [n_mats][R][R] row-major (the grouped kernel's copy), or null
    const float *table_f;     // the same in FP32 (FP32-mixed form with FP32 contractions), else null
    const int32_t *self_mat;  // [E]
    const int32_t *nbr;       // [E][slots], -1: unused slot
    const int32_t *nbr_mat;   // [E][slots]
    int R, slots, epb, n_mats;
};

template <typename CT>
__device__ __forceinline__ const CT *linear_table(const LinearGeom &g);
template <>
__device__ __forceinline__ const double *linear_table<double>(const LinearGeom &g) { return g.table; }
template <>
__device__ __forceinline__ const float *linear_table<float>(const LinearGeom &g) { return g.table_f; }

// threads and dynamic shared memory of one block of `epb` elements
__host__ __device__ inline int linear_threads(int R, int epb) { return ((epb * R + 31) / 32) * 32; }
__host__ __device__ inline size_t linear_smem(int R, int slots, int epb, size_t elem) {
    return elem * (size_t)epb * R * (1 + slots);
}

// Thread (el, r) of the block produces row r of element el: the matrices are
// stored transposed, so at every column j the threads of one element read
// consecutive entries.  KT: stage-vector type; CT: contraction type.
template <typename KT, typename CT>
__global__ void __launch_bounds__(256) linear_stage(const StageIOT<KT> io, const LinearGeom g) {
    extern __shared__ __align__(16) unsigned char linear_shared[];
    const int R = g.R, S = g.slots, epb = g.epb;
    CT *W = reinterpret_cast<CT *>(linear_shared);  // [epb][R]
    CT *WN = W + (size_t)epb * R;                  // [epb][S][R]
    const int tid = threadIdx.x;
    const int64_t e0 = (int64_t)blockIdx.x * epb;
    const int el = tid / R, r = tid % R;
    const int64_t e = e0 + el;
    const bool active = el < epb && e < io.n_elements;
    double u_own = 0.0;
    if (active) {
        const int64_t idx = e * R + r;
        u_own = io.u[idx];
        double w = u_own;
        for (int j = 0; j < io.nin; ++j) w += io.cin[j] * (double)io.kin[j][idx];
        W[el * R + r] = (CT)w;
    }
    for (int k = tid; k < epb * S * R; k += blockDim.x) {
        const int l = k / (S * R), s = (k / R) % S, rr = k % R;
        const int64_t ee = e0 + l;
        double v = 0.0;
        if (ee < io.n_elements) {
            const int32_t n = g.nbr[ee * S + s];
            if (n >= 0 && n < io.n_elements) v = stage_input(io, (int64_t)n * R + rr);
            else if (n >= 0) atomicOr(io.status, 1);
        }
        WN[(size_t)(l * S + s) * R + rr] = (CT)v;
    }
    __syncthreads();
    if (!active) return;

    const CT *T = linear_table<CT>(g);
    const size_t RR = (size_t)R * R;
    CT acc = CT(0);
    int32_t m = g.self_mat[e];
    if (m >= 0 && m < g.n_mats) {
        const CT *op = T + (size_t)m * RR + r;
        const CT *w = W + el * R;
#pragma unroll 8
        for (int j = 0; j < R; ++j) acc += op[(size_t)j * R] * w[j];
    } else {
        atomicOr(io.status, 4);
    }
    for (int s = 0; s < S; ++s) {
        m = g.nbr_mat[e * S + s];
        if (m < 0) continue;
        if (m >= g.n_mats) {
            atomicOr(io.status, 4);
            continue;
        }
        const CT *op = T + (size_t)m * RR + r;
        const CT *wn = WN + (size_t)(el * S + s) * R;
#pragma unroll 8
        for (int j = 0; j < R; ++j) acc += op[(size_t)j * R] * wn[j];
    }
    stage_output(io, e * R + r, u_own, (double)acc);
}

// ---------------------------------------------------------------------------
// grouped form: tiles of kLinTileN elements that share all their matrices
// ---------------------------------------------------------------------------
// On a structured mesh the elements fall into a few groups with identical
// matrices (one group on a hexahedral mesh, ten on the five-tetrahedron split),
// so a tile's stage is a dense product Out[R][64] = sum_s A_s[R][R] W_s[R][64]
// with W_s the stage inputs of the tile's elements (s = 0) or of their
// neighbours in slot s.  It runs on the FP64 tensor cores (DMMA, m8n8k4):
// 8 warps, warp w owns elements 8w..8w+7, each warp all row bands of 8.
constexpr int kLinTileN = 64;            // elements per tile
constexpr int kLinKC = 32;               // k (column) chunk staged in shared memory
constexpr int kLinRows = 64;             // output rows per pass
constexpr int kLinStride = kLinKC + 4;   // padded row stride (doubles): fragment loads conflict-free
constexpr int kLinOutStride = kLinRows + 1;
constexpr int kLinTileMinRows = 15;      // smaller elements run the row kernel

struct LinearTiles {
    const int32_t *elems;  // [n_tiles][kLinTileN] element ids, -1: padding
    const int32_t *mats;   // [n_tiles][1 + slots] the tile's matrices (-1: unused slot)
};

__device__ __forceinline__ void dmma_m8n8k4(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// One tile (256 threads).  Called by the one-problem launch (tile = blockIdx.x)
// and by the batch's persistent launch (tile = the block's index in its problem).
template <typename KT>
__device__ __forceinline__ void linear_tile_body(const StageIOT<KT> &io, const LinearGeom &g, const LinearTiles &t,
                                                 int64_t tile) {
    // A chunk [kLinRows][kLinStride] and B chunk [kLinTileN][kLinStride]; the
    // output tile [kLinTileN][kLinOutStride] reuses the same memory
    __shared__ __align__(16) double sm[(kLinRows + kLinTileN) * kLinStride];
    __shared__ int32_t tel[kLinTileN], src[kLinTileN];
    static_assert(kLinTileN * kLinOutStride <= (kLinRows + kLinTileN) * kLinStride, "output staging fits");
    double *As = sm, *Bs = sm + kLinRows * kLinStride;
    const int R = g.R, S = g.slots;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gid = lane >> 2, tig = lane & 3;
    if (tid < kLinTileN) tel[tid] = t.elems[tile * kLinTileN + tid];
    const int passes = (R + kLinRows - 1) / kLinRows;
    for (int pass = 0; pass < passes; ++pass) {
        const int r0 = pass * kLinRows;
        const int rows = min(kLinRows, R - r0);
        double acc[8][2];
#pragma unroll
        for (int b = 0; b < 8; ++b) acc[b][0] = acc[b][1] = 0.0;
        for (int s = 0; s <= S; ++s) {
            const int32_t m = t.mats[tile * (S + 1) + s];  // the same for the whole block
            if (m < 0) continue;
            if (m >= g.n_mats) {
                if (tid == 0) atomicOr(io.status, 4);
                continue;
            }
            __syncthreads();  // tel written; src, As, Bs free
            if (tid < kLinTileN) {
                const int32_t e = tel[tid];
                int32_t se = -1;
                if (e >= 0 && e < io.n_elements) se = s == 0 ? e : g.nbr[(int64_t)e * S + (s - 1)];
                if (se >= io.n_elements || se < -1) {
                    atomicOr(io.status, 1);
                    se = -1;
                }
                src[tid] = se;
            }
            const double *A = g.table_rm + (size_t)m * R * R;
            for (int kc = 0; kc < R; kc += kLinKC) {
                // only the fragments' extent is staged: rows up to the next band of 8,
                // columns up to the next multiple of 4 (zeros beyond R)
                const int kmax = min(kLinKC, R - kc), kw = (kmax + 3) & ~3, rw = (rows + 7) & ~7;
                __syncthreads();  // src written; the previous chunk's fragments read
                // lane = column, warp = row (no integer division; a row's columns coalesce)
                if (lane < kw) {
                    for (int r = warp; r < rw; r += 8) {
                        double v = 0.0;
                        if (r < rows && lane < kmax) v = A[(size_t)(r0 + r) * R + kc + lane];
                        As[r * kLinStride + lane] = v;
                    }
#pragma unroll
                    for (int n = warp; n < kLinTileN; n += 8) {  // eight passes: loads issue together
                        const int32_t se = src[n];
                        double v = 0.0;
                        if (se >= 0 && lane < kmax) v = stage_input_few(io, (int64_t)se * R + kc + lane);
                        Bs[n * kLinStride + lane] = v;
                    }
                }
                __syncthreads();
                for (int k4 = 0; k4 < kmax; k4 += 4) {
                    const double b = Bs[(warp * 8 + gid) * kLinStride + k4 + tig];
#pragma unroll
                    for (int band = 0; band < 8; ++band)
                        if (band * 8 < rows) dmma_m8n8k4(acc[band][0], acc[band][1],
                                                         As[(band * 8 + gid) * kLinStride + k4 + tig], b);
                }
            }
        }
        __syncthreads();  // fragments read: stage the outputs as [element][row]
        double *Os = sm;
#pragma unroll
        for (int band = 0; band < 8; ++band)
            if (band * 8 < rows) {
                const int n = warp * 8 + tig * 2;
                Os[n * kLinOutStride + band * 8 + gid] = acc[band][0];
                Os[(n + 1) * kLinOutStride + band * 8 + gid] = acc[band][1];
            }
        __syncthreads();
        for (int i = tid; i < kLinTileN * kLinRows; i += blockDim.x) {
            const int n = i / kLinRows, r = i % kLinRows;
            const int32_t e = tel[n];
            if (e < 0 || e >= io.n_elements || r >= rows) continue;
            const int64_t idx = (int64_t)e * R + r0 + r;
            stage_output_few(io, idx, io.u[idx], Os[n * kLinOutStride + r]);
        }
    }
}

template <typename KT>
__global__ void __launch_bounds__(256) linear_tile_stage(const StageIOT<KT> io, const LinearGeom g,
                                                          const LinearTiles t) {
    linear_tile_body<KT>(io, g, t, blockIdx.x);
}

// ---------------------------------------------------------------------------
// pipelined form of the tiles
// ---------------------------------------------------------------------------
// The products of linear_tile_body, in the same order (so the results are the same bit
// for bit), where the stage input is one vector: the solution, or the input the previous
// stage formed (io.win).  What bounds the tiles is the FP64 tensor pipe (64 FMAs per clock
// and SM, the rate of the CUDA cores); the form above left it idle between its barriers
// and for the 64-element tiles' last wave.  Here
//   * a block of four warps takes 32 elements (half a tile): twice the blocks, and four or
//     six of them share an SM (whole tiles per block: 3092 against 2586 us per RK4 step on
//     64^3 hexahedra at p = 3);
//   * the next chunk of 32 columns (matrix rows and gathered element rows) is copied
//     asynchronously while this one's products run: one barrier per chunk, and no load's
//     latency between barriers;
//   * a warp forms 16 elements times four bands of eight rows (8 elements times four where
//     an element has at most 32 rows), so six fragment loads feed eight products.
// Measured, us per RK4 step: hexahedra at p = 3 24 x 20 x 28 290 -> 167, 64^3 2928 -> 2586
// (23.3 TFLOP/s, 0.66 of cuBLAS DGEMM 8192^3); the wave on 12^3 x 5 tetrahedra at p = 2
// 203 -> 114.
constexpr int kLinPipeN = 32;
constexpr int kLinPipeThreads = 128;
__host__ __device__ constexpr int lin_pipe_rows(bool wide) { return wide ? kLinRows : 32; }  // rows per pass
__host__ __device__ constexpr int lin_pipe_smem(bool wide) {
    return 2 * (lin_pipe_rows(wide) + kLinPipeN) * kLinStride * (int)sizeof(double);
}
__host__ __device__ constexpr int lin_pipe_blocks(bool wide) { return wide ? 4 : 6; }  // per SM
// Narrow elements take it only while all blocks run at once: triangles at p = 5, FP32 form,
// 64^2 x 2 90 -> 66 us per RK4 step, but 128^2 x 2 115 (linear_tile_stage) and 135.
inline bool lin_pipe_wanted(int R, int64_t tiles, int num_sms) { return R > 32 || 2 * tiles <= 6 * (int64_t)num_sms; }

template <int BYTES>
__device__ __forceinline__ void lin_copy(double *dst, const double *src, bool valid) {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    const int n = valid ? BYTES : 0;  // the rest is filled with zeros
    if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

// WIDE: more than 32 rows per element.  PAIRS: an even number of rows (16-byte copies).
// block: two per tile.
template <typename KT, bool WIDE, bool PAIRS>
__device__ __forceinline__ void linear_pipe_body(const StageIOT<KT> &io, const LinearGeom &g, const LinearTiles &t,
                                                 int64_t block) {
    constexpr int ROWS = lin_pipe_rows(WIDE), EL = kLinPipeN, NT = WIDE ? 2 : 1, BUF = (ROWS + EL) * kLinStride;
    constexpr int PER = PAIRS ? 2 : 1, PARTS = kLinKC / PER;  // doubles per copy, copies per row
    constexpr int STEP = kLinPipeThreads / PARTS;             // rows copied at once
    extern __shared__ __align__(16) double lin_pipe_shared[];
    const int R = g.R, S = g.slots;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gid = lane >> 2, tig = lane & 3;
    const int n0 = WIDE ? (warp & 1) * (EL / 2) : warp * 8, b0 = WIDE ? (warp >> 1) * 4 : 0;  // the warp's elements, bands
    const int64_t tile = block >> 1;
    const int32_t *tel = t.elems + tile * kLinTileN + (block & 1) * EL;
    const int32_t *mats = t.mats + tile * (S + 1);
    const double *w = io.win ? io.win : io.u;
    const int crow = tid / PARTS, ccol = (tid % PARTS) * PER;  // this thread's copies: rows crow + STEP i, column ccol
    auto element = [&](int n) {  // of the block, -1: padding
        const int32_t e = __ldg(tel + n);
        return e >= 0 && e < io.n_elements ? e : -1;
    };
    int32_t el[EL / STEP];  // the elements whose rows this thread copies
    bool any = false;
#pragma unroll
    for (int i = 0; i < EL / STEP; ++i) {
        el[i] = element(crow + STEP * i);
        any = any || el[i] >= 0;
    }
    if (!__syncthreads_or(any)) return;  // (a group's last tile: its second half may be empty)
    // next slot with a matrix after s; S + 1 when there is none
    auto next_slot = [&](int s) {
        for (++s; s <= S; ++s) {
            const int32_t m = __ldg(mats + s);
            if (m >= g.n_mats && tid == 0) atomicOr(io.status, 4);
            if (m >= 0 && m < g.n_mats) break;
        }
        return s;
    };
    int32_t src[EL / STEP];  // of the slot being copied
    auto sources = [&](int s) {
#pragma unroll
        for (int i = 0; i < EL / STEP; ++i) {
            int32_t se = el[i];
            if (s > 0 && se >= 0) se = __ldg(g.nbr + (int64_t)se * S + (s - 1));
            if (se >= io.n_elements || se < -1) {
                atomicOr(io.status, 1);
                se = -1;
            }
            src[i] = se;
        }
    };
    for (int r0 = 0; r0 < R; r0 += ROWS) {
        const int rows = min(ROWS, R - r0), rw = (rows + 7) & ~7;
        auto copy = [&](int s, int kc, double *buf) {
            const double *A = g.table_rm + (size_t)__ldg(mats + s) * R * R;
            const bool in = kc + ccol < R;
#pragma unroll
            for (int i = 0; i < ROWS / STEP; ++i) {
                const int r = crow + STEP * i;
                if (r < rw) {
                    const bool ok = in && r < rows;
                    lin_copy<8 * PER>(buf + r * kLinStride + ccol, ok ? A + (size_t)(r0 + r) * R + kc + ccol : A, ok);
                }
            }
#pragma unroll
            for (int i = 0; i < EL / STEP; ++i) {
                const bool ok = in && src[i] >= 0;
                lin_copy<8 * PER>(buf + (ROWS + crow + STEP * i) * kLinStride + ccol,
                                  ok ? w + (int64_t)src[i] * R + kc + ccol : w, ok);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        double acc[NT][4][2];
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int b = 0; b < 4; ++b) acc[n][b][0] = acc[n][b][1] = 0.0;
        int s = next_slot(-1), kc = 0, at = 0;
        if (s <= S) {
            sources(s);
            copy(s, 0, lin_pipe_shared);
        }
        while (s <= S) {
            const double *As = lin_pipe_shared + at * BUF, *Bs = As + ROWS * kLinStride;
            const int kmax = min(kLinKC, R - kc);
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();  // this chunk is here, and the other buffer's products are done
            at ^= 1;
            kc += kLinKC;
            if (kc >= R) {
                kc = 0;
                s = next_slot(s);
                if (s <= S) sources(s);
            }
            if (s <= S) copy(s, kc, lin_pipe_shared + at * BUF);
#pragma unroll 2
            for (int k4 = 0; k4 < kmax; k4 += 4) {
                double b[NT];
#pragma unroll
                for (int n = 0; n < NT; ++n) b[n] = Bs[(n0 + 8 * n + gid) * kLinStride + k4 + tig];
#pragma unroll
                for (int band = 0; band < 4; ++band) {
                    if ((b0 + band) * 8 >= rows) continue;
                    const double a = As[((b0 + band) * 8 + gid) * kLinStride + k4 + tig];
#pragma unroll
                    for (int n = 0; n < NT; ++n) dmma_m8n8k4(acc[n][band][0], acc[n][band][1], a, b[n]);
                }
            }
        }
        __syncthreads();  // all products: stage the outputs as [element][row]
        constexpr int OS = ROWS + 1;
        double *Os = lin_pipe_shared;
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int band = 0; band < 4; ++band)
                if ((b0 + band) * 8 < rows) {
                    const int e = n0 + 8 * n + tig * 2, r = (b0 + band) * 8 + gid;
                    Os[e * OS + r] = acc[n][band][0];
                    Os[(e + 1) * OS + r] = acc[n][band][1];
                }
        __syncthreads();
#pragma unroll 4
        for (int i = tid; i < EL * ROWS; i += kLinPipeThreads) {
            const int n = i / ROWS, r = i % ROWS;
            const int32_t e = element(n);
            if (e < 0 || r >= rows) continue;
            const int64_t idx = (int64_t)e * R + r0 + r;
            stage_output_few(io, idx, io.u[idx], Os[n * OS + r]);
        }
        __syncthreads();  // the outputs are read (the next pass copies over them)
    }
}

template <typename KT, bool WIDE, bool PAIRS>
__global__ void __launch_bounds__(kLinPipeThreads, lin_pipe_blocks(WIDE))
    linear_pipe_stage(const StageIOT<KT> io, const LinearGeom g, const LinearTiles t) {
    linear_pipe_body<KT, WIDE, PAIRS>(io, g, t, blockIdx.x);
}

// calls f(WIDE, PAIRS) for elements of R rows and a stage input at `w` (a caller's vector
// may start at any double: 16-byte copies only where it starts at 16 bytes)
template <typename F>
void lin_pipe_dispatch(int R, const double *w, F &&f) {
    const bool pairs = R % 2 == 0 && reinterpret_cast<uintptr_t>(w) % 16 == 0;
    auto with = [&](auto wide) {
        if (pairs) f(wide, std::true_type{});
        else f(wide, std::false_type{});
    };
    if (R > 32) with(std::true_type{});
    else with(std::false_type{});
}

}  // namespace hgg
