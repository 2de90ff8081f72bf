// The device problem behind an hgg_handle, shared by the translation units of
// the library: the entry points (capi.cu), the stage launchers
// (stage_tensor.cu, stage_dense.cu) and the batch and serving loop (batch.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <memory>
#include <string>
#include <utility>
#include <vector>

#include "../../include/hpgem_b200.h"
#include "dg_kernels.cuh"
#include "lane_stage.cuh"
#include "linear_stage.cuh"
#include "linear_umma.cuh"
#include "tensor_lane.cuh"
#include "tensor_pipe.cuh"
#include "tensor_slice.cuh"
#include "host/linear.h"
#include "host/operators.h"
#include "host/setup.h"

namespace hgg {
struct SourceState;  // sources.cu
struct DevBuf {
    void *p = nullptr;
    size_t bytes = 0;
};
}  // namespace hgg

struct hgg_handle {
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaStream_t own_stream = nullptr;
    hgg::HostOperators op;
    std::unique_ptr<hgg::StructuredProblem> sp;  // set when built from a structured description
    int S = 0;
    std::vector<double> rk_a, rk_b, rk_c;
    std::vector<double> rk_err;   // error coefficients of an embedded tableau (empty: none)
    int rk_order = 0;
    int64_t N = 0;                 // doubles per vector
    int64_t N_alloc = 0;           // doubles allocated per vector (whole tiles)
    double *sol[2] = {nullptr, nullptr};
    int cur = 0;                   // which sol[] holds the solution
    std::vector<void *> k;         // S stage vectors (double, or float in the FP32-mixed form)
    bool mixed = false;            // FP32-mixed form: float stage vectors and contractions
    std::vector<hgg::DevBuf> bufs;      // every device allocation
    // device operator / geometry arrays
    double *d_vol = nullptr, *d_pairs = nullptr, *d_elem_geo = nullptr, *d_face_geo = nullptr;
    float *d_vol_f = nullptr, *d_pairs_f = nullptr;  // FP32-mixed form: the dense operators in FP32
    int32_t *d_nbr = nullptr, *d_self = nullptr, *d_nbrp = nullptr;
    int8_t *d_mode = nullptr;
    double *d_ahat = nullptr, *d_tsigma = nullptr;
    int32_t *d_tnbr = nullptr;
    int8_t *d_tmode = nullptr;
    unsigned char *d_pgeo = nullptr;  // packed per-element geometry of the pipelined kernel
    int tile_elems = 1;               // elements per tile (common multiple of the tensor kernels' tiles)
    int variant = 0;                  // 0: automatic, 1: one-shot, 2: pipelined kernel
    bool tensor_layout = false;       // device vectors in tensor order (signs folded)
    bool tiled = false;               // ... and in tiles of 32 elements, coefficient-major (slice kernel)
    double *d_scratch = nullptr;      // one vector, for layout conversion of set/get_state
    double *d_reduce = nullptr;       // adaptive steps and error norms: per-element values, partial sums
    double *d_exact = nullptr;        // error norms: the caller's exact values on the device
    size_t exact_cap = 0;
    double *d_maxbuf = nullptr;
    double *d_err_basis = nullptr, *d_err_w = nullptr, *d_elem_basis = nullptr, *d_absdet = nullptr;
    int32_t *d_tpos = nullptr;        // hpGEM index -> tensor position
    double *d_tsign = nullptr;
    // slice kernel (hexahedra, p = 3): per-element records of SliceShape::GR doubles
    bool slice_ok = false;
    double *d_slice_geo = nullptr;
    // one-element-per-thread kernels (lane = element, tiled layout): the handle has one, and
    // its vectors are in that kernel's layout (kernel variant 0)
    bool lane_ok = false, lane = false;
    // batches that have the handle as a member: their tables hold its vectors' layout, so a
    // change of the variant moves them when the last has let go (shared with the batch,
    // which may outlive the handle)
    std::shared_ptr<int> memberships;  // (null: never in one)
    bool overlap = true;                  // chained launches start early (hgg_test_set_overlap)
    hgg::TensorLaneGeom tlane{};          // sum-factorised handles
    hgg::LaneGeom lgeo{};                  // simplices and the wave
    double *d_lane_win[2] = {nullptr, nullptr};  // ... the wave: stage inputs formed ahead (contraction type)
    int lane_tiles = 1;                    // ... tiles of a chunk at most
    // ... mostly padding: faster than the general kernels only while all tiles run at once
    // (see hgg_batch_add)
    bool lane_sparse = false;
    std::vector<int32_t> slot;            // place of each element in the lane layout (empty: its own number)
    int32_t *d_slot = nullptr;            // slot on the device while the lane layout is in use, else null
    int32_t *d_slot_lane = nullptr;
    // stored-matrix form (HpgemAPILinear): distinct folded matrices, transposed
    bool linear = false;
    int lin_R = 0, lin_slots = 0, lin_mats = 0;
    double *d_lin_table = nullptr;
    float *d_lin_table_f = nullptr;  // FP32-mixed form with FP32 contractions (R <= kMixedFp32MaxBasis)
    int32_t *d_lin_self = nullptr, *d_lin_nbr = nullptr, *d_lin_mat = nullptr;
    // grouped DMMA kernel: tiles of elements with identical matrices (0 tiles: not used)
    double *d_lin_table_rm = nullptr;
    int32_t *d_lin_tile_elems = nullptr, *d_lin_tile_mats = nullptr;
    int64_t lin_tiles = 0;
    double *d_lin_win[2] = {nullptr, nullptr};  // stage inputs formed ahead (tiles, see lin_forms_input)
    int lin_min_rows = hgg::kLinTileMinRows;  // fewer rows per element: the row kernel
    // mixed forms on the tensor cores (tcgen05): tiles of 128 elements with identical
    // matrices, matrix operand images split into hi / lo parts
    int precision = 0;                     // enum hgg_precision
    int64_t umma_tiles = 0;                // 0: not used
    int32_t *d_umma_tile_elems = nullptr, *d_umma_tile_mats = nullptr;
    unsigned char *d_umma_img = nullptr;
    unsigned char *d_umma_planes = nullptr;  // split stage input, two planes [E][KP]
    // grouped dense kernel: tiles of group_tile_elems(nB) elements with the same operator signature
    int32_t *d_group_tiles = nullptr;
    double *d_win[2] = {nullptr, nullptr};  // stage inputs formed ahead (grouped wave kernel)
    int64_t group_tiles = 0;
    int num_sms = 148;
    int *d_status = nullptr;
    uint32_t test_arm_polls = 0;  // hgg_test_arm_without_copy: poll limit of the next pipelined launch
    // HpgemAPILinear source terms (sources.cu)
    bool linear_api = false;            // HpgemAPILinear built from a structured mesh or a mesh file
    std::vector<double> lin_mass;       // its distinct element mass matrices [n][R][R]
    std::vector<int32_t> lin_mass_of;   // [E]
    hgg::SourceState *src = nullptr;    // set: every stage adds the caller's source terms
    bool store_last = true;
    int64_t launches = 0;
    int64_t graph_launches = 0;  // kernels in one captured step
    // graphs of one step and of kRunSteps steps, per starting buffer, valid for (dt,
    // store_last); made when first needed
    static constexpr int kRunSteps = 8;
    cudaGraphExec_t graph[2] = {nullptr, nullptr}, graph_run[2] = {nullptr, nullptr};
    double graph_dt = 0.0;
    bool graph_store_last = true;
    std::string err = "no error";
};

namespace hgg {

// records msg as the handle's last error (or the last create error) and returns code
int fail(hgg_handle *h, int code, const std::string &msg);

#define HGG_CUDA(h, call)                                                                    \
    do {                                                                                     \
        cudaError_t _e = (call);                                                             \
        if (_e != cudaSuccess)                                                               \
            return fail(h, HGG_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(_e)); \
    } while (0)

// Device memory of a handle is stream-ordered (cudaMallocAsync / cudaFreeAsync on the
// handle's stream, from the device's default pool): freeing a handle never waits for
// work of other streams, so a solve that finishes inside a batch or a server is freed
// while the other members keep stepping.

int alloc(hgg_handle *h, size_t bytes, void **dst);
// device copy of a host vector, owned by the handle
template <typename T>
int upload(hgg_handle *h, const std::vector<T> &v, T **dst) {
    *dst = nullptr;
    if (v.empty()) return 0;
    const size_t bytes = v.size() * sizeof(T);
    void *p = nullptr;
    if (int rc = alloc(h, bytes, &p)) return rc;
    cudaError_t e = cudaMemcpyAsync(p, v.data(), bytes, cudaMemcpyHostToDevice, h->stream);
    if (e != cudaSuccess) return fail(h, HGG_ERR_CUDA, std::string("cudaMemcpyAsync: ") + cudaGetErrorString(e));
    *dst = (T *)p;
    return 0;
}

// coefficients per element (all variables)
inline int coefficients(const hgg_handle *h) { return h->op.V * h->op.nB; }
// the wave runs the grouped tile kernel (alone and in a batch): kernel variant 2, or
// the automatic choice where it measured faster than the per-row kernel
bool group_wave_wanted(const hgg_handle *h);
void release_graphs(hgg_handle *h);
// the vectors into the layout of the kernel variant, or (general) of the general kernels,
// unless a batch steps them
int settle_layout(hgg_handle *h, bool general = false);
// the current solution in hpGEM order with no kernel on the device: one copy of the
// device vector into `staging` (pinned, h->N_alloc doubles), the layout change on the host
int solution_to_host(hgg_handle *h, double *staging, double *out);

// Launch of a stage kernel that calls chain_next and chain_wait: with `overlap` its start
// overlaps the previous kernel's end on the same stream (anything else before it is waited
// for in full), which takes part of the gap between two stages out.  Per RK4 step in graphs
// of eight steps: 32^2 quadrilaterals at p = 2 10.3 -> 9.5 us, triangles 192 x 160 at p = 3
// 20.4 -> 17.9, the FP32 wave on 14 x 18 x 12 x 5 tetrahedra at p = 3 130 -> 127.  (Letting
// the next stage start at a lane kernel's beginning instead of before its outputs spreads
// its blocks unevenly over the SMs: the triangles took 23.7.)
template <typename... K, typename... A>
void launch_chained(bool overlap, void (*kern)(K...), unsigned grid, unsigned threads, size_t smem, cudaStream_t s,
                    A &&...args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = overlap;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);  // (the caller checks cudaGetLastError)
}

template <int P, int DIM>
TensorConsts<P, DIM> tensor_consts(const HostOperators &op) {
    using TC = TensorConsts<P, DIM>;
    TC tc;
    for (int i = 0; i < TC::NP * TC::NP; ++i) tc.D1[i] = op.D1[i];
    for (int i = 0; i < 2 * TC::NP; ++i) tc.lift[i] = op.lift[i];
    tc.trace_pos[0] = op.trace_pos[0];
    tc.trace_pos[1] = op.trace_pos[1];
    for (int i = 0; i < TC::NB; ++i) {
        tc.tpos[i] = (short)i;
        tc.tinv[i] = (short)i;
        tc.tsign[i] = 1.0;
    }
    return tc;
}

// layout conversion index (hpGEM order <-> tensor order, signs folded; tiled:
// 32-element tiles, coefficient-major inside a tile)
// slot: the place of each element in the tiles, or null for its own number
__host__ __device__ __forceinline__ int64_t device_index(int64_t e, int pos, int nb, bool tiled,
                                                         const int32_t *slot = nullptr) {
    if (slot) e = slot[e];
    return tiled ? (e >> 5) * ((int64_t)nb << 5) + (int64_t)pos * 32 + (e & 31) : e * nb + pos;
}
// stage vectors and per-stage coefficients of the error estimate and the rewind
template <typename KT>
struct ErrStages {
    const KT *k[kMaxStages];
    double err[kMaxStages];
    double dt;
    int n;
};

// elements per tile of the pipelined kernel for (order, dim); bytes of its packed geometry
int pipe_tile_elems(int order, int dim);
int pipe_geo_bytes(int dim);
// wave speed factor of the upwind wave flux, 0 for the central flux
double upwind_speed(const HostOperators &op);

// one stage launch of the handle's kernel (stage_tensor.cu: slice and
// sum-factorised kernels; stage_dense.cu: dense and stored-matrix kernels)
int launch_stage_tensor(hgg_handle *h, const StageIOT<double> &io);
int launch_stage_tensor(hgg_handle *h, const StageIOT<float> &io);
int launch_stage_dense(hgg_handle *h, const StageIOT<double> &io);
int launch_stage_dense(hgg_handle *h, const StageIOT<float> &io);
int launch_stage_lane(hgg_handle *h, const StageIOT<double> &io);
int launch_stage_lane(hgg_handle *h, const StageIOT<float> &io);
int launch_stage_linear(hgg_handle *h, const StageIOT<double> &io);
int launch_stage_linear(hgg_handle *h, const StageIOT<float> &io);
// the handle's stage kernel, counted, with the launch error checked
int launch_stage(hgg_handle *h, const StageIO &io);
int launch_stage(hgg_handle *h, const StageIOT<float> &io);

void *vector_ptr(hgg_handle *h, int vec);
bool vector_is_float(const hgg_handle *h, int vec);

// the wave's lane kernel reads one vector: every stage but the last forms the next one's input
inline bool lane_forms_input(const hgg_handle *h) {
    return h->lane && !h->op.tensor && h->op.physics != HGG_PHYSICS_ADVECTION;
}

// every stage input has exactly one earlier vector, the previous one (explicit RK4, midpoint)
inline bool chain_tableau(const hgg_handle *h) {
    const int S = h->S;
    for (int i = 1; i < S; ++i)
        for (int j = 0; j < i; ++j)
            if ((h->rk_a[i * S + j] != 0.0) != (j == i - 1)) return false;
    return true;
}
// the stored-matrix tiles: each stage then forms the next one's input, one vector, which
// the pipelined kernel can copy (a source term is added after the stage: not with one; a
// batch steps its members without their sources, and with its class's kernel)
inline bool lin_forms_input(const hgg_handle *h, bool in_batch) {
    return h->d_lin_win[0] && !h->lane && chain_tableau(h) &&
           (in_batch || (!h->src && lin_pipe_wanted(h->lin_R, h->lin_tiles, h->num_sms)));
}

// Inputs and outputs of stage i of one Runge-Kutta step from sol[from] into
// sol[1 - from] (stages as in HpgemAPISimplified_Impl.h:788-820; zero tableau
// entries are skipped).
template <typename KT>
StageIOT<KT> make_stage_io(const hgg_handle *h, int from, double dt, int i, int *status, bool in_batch = false) {
    const int S = h->S;
    auto kv = [&](int j) { return static_cast<KT *>(h->k[j]); };
    StageIOT<KT> io{};
    io.u = h->sol[from];
    io.n_elements = h->op.nE;
    io.status = status;
    for (int j = 0; j < i; ++j) {
        double c = dt * h->rk_a[i * S + j];
        if (c != 0.0) {
            io.kin[io.nin] = kv(j);
            io.cin[io.nin] = c;
            io.nin++;
        }
    }
    const bool last = i == S - 1;
    io.kout = (!last || h->store_last) ? kv(i) : nullptr;
    if (last) {
        io.unew = h->sol[1 - from];
        for (int j = 0; j < S - 1; ++j) {
            double b = dt * h->rk_b[j];
            if (b != 0.0) {
                io.kfin[io.nfin] = kv(j);
                io.bfin[io.nfin] = b;
                io.nfin++;
            }
        }
        io.blast = dt * h->rk_b[S - 1];
    }
    if (lin_forms_input(h, in_batch)) {
        if (i > 0) io.win = h->d_lin_win[(i - 1) & 1];
        if (!last) {
            io.wnext = h->d_lin_win[i & 1];
            io.wcoef = dt * h->rk_a[(i + 1) * S + i];
        }
    }
    if (lane_forms_input(h)) {
        if (i > 0) io.win = h->d_lane_win[(i - 1) & 1];
        if (!last) {
            io.wnext = h->d_lane_win[i & 1];
            for (int j = 0; j < i; ++j) {
                const double c = dt * h->rk_a[(i + 1) * S + j];
                if (c != 0.0) {
                    io.kfin[io.nfin] = kv(j);
                    io.bfin[io.nfin] = c;
                    io.nfin++;
                }
            }
            io.wcoef = dt * h->rk_a[(i + 1) * S + i];
        }
    }
    return io;
}

// source terms (sources.cu): the caller's functions evaluated at the stage times
// t + c_i dt of one step (buf 0 / 1: the step from sol[0] / sol[1]) or at
// `times` (buf 2) and copied to the device; the lift of stage `stage` added to
// kout (and blast times it to unew) after the stage kernel
int fill_sources(hgg_handle *h, int buf, double t, double dt);
int fill_source_values(hgg_handle *h, int buf, const double *times, int n);
int enqueue_source(hgg_handle *h, int buf, int stage, double *kout, double *unew, double blast);
int enqueue_source(hgg_handle *h, int buf, int stage, float *kout, double *unew, double blast);
void destroy_sources(hgg_handle *h);
// hgg_time_derivative (time null) and hgg_time_derivative_at
int time_derivative_impl(hgg_handle *h, int32_t in_vec, int32_t out_vec, const double *time);

// the failures a device status word records (bit 0: bad neighbour index, bit 1:
// a bounded wait ran out, bit 2: bad matrix index)
std::string status_message(int st);
// reads the device status word (synchronises the handle's stream)
int check_status(hgg_handle *h);

}  // namespace hgg
