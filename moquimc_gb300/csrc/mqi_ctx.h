// Host-side state of a context (struct mqi_ctx of the C ABI) and the helpers every entry-point
// file uses.
//
// The reference keeps its device state in globals (mc::mc_world, mc_materials, mc_vertices,
// moqui/kernel_functions/mqi_variables.hpp:8-17) built by <<<1,1>>> kernels that call device-side
// `new` (mqi_upload_data.hpp:69-142).  Here a context owns flat device buffers, and every kernel
// receives what it reads by value.
#pragma once

#include <algorithm>
#include <array>
#include <cstdint>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "mqi_gpu.h"
#include "mqi_internal.h"

namespace mqi_gpu
{

/// A child's material table at one density scale.
struct Material {
    float   scale = 1.0f;
    float4* mat = nullptr;
};

struct ChildHost {
    int    nx = 0, ny = 0, nz = 0;
    float* xe = nullptr;
    float* ye = nullptr;
    float* ze = nullptr;
    float* rho = nullptr;
    bool   has_rho = false;
    std::vector<Material> mats;   // built by the first transport after the density or the curves changed
    float  rf[9], ri[9], tr[3];
    int    identity = 1;
};

/// A Dij scorer's built matrix: spot rows (the transposed operator, the reference's npz layout)
/// and voxel rows (only voxels with an entry).
struct DijCsr {
    bool      built = false;
    void*     slab = nullptr;       // one allocation that holds all arrays; kept for the next build (dij_reset)
    size_t    slab_bytes = 0;
    uint32_t  n_spots = 0;
    uint64_t  n_voxels = 0;
    uint64_t  nnz = 0;
    uint64_t  n_vrows = 0;
    uint64_t* s_indptr = nullptr;   // n_spots + 1
    uint32_t* s_voxel = nullptr;    // nnz
    float*    s_value = nullptr;    // nnz
    uint32_t* v_row = nullptr;      // n_vrows: voxel of each voxel row
    uint16_t* v_off = nullptr;      // n_vrows: the row's first entry, modulo kFwdEntries
    void*     v_spot = nullptr;     // nnz: uint16_t with spot16, else uint32_t
    bool      spot16 = false;       // n_spots <= 65536
    float*    v_value = nullptr;    // nnz
    uint64_t  n_seg = 0;            // backward segments: contiguous runs of one row's entries
    uint64_t* seg_start = nullptr;  // n_seg + 1
    uint32_t* row_seg = nullptr;    // n_spots + 1: first segment of each row
    uint32_t* seg_order = nullptr;  // n_seg: segments by first voxel (the backward's work order)
    uint32_t* bwd_cursor = nullptr; // the backward's work cursor (zero between calls)
    double*   partial = nullptr;    // n_seg
    uint64_t  n_fwd_blocks = 0;     // forward blocks: kFwdEntries entries' worth of voxel rows each
    uint32_t* fwd_row_first = nullptr;   // n_fwd_blocks + 1: first voxel row of each forward block
    uint64_t* fwd_run_k = nullptr;       // n_fwd_blocks + 1: first entry of each forward block's rows
};

// The largest build scratch that a context keeps, and the largest memory of a matrix that a reset leaves to
// the next build: allocating takes a small part of the time of a larger build.
constexpr size_t kKeepScratch = (size_t) 512 << 20;

struct ScorerHost {
    int       child = 0;
    int       type = 0;
    int       roi_method = 0;
    int       stat_mode = 0;
    uint32_t  roi_len = 0;
    uint32_t* start = nullptr;
    uint32_t* stride = nullptr;
    uint32_t* acc = nullptr;
    uint2*    roi_words = nullptr; // a CONTOUR ROI by voxel (ScorerDev::roi_words)
    double*   tally = nullptr;
    uint64_t  tally_len = 0;       // per scenario; the tally holds copies * tally_len values
    uint32_t  copies = 1;          // robust scenarios: one tally per scenario, scenario-major
    uint32_t  tstride = 1;         // doubles between consecutive values (2: the interleaved stat pair)
    int       partner = -1;        // the stat pair's other scorer (shares the buffer)
    bool      owns = true;         // this scorer allocated `tally` (the dose half of the stat pair does)
    double*   batch_s1 = nullptr;   // batch estimator: running sums of batch tallies and squares
    double*   batch_s2 = nullptr;
    uint64_t  n_batches = 0;
    DijSlot*  dij = nullptr;        // MQI_SCORER_DIJ: hash table of dij_cap slots (power of two)
    uint64_t  dij_cap = 0;
    unsigned long long* dij_count = nullptr;   // device: occupied slots, counted on demand (dij_count())
    DijHit*   hit_log = nullptr;    // mqi_dij_record_hits: recorded insertions
    unsigned long long* hit_count = nullptr;
    uint64_t  hit_cap = 0;
    DijCsr    csr;

    uint64_t total() const { return tally_len * copies; }   // values (not doubles: see tstride)
};

struct QueueBuf {
    Queue    q{};
    void*    base = nullptr;
};

/// The calling thread's last error message.
std::string& thread_error_slot();

/// Free a Dij scorer's table and matrix (mqi_capi_dij.cu).
void dij_release(ScorerHost& s);
/// Free a Dij scorer's matrix.
void dij_drop_matrix(ScorerHost& s);
/// Empty a Dij scorer's table; its matrix is no longer built.
cudaError_t dij_reset(ScorerHost& s, int sms, cudaStream_t st);

/// The shape of a draining wave over n queue entries.  While every track has a lane of its own, the
/// wave lasts as long as a chain of steps takes, and 12 warps per SM (168 registers, hardly a spill) take
/// them sooner than 16 with 128 registers (5000 histories on the slab phantom 1.40 -> 1.19 ms, 50 000 in
/// water 4.55 -> 4.03, twelve CT spots of 2500, one call each, 15.8 -> 13.8); beyond that throughput
/// counts, and 20 warps do (with 12, 100 000 in water 5.2 -> 6.7).  Few tracks are spread over the
/// resident warps, and no more blocks are launched than hold a lane for each, the warps that only run
/// post-steps (kPostEvery) and a few to spare: those without a track poll, and fetch other code than
/// their neighbours (with twice the warps 600 tracks took 0.637 instead of 0.615 ms, twelve CT spots 13.7
/// instead of 12.9, 30 000 histories in water 3.9 instead of 3.7).
inline void
plan_drain(WaveParams& P, uint32_t n, int sms) {
    P.drain_warps        = n <= (uint32_t) (sms * 12 * 32) ? 12 : 20;
    const uint32_t warps = (uint32_t) (sms * P.drain_warps) / kPostEvery * (kPostEvery - 1);
    P.lanes              = (int) std::min<uint32_t>((n + warps - 1) / warps, 32u);
    const uint32_t need  = (n + P.lanes - 1) / P.lanes;
    P.max_blocks         = std::max<int>(sms, (int) ((need + need / 64 + 7) / 4));
}

struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        cudaGetDevice(&prev);
        if (prev != dev) cudaSetDevice(dev);
    }
    ~DeviceGuard() {
        int cur = -1;
        cudaGetDevice(&cur);
        if (prev >= 0 && cur != prev) cudaSetDevice(prev);
    }
};

}   // namespace mqi_gpu

struct mqi_ctx {
    int                     device = 0;
    cudaStream_t            stream = nullptr;
    bool                    own_stream = false;
    std::string             err;
    int                     physics_debug = 0;
    int                     score_local = 1;
    std::vector<mqi_gpu::ChildHost>  children;
    std::vector<mqi_gpu::ScorerHost> scorers;
    mqi_vertex*             vertices = nullptr;
    uint64_t                n_vertices = 0;
    uint64_t                vertex_cap = 0;
    uint32_t*               spot_ids = nullptr;
    uint64_t                spot_cap = 0;
    bool                    has_spots = false;
    mqi_gpu::QueueBuf       qa, qb;
    uint32_t                queue_cap = 0;
    mqi_gpu::Deferred*      def = nullptr;          // tracks a wave stopped at nuclear interactions
    uint32_t                def_cap = 0;
    mqi_gpu::QueueBuf       qsort;                  // scratch of the energy-bin queue sort (queue_cap, on first use)
    uint32_t*               sort_bins = nullptr;    // 2 x kSortBins counters of the sort
    uint32_t                sort_min = 1u << 18;    // sort waves of at least this many entries (0: never)
    uint32_t*               ready = nullptr;        // marks of the entries a draining wave appended (queue_cap)
    uint32_t                epoch = 0;              // the last draining wave's number
    uint32_t*               counters = nullptr;     // 12 words: [0] entries of the queue read, [1] of the next,
                                                    // [2] head, [3] error flag, [8 ..] DrainState
    unsigned long long*     stats = nullptr;        // 8 x u64
    uint32_t*               host_counts = nullptr;  // pinned: 12 x u32
    float*                  tables = nullptr;       // 6*600 physics + 3996 HU densities
    mqi_gpu::CalibDev       calib{};                // SPR / X0 curves (mode 0: the defaults)
    float*                  calib_buf = nullptr;    // device: the tables of calib (SPR then X0)
    int                     num_sms = 0;
    int                     wave_block = 128;         // threads per block and blocks per SM asked for
    int                     wave_bps = 5;             // (launch_wave runs their product, as one block)
    uint32_t                max_slice_steps = 0;
    uint32_t                primary_chunk = 1u << 21;
    uint64_t                waves = 0;
    uint64_t                loaded = 0;               // primaries put into the queue, once per scenario
    uint64_t                kernel_launches = 0;
    uint64_t                wave_launches = 0;
    double                  wave_ms = 0.0;
    cudaEvent_t             ev0 = nullptr, ev1 = nullptr;
    uint64_t                give_backs = 0;           // times that give_back freed something
    void*                   build_scratch = nullptr;  // the last Dij build's sort buffers, when at most kKeepScratch
    size_t                  build_scratch_bytes = 0;
    unsigned long long*     stat_scratch = nullptr;   // 3 x u64 for the statistics reductions
    mqi_spot*               plan_spots = nullptr;     // spot plan (device)
    uint64_t*               plan_cum = nullptr;       // cumulative histories, n_plan_spots + 1 (device)
    uint32_t                n_plan_spots = 0;
    uint64_t                plan_histories = 0;
    std::vector<uint64_t>   plan_cum_host;
    int                     streamed = 1;             // 1: the queue is topped up before every wave; 0: generations
    int                     post_step_mode = -1;      // nuclear post-steps: -1 automatic, 0 in draining waves, 1 post-step kernel
    int                     graph_waves = 8;          // kept for the tuner's records
    uint32_t                n_scen = 1;               // robust scenarios (1: none)
    int                     scen_child = -1;
    float*                  scen_edges = nullptr;     // device: the scenarios' different edge arrays
    int                     scen_floats = 0;
    std::vector<std::array<uint32_t, 3>> scen_off;    // each scenario's x, y and z arrays in it
    std::vector<float>      scen_scale;
};

namespace mqi_gpu
{

inline int
fail(mqi_ctx* c, int code, const std::string& msg) {
    if (c) c->err = msg;
    thread_error_slot() = msg;
    return code;
}

/// Report a failed CUDA call.  The runtime keeps a non-sticky error as its "last error" until it
/// is read; it is read here, so that the next launch's cudaGetLastError reports that launch.
inline int
cuda_fail(mqi_ctx* c, cudaError_t e, const char* what) {
    (void) cudaGetLastError();
    return fail(c, e == cudaErrorMemoryAllocation ? MQI_ERR_NOMEM : MQI_ERR_CUDA,
                std::string(what) + ": " + cudaGetErrorString(e));
}

inline bool
valid_ctx(const mqi_ctx* c) {
    return c != nullptr;
}

/// Free what the context can do without: the material tables, the kept sort buffers of a Dij build and the
/// memory of matrices that are no longer built.  False when there was nothing.  Not while a wave runs.
bool give_back(mqi_ctx* c);

/// Device memory that a call cannot do without: before it fails for want of memory, the context gives
/// back what it can.
template<typename T>
cudaError_t
device_alloc(mqi_ctx* c, T*& p, size_t bytes) {
    p             = nullptr;
    cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&p), bytes);
    if (e == cudaErrorMemoryAllocation && give_back(c)) {
        (void) cudaGetLastError();
        e = cudaMalloc(reinterpret_cast<void**>(&p), bytes);
    }
    if (e != cudaSuccess) p = nullptr;
    return e;
}

/// Host data to device memory, and zeroes there, in the order of the context's stream and done on return.
/// (cudaMemcpy and cudaMemset run on the legacy stream, which a non-blocking stream does not wait
/// for, and may return before the device has the data.)
inline cudaError_t
upload(mqi_ctx* c, void* dst, const void* src, size_t bytes) {
    const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, c->stream);
    return e == cudaSuccess ? cudaStreamSynchronize(c->stream) : e;
}

inline cudaError_t
zero_out(mqi_ctx* c, void* dst, size_t bytes) {
    const cudaError_t e = cudaMemsetAsync(dst, 0, bytes, c->stream);
    return e == cudaSuccess ? cudaStreamSynchronize(c->stream) : e;
}

}   // namespace mqi_gpu

#define MQI_CUDA(c, expr, what)                                        \
    do {                                                               \
        cudaError_t _e = (expr);                                       \
        if (_e != cudaSuccess) return mqi_gpu::cuda_fail(c, _e, what); \
    } while (0)
