// nf_internal.h -- host-side internals shared by the library's translation units.
#pragma once
#include <cuda_runtime.h>

#include <array>
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <deque>
#include <list>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <unordered_map>
#include <vector>

#include "nf_capi.h"

namespace nf {

// thread-local error text behind nf_last_error()
void set_error(const std::string &msg);
nf_status cuda_fail(cudaError_t e, const char *what);

#define NF_CUDA(call)                                          \
    do {                                                       \
        cudaError_t _e = (call);                               \
        if (_e != cudaSuccess) return nf::cuda_fail(_e, #call); \
    } while (0)

// A pencil partial of one sink and component: a compensated FP32 sum kept as
// (hi, lo), value hi + lo.  The co-add sums the 2R+1 partials of a sink with
// compensated FP32 arithmetic too, so no FP64 enters the accumulation.
typedef float2 Partial;

// One warp work item of the pencil kernel (32 bytes).
struct Item {
    int32_t pencil;      // linear id of the pencil's centre cell (x, y, zc)
    int32_t sink_begin;  // first sink of the tile in the pencil's sink stream
    int32_t nsink;       // sinks in the tile (1 .. 32*S)
    int32_t S;           // sinks per lane: 1, 2 or 4
    int32_t src_begin;   // source stream range [src_begin, src_end)
    int32_t src_end;
    int32_t pad0, pad1;
};

// One warp work item of the mutual sweep (nf_mutual.cu): chunks [c0, c1) of
// the tile's stream of sources.
struct MutualItem {
    int32_t pencil;             // linear id of the pencil's centre cell
    int32_t sink_begin, nsink;  // the tile, in the pencil's sink stream
    int32_t S;                  // sinks per lane
    int32_t c0, c1;
    int32_t pad0, pad1;
};

struct Plan {
    int lo = 0, hi = 0;
    int variant = 0;  // kernel shape (index into the engine's table)
    int64_t p0 = 0, n_range = 0;
    Item *d_heavy = nullptr;
    int n_heavy_groups = 0;
    Item *d_light = nullptr;
    int n_light = 0;
    // the mutual sweep's work list and fixed-point units (2^-bits)
    bool mutual = false;
    MutualItem *d_mutual = nullptr;
    int n_mutual = 0;
    bool onesided = false;  // met one-sided throughout (drop-in SICs)
    int fbits = 0, wbits = 0;
    int *d_counters = nullptr;
    void *d_out = nullptr;
    size_t out_bytes = 0;
    uint64_t pairs = 0, padded_pairs = 0;
    int grid = 0, warps = 0;
    cudaGraphExec_t graph = nullptr;  // the sweep, captured when it is run again
    int runs = 0;
};

// A kernel shape chosen by the autotuner, and what each candidate took.
struct Tuned {
    int variant = -1;
    float ms[8] = {};
};

// What two sweeps have to have in common for one's shape to serve the other:
// engine, slabs of the range (log2; the whole box -1), particles, pairs per
// particle, and the spline's reach in cells (log2; 0 without one).
typedef std::array<int, 5> TuneKey;

}  // namespace nf
struct nf_box;
namespace nf {

// The pencil engine, shared by the batched form (nf_box.cu) and the plain
// drop-in (nf_sic.cu).  A launch covers the pencils listed in `items` of a
// box described by float4 positions and a cell prefix array whose linear
// cell id is ((x*cpd)+y)*cpd+z for x in [0, nx).
struct EngineLaunch {
    const float4 *pos = nullptr;
    const int64_t *cs = nullptr;
    int cpd = 0;
    const Item *heavy = nullptr;  // CTA-split groups (WARPS_PER_CTA items each)
    int n_heavy_groups = 0;
    const Item *light = nullptr;
    int n_light = 0;
    int *counters = nullptr;      // 2 ints, zeroed by engine_launch
    Partial *part = nullptr;      // (2R+1) * nc * n_range partials
    int64_t p0 = 0, n_range = 0;  // the sinks' particle range
    int variant = 0;
    int grid = 0;                 // CTAs (0: one full wave)
    float eps = 0.f;              // softening parameter (0: the context's)
};
nf_status engine_launch(nf_ctx *ctx, const EngineLaunch &L, double box_h, cudaStream_t st);
// The sweep of a mutual plan: scratch (mutual_scratch_bytes) and counter are
// zeroed first; `before`, if given, is recorded between that and the sweep.
struct MutualLaunch {
    const Plan *plan = nullptr;
    const float4 *pos = nullptr;
    const int64_t *cs = nullptr;
    int cpd = 0;
    float eps = 0.f;  // softening parameter (0: the context's)
    void *scratch = nullptr;
    int *counter = nullptr;
    bool zeroed = false;  // scratch and counter are zero already (mutual_unpack)
    cudaEvent_t before = nullptr;
    unsigned event_flags = 0;
};
constexpr int MUTUAL_SHAPES = 5;  // kernel shapes the autotuner chooses among
const char *mutual_shape_name(int v);
int mutual_grid(nf_ctx *ctx, int variant);
nf_status mutual_noalloc_begin(int sms, const nf_config &cfg, int cpd, const int64_t *cs, int lo, int hi,
                               int64_t max_n, void *acc, int *counters, int64_t *bounds,
                               cudaStream_t st);
nf_status mutual_noalloc(int dev, int sms, const nf_config &cfg, const MutualLaunch &L, Plan &pl,
                         int64_t np_total, bool *done, cudaStream_t st);
// A SIC's positions (x, y, z of n4 each, a multiple of four, 16-byte aligned)
// to float4 records; zeroes scratch and counter.
nf_status mutual_unpack(nf_ctx *ctx, const Plan &pl, const float *xyz, int64_t n4, float4 *pos,
                        void *scratch, int *counter, cudaStream_t st);
// A sink pencil of a drop-in SIC: centre cell (y, z) of the middle slab, its
// sinks [first, first + n) in the pencil's sink stream, its sources.
struct SicPencil {
    int y, z;
    int64_t first, n, sources;
};
bool mutual_sic_list(const nf_config &cfg, int cpd, const std::vector<SicPencil> &pencils, const int64_t *cs,
                     int warps, Plan &pl, std::vector<MutualItem> &items);
nf_status mutual_plan(nf_ctx *ctx, const nf_box *box, int lo, int hi, int variant, Plan &pl);
nf_status mutual_launch(nf_ctx *ctx, const MutualLaunch &L, cudaStream_t st);
// Device memory of a context's boxes and plans.  What is freed stays for the
// next box, up to KEEP_BYTES + KEEP_POOL_BYTES: a simulation that makes a box
// each step asks for the same blocks again (1.2 GB for 256^3 particles: 55.5 ms
// a step, 60 ms with half of it kept).  It goes back to the device at
// nf_shutdown, when a server starts, by nf_trim, and when any allocation of
// this library runs out.
// Blocks below BIG come from a memory pool, made when the first is asked for (a
// context without boxes, as a driver's, makes none); others from cudaMalloc,
// kept in a list.  New memory costs a pool 6 ms a GB (a block of 256 MB 1.5
// ms) and cudaMalloc 0.35 ms whatever the size, so boxes of 256^3 take 8.5 ms to
// make from the pool and 4.5 so; and cudaMalloc waits for the device, which
// the work lists of a server's 90 slabs, made while requests run, cannot afford
// (first pass of serving 95 ms, with cudaMalloc for all 107-167).
// A block handed to free() is idle: no work that uses it is in flight.
class DeviceMemory {
  public:
    static constexpr size_t BIG = (size_t)32 << 20;
    static constexpr size_t KEEP_BYTES = (size_t)1792 << 20, KEEP_POOL_BYTES = (size_t)256 << 20;
    ~DeviceMemory();
    // own: the context's own stream, on which the pool's blocks are handed out
    // and freed
    cudaError_t alloc(int device, cudaStream_t own, void **p, size_t bytes);
    void free(cudaStream_t own, void *p);
    void trim();   // gives back what is unused
    void close();  // before the stream goes
    static void trim_all();  // of every context of the process

  private:
    cudaError_t alloc_big(void **p, size_t bytes);
    struct Block {
        void *p;
        size_t bytes;
    };
    std::mutex mu;
    bool known = false;  // to trim_all(): from the first block on, so that the
                         // allocation-free call's context costs nothing
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;
    std::list<Block> kept;  // oldest first
    size_t kept_bytes = 0;
    std::unordered_map<void *, size_t> big;  // handed out
};
// cudaMalloc that takes back what contexts keep before it gives up.
cudaError_t device_malloc(void **p, size_t bytes);
template <class T>
cudaError_t device_malloc(T **p, size_t bytes) {
    return device_malloc((void **)p, bytes);
}
cudaError_t pool_alloc(nf_ctx *ctx, void **p, size_t bytes);
template <class T>
cudaError_t pool_alloc(nf_ctx *ctx, T **p, size_t bytes) {
    return pool_alloc(ctx, (void **)p, bytes);
}
void pool_free(nf_ctx *ctx, void *p);  // null ctx: of a context that is gone
size_t mutual_scratch_bytes(int64_t n_range, int nc);
// Records of a plan's sums (one-sided: partials; mutual: fixed point).
nf_status engine_coadd_plan(nf_ctx *ctx, const Plan &pl, const void *scratch, void *out,
                            cudaStream_t st, float eps, const uint32_t *perm);
// perm (optional): the caller's index of each packed slot; record p of the
// range [p0, p0 + n) is written at perm[p0 + p] - p0.
nf_status engine_coadd(nf_ctx *ctx, const Partial *part, int64_t n, void *out, cudaStream_t st,
                       float eps = 0.f, const uint32_t *perm = nullptr, int64_t p0 = 0);
nf_status engine_pack(nf_ctx *ctx, const float *x, const float *y, const float *z, int64_t n,
                      float4 *out, cudaStream_t st);
int engine_grid(nf_ctx *ctx, int variant);
int engine_plain_variant();
const char *engine_shape_name(int v);
constexpr int ENGINE_WARPS_PER_CTA = 8;
// SIC size limits from a buffer budget (the reference's bytes-per-block model).
nf_status sic_limits(int out_kind, int cpd, uint64_t max_buffer_bytes, nf_gpu_limits *lim);
// The cached work list of a box's slab range (nf_box.cu).
nf_status box_plan(nf_ctx *ctx, nf_box *box, int lo, int hi, const Plan **out);

}  // namespace nf

struct nf_box {
    int cpd = 0;
    int64_t np = 0;
    std::vector<int64_t> cell_start;  // host copy, cpd^3 + 1
    float4 *d_pos = nullptr;          // np records (x, y, z, 0), cell order
    int64_t *d_cs = nullptr;          // cell_start on the device
    nf::Partial *d_part = nullptr;    // pencil partials scratch
    float *d_stage = nullptr;         // position upload staging, 3 * np floats
    uint32_t *d_perm = nullptr;       // caller's index of the particle in each packed slot
    void *d_sort = nullptr;           // in-cell ordering scratch (keys, values, sort temp)
    size_t sort_bytes = 0;
    // pipelined step (nf_box_step): copy-in and copy-out streams, per-chunk events
    cudaStream_t s_in = nullptr, s_out = nullptr;
    cudaStream_t s_sweep = nullptr;   // every other chunk's sweep, with sums of its own
    void *d_part2 = nullptr;
    size_t part2_bytes = 0;
    std::vector<cudaEvent_t> step_ev;
    size_t part_bytes = 0;
    std::map<std::pair<int, int>, std::unique_ptr<nf::Plan>> plans;
    nf::Tuned tuned[2];  // kernel shape by engine (NF_ENGINE_*), as chosen by the autotuner
    int engine = 0;      // of the plan built last
    std::atomic<int> serving{0};  // admitted requests whose work may still read the box
    float eps = 0.f;        // the box's own softening parameter (0: the context's)
    size_t device_bytes() const;
};

struct nf_ctx {
    nf_config cfg{};
    int device = 0;
    int sms = 0;
    cudaStream_t stream = nullptr;      // where work is enqueued (own or caller's)
    cudaStream_t own_stream = nullptr;  // created by nf_init
    cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
    nf_timing last{};
    std::atomic<int> engine{-1};  // of the last sweep (NF_ENGINE_*)
    std::mutex mu;  // serialises nf_box_forces on one context
    nf::DeviceMemory memory;  // of boxes and plans
    std::map<nf::TuneKey, nf::Tuned> tuned;  // shapes chosen so far
    // plain drop-in GPU control (nf_sic.cu)
    struct Sic;
    Sic *sic = nullptr;
};
