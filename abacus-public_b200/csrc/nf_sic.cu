// nf_sic.cu -- plain drop-in: GPU control and SetInteractionCollection execution.
//
// Replaces singlestep/Direct/GPUControl.cu (GPUSetup, GPUReset, the queue
// watchers) and PencilTask.cu (GPUPencilTask).  The contract kept from the
// reference: one SIC covers every sink z-pencil of rows [j_low, j_high) of
// one x-slab and the 2R+1 source slabs around it; after it completes, the
// caller's AccSlab rows [j_low, j_high) hold the near-field accelerations and
// the SIC's completion flag is set.  SICs are queued to worker threads, one
// per (GPU x buffers-per-device) buffer, each with its own stream.
//
// How a SIC runs here (B200-first, not the reference's pencil gather):
//   1. the SIC's source rows of the 2R+1 slabs (each particle once, rather
//      than the reference's five copies per pencil, PencilPlan.cc:22-90,
//      214-255) are packed into pinned staging with the work list and the cell table, and
//      copied to the device at once;
//   2. a pack kernel builds float4 records, forming a "mini box" of 2R+1
//      slabs with the SIC's cell offsets;
//   3. one launch of the engine of nf_mutual.cu, one-sided, sums the 2R+1
//      pencils of each sink on the device (PencilPlan.cc:140-207 co-adds on
//      the host);
//   4. the rows' accelerations are copied back and stored into AccSlab.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>

#include "nf_internal.h"

namespace nf {

static_assert(ENGINE_WARPS_PER_CTA == 8, "engine CTA shape");

constexpr int NFBLOCK = 64;    // NFBlockSize (configure.ac:160-162)
constexpr int SPLIT_MIN_SOURCES = 64;  // sources per warp of a split tile (one staged chunk)
constexpr int REF_WIDTH = 5;   // WIDTH = 2*NFRADIUS+1, NFRADIUS = 2 (GPUControl.cu:109-113)

struct SicTask {
    nf_sic_desc d;  // shallow copy: the arrays stay owned by the caller
    int jlow = 0, jhigh = 0;
    volatile int *completion = nullptr;
};

struct SicBuffer {
    int index = 0, device = 0;
    bool pinned = true;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;  // around the pencil kernel of a SIC
    std::mutex mu;
    float *d_raw = nullptr;
    float4 *d_pos = nullptr;
    int64_t *d_cs = nullptr;
    Item *d_items = nullptr;
    void *d_part = nullptr;  // the sums: fixed point, or pencil partials
    void *d_out = nullptr;
    int *d_counters = nullptr;
    float *h_raw = nullptr;
    void *h_out = nullptr;
    int64_t *h_cs = nullptr;
    Item *h_items = nullptr;
    size_t cap_particles = 0, cap_sinks = 0, cap_part = 0, cap_items = 0, cap_cells = 0;
    // mutual form: cell table, work list and positions in one block, one copy
    void *h_block = nullptr, *d_block = nullptr;
    size_t cap_block = 0, cap_pos = 0;
    int grid = 0;  // CTAs of a full mutual launch
    std::vector<int64_t> cnt, rowstart, cellstart, cs;
    std::vector<SicPencil> pencils;
    std::vector<MutualItem> list;
};

static void host_free(void *p, bool pinned) {
    if (!p) return;
    if (pinned)
        cudaFreeHost(p);
    else
        free(p);
}

static cudaError_t host_alloc(void **p, size_t bytes, bool pinned, bool wc) {
    if (pinned) return cudaHostAlloc(p, bytes, wc ? cudaHostAllocWriteCombined : cudaHostAllocDefault);
    *p = aligned_alloc(4096, (bytes + 4095) / 4096 * 4096);
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}

static void release(SicBuffer &b) {
    cudaSetDevice(b.device);
    cudaFree(b.d_raw);
    cudaFree(b.d_pos);
    cudaFree(b.d_cs);
    cudaFree(b.d_items);
    cudaFree(b.d_part);
    cudaFree(b.d_out);
    cudaFree(b.d_counters);
    cudaFree(b.d_block);
    host_free(b.h_block, b.pinned);
    b.d_block = b.h_block = nullptr;
    b.cap_block = b.cap_pos = 0;
    host_free(b.h_raw, b.pinned);
    host_free(b.h_out, b.pinned);
    host_free(b.h_cs, b.pinned);
    host_free(b.h_items, b.pinned);
    if (b.stream) cudaStreamDestroy(b.stream);
    if (b.ev0) cudaEventDestroy(b.ev0);
    if (b.ev1) cudaEventDestroy(b.ev1);
    b.ev0 = b.ev1 = nullptr;
    b.d_raw = nullptr;
    b.d_pos = nullptr;
    b.d_cs = nullptr;
    b.d_items = nullptr;
    b.d_part = nullptr;
    b.d_out = nullptr;
    b.d_counters = nullptr;
    b.h_raw = nullptr;
    b.h_out = nullptr;
    b.h_cs = nullptr;
    b.h_items = nullptr;
    b.stream = nullptr;
    b.cap_particles = b.cap_sinks = b.cap_part = b.cap_items = b.cap_cells = 0;
}

// Grow a buffer's arrays to hold a task (1.25x headroom; never shrinks).
// block: bytes of the mutual form's block, 0 for the one-sided form.
static nf_status grow(nf_ctx *ctx, SicBuffer &b, size_t particles, size_t sinks, size_t items,
                      size_t cells, size_t block) {
    const int W = 2 * ctx->cfg.near_field_radius + 1;
    const int nc = ctx->cfg.b2 > 0.f ? 4 : 3;
    const size_t rec = ctx->cfg.out_kind == NF_OUT_FLOAT4 ? 16 : 12;
    auto up = [](size_t n) { return n + n / 4 + 1024; };
    if (particles > b.cap_pos) {
        size_t c = up(particles);
        cudaFree(b.d_pos);
        b.d_pos = nullptr;
        b.cap_pos = 0;
        NF_CUDA(device_malloc(&b.d_pos, c * sizeof(float4)));
        b.cap_pos = c;
    }
    if (block > b.cap_block) {
        size_t c = up(block);
        cudaFree(b.d_block);
        host_free(b.h_block, b.pinned);
        b.d_block = b.h_block = nullptr;
        b.cap_block = 0;
        NF_CUDA(device_malloc(&b.d_block, c));
        NF_CUDA(host_alloc(&b.h_block, c, b.pinned, true));
        b.cap_block = c;
    }
    if (block == 0 && particles > b.cap_particles) {
        size_t c = up(particles);
        cudaFree(b.d_raw);
        host_free(b.h_raw, b.pinned);
        b.d_raw = nullptr;
        b.h_raw = nullptr;
        b.cap_particles = 0;
        NF_CUDA(device_malloc(&b.d_raw, 3 * c * sizeof(float)));
        NF_CUDA(host_alloc((void **)&b.h_raw, 3 * c * sizeof(float), b.pinned, true));
        b.cap_particles = c;
    }
    const size_t part = block ? mutual_scratch_bytes((int64_t)sinks, nc) : (size_t)W * nc * sinks * sizeof(Partial);
    if (part > b.cap_part) {
        size_t c = up(part);
        cudaFree(b.d_part);
        b.d_part = nullptr;
        b.cap_part = 0;
        NF_CUDA(device_malloc(&b.d_part, c));
        b.cap_part = c;
    }
    if (sinks > b.cap_sinks) {
        size_t c = up(sinks);
        cudaFree(b.d_out);
        host_free(b.h_out, b.pinned);
        b.d_out = nullptr;
        b.h_out = nullptr;
        b.cap_sinks = 0;
        NF_CUDA(device_malloc(&b.d_out, c * rec));
        NF_CUDA(host_alloc(&b.h_out, c * rec, b.pinned, false));
        b.cap_sinks = c;
    }
    if (items > b.cap_items) {
        size_t c = up(items);
        cudaFree(b.d_items);
        host_free(b.h_items, b.pinned);
        b.d_items = nullptr;
        b.h_items = nullptr;
        b.cap_items = 0;
        NF_CUDA(device_malloc(&b.d_items, c * sizeof(Item)));
        NF_CUDA(host_alloc((void **)&b.h_items, c * sizeof(Item), b.pinned, true));
        b.cap_items = c;
    }
    if (cells > b.cap_cells) {
        size_t c = cells;
        cudaFree(b.d_cs);
        host_free(b.h_cs, b.pinned);
        b.d_cs = nullptr;
        b.h_cs = nullptr;
        b.cap_cells = 0;
        NF_CUDA(device_malloc(&b.d_cs, c * sizeof(int64_t)));
        NF_CUDA(host_alloc((void **)&b.h_cs, c * sizeof(int64_t), b.pinned, true));
        b.cap_cells = c;
    }
    if (!b.d_counters) NF_CUDA(device_malloc(&b.d_counters, 2 * sizeof(int)));
    return NF_OK;
}

static inline int wrapi(int i, int n) {
    i %= n;
    return i < 0 ? i + n : i;
}

// Validate the descriptor against the SIC geometry (the reference asserts
// the same sizes, PencilOnPencil.cc:221-236, 380-401).
static nf_status check_desc(nf_ctx *ctx, const nf_sic_desc &d, int jlow, int jhigh) {
    const int R = d.nfradius, W = 2 * R + 1;
    if (R != ctx->cfg.near_field_radius) {
        set_error("nf_sic_execute: nfradius differs from the context's near_field_radius");
        return NF_EINVAL;
    }
    const bool two_d = d.node_z_size > 0;
    if (d.cpd < W || (d.cpd & 1) == 0 || jlow < 0 || jhigh > d.cpd || jlow >= jhigh ||
        (!two_d && d.nk != d.cpd) ||
        (two_d && (d.nk != d.node_z_size + 2 * R || d.node_z_size + 2 * R > d.cpd ||
                   d.node_z_start < 0 || d.node_z_start >= d.cpd))) {
        set_error("nf_sic_execute: bad geometry (odd cpd >= 2R+1, 0 <= jlow < jhigh <= cpd, Nk == "
                  "cpd; 2D: Nk == node_z_size + 2R, node_z_size + 2R <= cpd)");
        return NF_EINVAL;
    }
    const int jw = jhigh - jlow;
    if (d.nsinksets != jw * d.nk || d.nsourcesets != d.nk * (jw + 2 * R) ||
        d.interaction_count != W * d.nsinksets) {
        set_error("nf_sic_execute: set counts do not match j_width, Nk and nfradius");
        return NF_EINVAL;
    }
    if (!d.sink_plan || !d.source_plan || !d.sink_pos_slab || !d.source_pos_slab ||
        !d.source_nslab || !d.sink_acc_slab || !d.sink_set_count || !d.source_set_count) {
        set_error("nf_sic_execute: null array in the descriptor");
        return NF_EINVAL;
    }
    if (d.interaction_list) {
        for (int j = 0; j < jw; j++)
            for (int k = 0; k < d.nk; k++)
                for (int y = 0; y < W; y++)
                    if (d.interaction_list[(j * d.nk + k) * W + y] != (j + y) * d.nk + k) {
                        set_error("nf_sic_execute: interaction list is not the pencil pattern");
                        return NF_EINVAL;
                    }
    }
    return NF_OK;
}

// Pencil k of a row is centred on z = (k + R) mod cpd (index_to_zcen,
// PencilOnPencil.cc:37-43, one z-domain per node); 2D: on node_z_start + k + R,
// brought back by node_z_size + 2R past the upper ghost edge, so the centres
// cover the primary cells and R ghost cells on each side.
static int pencil_z(const nf_sic_desc &d, int k) {
    const int R = d.nfradius, zs = d.node_z_start, zn = d.node_z_size;
    if (zn == 0) return (k + R) % d.cpd;
    int kk = k + zs + R;
    if (kk >= zs + zn + R) kk -= zn + 2 * R;
    return wrapi(kk, d.cpd);
}

static bool primary_z(const nf_sic_desc &d, int z) {
    return d.node_z_size == 0 || wrapi(z - d.node_z_start, d.cpd) < d.node_z_size;
}

static void sic_account(nf_ctx *ctx, float kernel_ms, uint64_t pairs);

// Stage the SIC's source cells (each particle once) as SoA at hx, hy, hz; runs
// that follow each other in the slab and in the mini box go as one copy.  1D:
// whole rows; 2D: cell by cell (ghost cells included).
static nf_status stage_sources(const SicBuffer &b, const SicTask &t, float *hx, float *hy, float *hz) {
    const nf_sic_desc &d = t.d;
    const int R = d.nfradius, W = 2 * R + 1, cpd = d.cpd;
    const bool two_d = d.node_z_size > 0;
    const int step = two_d ? 1 : cpd;  // cells of a unit
    for (int s = 0; s < W; s++) {
        const float *slab = d.source_pos_slab[s];
        const uint64_t ns = d.source_nslab[s];
        int64_t run_src = 0, run_dst = 0, run_n = 0;
        auto flush = [&]() {
            if (run_n == 0) return;
            memcpy(hx + run_dst, slab + run_src, run_n * sizeof(float));
            memcpy(hy + run_dst, slab + ns + run_src, run_n * sizeof(float));
            memcpy(hz + run_dst, slab + 2 * ns + run_src, run_n * sizeof(float));
        };
        const int64_t c_end = (int64_t)(s + 1) * cpd * cpd;
        for (int64_t c = (int64_t)s * cpd * cpd; c < c_end; c += step) {
            const int64_t dst = b.cs[c], n = b.cs[c + step] - dst;
            if (n == 0) continue;
            const int64_t src = two_d ? b.cellstart[c] : b.rowstart[c / cpd];
            if (src < 0 || (uint64_t)(src + n) > ns) {
                set_error(two_d ? "nf_sic_execute: source cell outside its slab"
                                : "nf_sic_execute: source row outside its slab");
                return NF_EINVAL;
            }
            if (run_n > 0 && src == run_src + run_n && dst == run_dst + run_n) {
                run_n += n;
            } else {
                flush();
                run_src = src;
                run_dst = dst;
                run_n = n;
            }
        }
        flush();
    }
    return NF_OK;
}

// Copy a SIC's records to AccSlab.  1D: rows [jlow, jhigh) are contiguous from
// the first sink cell of row jlow, the centre cell of the row-jlow pencil
// centred on z = 0.  2D: primary cells only, each at its AccSlab start (the
// centre cell of the pencil centred on it); cells adjacent in both go as one
// run.
static nf_status store_records(nf_ctx *ctx, const SicBuffer &b, const SicTask &t, int64_t p0,
                               int64_t n_sinks) {
    const nf_sic_desc &d = t.d;
    const int R = d.nfradius, W = 2 * R + 1, cpd = d.cpd, nk = d.nk;
    const size_t rec = ctx->cfg.out_kind == NF_OUT_FLOAT4 ? 16 : 12;
    if (d.node_z_size == 0) {
        if (n_sinks <= 0) return NF_OK;
        const int k0 = (cpd - R) % cpd;
        const int64_t acc0 = d.sink_plan[(int64_t)k0 * W + R].start;
        memcpy((char *)d.sink_acc_slab + acc0 * rec, b.h_out, (size_t)n_sinks * rec);
        return NF_OK;
    }
    size_t run_acc = 0, run_out = 0, run_bytes = 0;
    auto flush = [&]() {
        if (run_bytes) memcpy((char *)d.sink_acc_slab + run_acc, (char *)b.h_out + run_out, run_bytes);
        run_bytes = 0;
    };
    for (int j = 0; j < t.jhigh - t.jlow; j++)
        for (int k = 0; k < nk; k++) {
            const int y = t.jlow + j, zc = pencil_z(d, k);
            if (!primary_z(d, zc)) continue;
            const nf_cell_plan &ce = d.sink_plan[((int64_t)j * nk + k) * W + R];
            const int64_t c = ((int64_t)R * cpd + y) * cpd + zc;
            if (ce.n != b.cnt[c]) {
                set_error("nf_sic_execute: sink plan and source plan disagree on a cell");
                return NF_EINVAL;
            }
            if (ce.n == 0) continue;
            const size_t acc = (size_t)ce.start * rec, out = (size_t)(b.cs[c] - p0) * rec;
            const size_t bytes = (size_t)ce.n * rec;
            if (run_bytes && acc == run_acc + run_bytes && out == run_out + run_bytes) {
                run_bytes += bytes;
            } else {
                flush();
                run_acc = acc;
                run_out = out;
                run_bytes = bytes;
            }
        }
    flush();
    return NF_OK;
}

// A SIC on the engine of nf_mutual.cu, every pair met one-sided: tiles are up
// to 128 sinks and split until the launch is full.  Work list, cell table and
// positions go over in one copy.
static nf_status launch_list(nf_ctx *ctx, SicBuffer &b, const SicTask &t, Plan &pl, int64_t n_mini,
                             uint64_t *bytes_to_device) {
    const size_t items_b = b.list.size() * sizeof(MutualItem);
    const size_t cs_b = (b.cs.size() * sizeof(int64_t) + 15) / 16 * 16, tables = items_b + cs_b;
    const size_t n4 = ((size_t)n_mini + 3) / 4 * 4, bytes = tables + 3 * n4 * sizeof(float);
    nf_status st = grow(ctx, b, n4, (size_t)pl.n_range, 0, 0, bytes);
    if (st != NF_OK) return st;
    char *h = (char *)b.h_block, *dev = (char *)b.d_block;
    memcpy(h, b.list.data(), items_b);
    memcpy(h + items_b, b.cs.data(), b.cs.size() * sizeof(int64_t));
    float *hx = (float *)(h + tables);
    st = stage_sources(b, t, hx, hx + n4, hx + 2 * n4);
    if (st != NF_OK) return st;
    cudaStream_t sm = b.stream;
    NF_CUDA(cudaMemcpyAsync(dev, h, bytes, cudaMemcpyHostToDevice, sm));
    st = mutual_unpack(ctx, pl, (const float *)(dev + tables), (int64_t)n4, b.d_pos, b.d_part,
                       b.d_counters, sm);
    if (st != NF_OK) return st;
    pl.d_mutual = (MutualItem *)dev;
    // a short list takes no more CTAs than it fills: the rest is for other SICs
    pl.grid = (int)std::min<int64_t>(b.grid, (pl.n_mutual + ENGINE_WARPS_PER_CTA - 1) / ENGINE_WARPS_PER_CTA);
    MutualLaunch L;
    L.zeroed = true;
    L.plan = &pl;
    L.pos = b.d_pos;
    L.cs = (const int64_t *)(dev + items_b);
    L.cpd = t.d.cpd;
    L.scratch = b.d_part;
    L.counter = b.d_counters;
    L.before = b.ev0;
    st = mutual_launch(ctx, L, sm);
    if (st != NF_OK) return st;
    NF_CUDA(cudaEventRecord(b.ev1, sm));
    *bytes_to_device = bytes;
    // the records: written to pinned host memory by the co-add itself
    return engine_coadd_plan(ctx, pl, b.d_part, b.pinned ? b.h_out : b.d_out, sm, 0.f, nullptr);
}

// A SIC on the one-sided engine of nf_box.cu (plain accumulation, softenings
// below the other's fixed-point range): tiles of 64 sinks (the reference
// block).
static nf_status launch_tiles(nf_ctx *ctx, SicBuffer &b, const SicTask &t, int64_t n_mini, int64_t p0,
                              int64_t n_sinks, uint64_t *bytes_to_device) {
    const int cpd = t.d.cpd, R = t.d.nfradius;
    std::vector<Item> items;
    items.reserve(2 * b.pencils.size());
    for (const SicPencil &p : b.pencils)
        for (int64_t b0 = 0; b0 < p.n; b0 += NFBLOCK) {
            const int take = (int)std::min<int64_t>(NFBLOCK, p.n - b0);
            items.push_back(Item{(int)(((int64_t)R * cpd + p.y) * cpd + p.z), (int)(p.first + b0), take,
                                 take <= 32 ? 1 : 2, 0, (int)p.sources, 0, 0});
        }
    // longest tiles first (the order of execution does not change any
    // result: every tile writes its own partials)
    std::stable_sort(items.begin(), items.end(), [](const Item &a, const Item &b) {
        return (int64_t)a.nsink * a.src_end > (int64_t)b.nsink * b.src_end;
    });
    // A SIC with fewer tiles than the launch has warps (small boxes, thin
    // y-splits) would leave most of the GPU idle: then every tile with at
    // least 64 sources per warp is split over the 8 warps of a CTA along its
    // source stream (summed in warp order in shared memory), the engine's
    // CTA-split path.  Launch order: split tiles, then the others.
    std::vector<Item> launch_items;
    int n_split = 0;
    {
        const int warps = engine_grid(ctx, engine_plain_variant()) * ENGINE_WARPS_PER_CTA;
        std::vector<Item> keep;
        if ((int64_t)items.size() < warps) {
            for (const Item &t : items) {
                const int M = t.src_end;
                if (M < SPLIT_MIN_SOURCES * ENGINE_WARPS_PER_CTA) {
                    keep.push_back(t);
                    continue;
                }
                const int per = ((M + ENGINE_WARPS_PER_CTA - 1) / ENGINE_WARPS_PER_CTA +
                                 SPLIT_MIN_SOURCES - 1) / SPLIT_MIN_SOURCES * SPLIT_MIN_SOURCES;
                for (int w = 0; w < ENGINE_WARPS_PER_CTA; w++) {
                    Item it = t;
                    it.src_begin = std::min(M, w * per);
                    it.src_end = std::min(M, (w + 1) * per);
                    launch_items.push_back(it);
                }
                n_split++;
            }
        } else {
            keep = items;
        }
        launch_items.insert(launch_items.end(), keep.begin(), keep.end());
    }
    const size_t nitems = launch_items.size();
    nf_status st = grow(ctx, b, (size_t)n_mini, (size_t)n_sinks, nitems, b.cs.size(), 0);
    if (st != NF_OK) return st;
    float *hx = b.h_raw, *hy = b.h_raw + b.cap_particles, *hz = b.h_raw + 2 * b.cap_particles;
    st = stage_sources(b, t, hx, hy, hz);
    if (st != NF_OK) return st;
    memcpy(b.h_cs, b.cs.data(), b.cs.size() * sizeof(int64_t));
    if (nitems) memcpy(b.h_items, launch_items.data(), nitems * sizeof(Item));
    cudaStream_t sm = b.stream;
    const size_t pb = (size_t)n_mini * sizeof(float), cs_b = b.cs.size() * sizeof(int64_t);
    NF_CUDA(cudaMemcpyAsync(b.d_raw, hx, pb, cudaMemcpyHostToDevice, sm));
    NF_CUDA(cudaMemcpyAsync(b.d_raw + b.cap_particles, hy, pb, cudaMemcpyHostToDevice, sm));
    NF_CUDA(cudaMemcpyAsync(b.d_raw + 2 * b.cap_particles, hz, pb, cudaMemcpyHostToDevice, sm));
    NF_CUDA(cudaMemcpyAsync(b.d_cs, b.h_cs, cs_b, cudaMemcpyHostToDevice, sm));
    if (nitems)
        NF_CUDA(cudaMemcpyAsync(b.d_items, b.h_items, nitems * sizeof(Item), cudaMemcpyHostToDevice, sm));
    st = engine_pack(ctx, b.d_raw, b.d_raw + b.cap_particles, b.d_raw + 2 * b.cap_particles, n_mini,
                     b.d_pos, sm);
    if (st != NF_OK) return st;
    EngineLaunch L;
    L.pos = b.d_pos;
    L.cs = b.d_cs;
    L.cpd = cpd;
    L.heavy = b.d_items;
    L.n_heavy_groups = n_split;
    L.light = b.d_items + (size_t)n_split * ENGINE_WARPS_PER_CTA;
    L.n_light = (int)nitems - n_split * ENGINE_WARPS_PER_CTA;
    L.counters = b.d_counters;
    L.part = (Partial *)b.d_part;
    L.p0 = p0;
    L.n_range = n_sinks;
    L.variant = engine_plain_variant();
    NF_CUDA(cudaEventRecord(b.ev0, sm));
    st = engine_launch(ctx, L, 1.0 / cpd, sm);
    if (st != NF_OK) return st;
    NF_CUDA(cudaEventRecord(b.ev1, sm));
    *bytes_to_device = 3 * pb + cs_b + nitems * sizeof(Item);
    return engine_coadd(ctx, (const Partial *)b.d_part, n_sinks, b.d_out, sm);
}

static nf_status run_task(nf_ctx *ctx, SicBuffer &b, const SicTask &t) {
    const nf_sic_desc &d = t.d;
    nf_status st = check_desc(ctx, d, t.jlow, t.jhigh);
    if (st != NF_OK) return st;
    NF_CUDA(cudaSetDevice(b.device));
    const int R = d.nfradius, W = 2 * R + 1, cpd = d.cpd, nk = d.nk;
    const int jw = t.jhigh - t.jlow, nrows = jw + 2 * R;
    const int64_t ncell = (int64_t)W * cpd * cpd;
    const bool two_d = d.node_z_size > 0;
    // cell counts of the mini box: slot s = source slab x-R+s, rows of the SIC
    std::vector<int64_t> &cnt = b.cnt, &cs = b.cs;
    cnt.assign(ncell, 0);
    b.rowstart.assign(W * cpd, -1);
    if (two_d) b.cellstart.assign(ncell, -1);
    for (int r = 0; r < nrows; r++) {
        const int y = wrapi(t.jlow - R + r, cpd);
        for (int k = 0; k < nk; k++) {
            const int z = pencil_z(d, k);
            const nf_cell_plan *pl = d.source_plan + ((int64_t)r * nk + k) * W;
            for (int s = 0; s < W; s++) {
                if (pl[s].n < 0) {
                    set_error("nf_sic_execute: negative cell count");
                    return NF_EINVAL;
                }
                const int64_t c = ((int64_t)s * cpd + y) * cpd + z;
                cnt[c] = pl[s].n;
                if (two_d) b.cellstart[c] = pl[s].start;
                else if (z == 0) b.rowstart[s * cpd + y] = pl[s].start;
            }
        }
    }
    // dense mirror offsets (linear cell order)
    cs.resize(ncell + 1);
    cs[0] = 0;
    for (int64_t c = 0; c < ncell; c++) cs[c + 1] = cs[c] + cnt[c];
    const int64_t n_mini = cs[ncell];
    const int64_t p0 = cs[((int64_t)R * cpd + t.jlow) * cpd];
    const int64_t p1 = cs[((int64_t)R * cpd + t.jhigh) * cpd];
    const int64_t n_sinks = p1 - p0;
    // sink pencils, checked against the descriptor
    auto count = [&](int s, int y, int z) {
        return cnt[((int64_t)s * cpd + wrapi(y, cpd)) * cpd + wrapi(z, cpd)];
    };
    b.pencils.clear();
    for (int j = 0; j < jw; j++)
        for (int k = 0; k < nk; k++) {
            SicPencil p{t.jlow + j, pencil_z(d, k), 0, 0, 0};
            // 2D: the primary cells of a pencil are contiguous in its sink
            // stream, after `first` ghost sinks; only they are swept (the
            // reference truncates sink pencils the same way,
            // PencilPlan.cc:110-116)
            bool seen_primary = false;
            for (int a = -R; a <= R; a++) {
                if (primary_z(d, p.z + a)) {
                    p.n += count(R, p.y, p.z + a);
                    seen_primary = true;
                } else if (!seen_primary) {
                    p.first += count(R, p.y, p.z + a);
                }
            }
            if (p.n != d.sink_set_count[j * nk + k]) {
                set_error("nf_sic_execute: SinkSetCount disagrees with the source plans");
                return NF_EINVAL;
            }
            if (p.n == 0) continue;
            for (int dx = -R; dx <= R; dx++)
                for (int dy = -R; dy <= R; dy++) p.sources += count(R + dx, p.y + dy, p.z);
            b.pencils.push_back(p);
        }
    uint64_t pairs = 0, to_device = 0;
    for (const SicPencil &p : b.pencils) pairs += (uint64_t)p.n * (uint64_t)p.sources;
    if (!b.grid) b.grid = mutual_grid(ctx, 0);
    Plan pl;
    pl.p0 = p0;
    pl.n_range = n_sinks;
    const bool listed =
        mutual_sic_list(ctx->cfg, cpd, b.pencils, cs.data(), b.grid * ENGINE_WARPS_PER_CTA, pl, b.list);
    if (listed)
        st = launch_list(ctx, b, t, pl, n_mini, &to_device);
    else
        st = launch_tiles(ctx, b, t, n_mini, p0, n_sinks, &to_device);
    if (st != NF_OK) return st;
    const size_t rec = ctx->cfg.out_kind == NF_OUT_FLOAT4 ? 16 : 12;
    cudaStream_t sm = b.stream;
    if (n_sinks && !(listed && b.pinned))
        NF_CUDA(cudaMemcpyAsync(b.h_out, b.d_out, (size_t)n_sinks * rec, cudaMemcpyDeviceToHost, sm));
    NF_CUDA(cudaStreamSynchronize(sm));
    float kms = 0.f;
    NF_CUDA(cudaEventElapsedTime(&kms, b.ev0, b.ev1));
    sic_account(ctx, kms, pairs);
    st = store_records(ctx, b, t, p0, n_sinks);
    if (st != NF_OK) return st;
    if (d.bytes_to_device) *d.bytes_to_device += to_device;
    if (d.bytes_from_device) *d.bytes_from_device += (size_t)n_sinks * rec;
    return NF_OK;
}

}  // namespace nf

using namespace nf;

struct nf_ctx::Sic {
    std::vector<std::unique_ptr<SicBuffer>> buffers;
    std::deque<SicTask> queue;
    std::mutex mu;
    std::condition_variable cv, idle;
    bool stop = false;
    int active = 0;
    std::vector<std::thread> workers;
    nf_gpu_limits limits{};
    int cpd = 0;
    std::string error;  // first failure seen by a worker
    // pencil-kernel time of completed SICs (CUDA events around each launch)
    double kernel_ms = 0.0;
    uint64_t sics = 0, pairs = 0;
};

void nf::sic_account(nf_ctx *ctx, float kernel_ms, uint64_t pairs) {
    std::lock_guard<std::mutex> lk(ctx->sic->mu);
    ctx->sic->kernel_ms += kernel_ms;
    ctx->sic->sics++;
    ctx->sic->pairs += pairs;
}

static void finish(nf_ctx *ctx, const SicTask &t, nf_status st) {
    if (st != NF_OK) {
        std::lock_guard<std::mutex> lk(ctx->sic->mu);
        if (ctx->sic->error.empty()) ctx->sic->error = nf_last_error();
    }
    __atomic_store_n((int *)t.completion, st == NF_OK ? 1 : -1, __ATOMIC_RELEASE);
}

static void worker_main(nf_ctx *ctx, SicBuffer *b) {
    cudaSetDevice(b->device);
    auto *S = ctx->sic;
    for (;;) {
        SicTask t;
        {
            std::unique_lock<std::mutex> lk(S->mu);
            S->cv.wait(lk, [&] { return S->stop || !S->queue.empty(); });
            if (S->queue.empty()) break;  // stop requested and drained
            t = S->queue.front();
            S->queue.pop_front();
            S->active++;
        }
        nf_status st;
        {
            std::lock_guard<std::mutex> bl(b->mu);
            st = run_task(ctx, *b, t);
        }
        finish(ctx, t, st);
        {
            std::lock_guard<std::mutex> lk(S->mu);
            S->active--;
        }
        S->idle.notify_all();
    }
}

void nf_sic_shutdown(nf_ctx *ctx) {
    if (!ctx || !ctx->sic) return;
    auto *S = ctx->sic;
    {
        std::lock_guard<std::mutex> lk(S->mu);
        S->stop = true;
    }
    S->cv.notify_all();
    for (auto &th : S->workers)
        if (th.joinable()) th.join();
    for (auto &b : S->buffers) release(*b);
    delete S;
    ctx->sic = nullptr;
    cudaSetDevice(ctx->device);
}

// MaxSinkBlocks and friends from a buffer budget, GPUControl.cu:374-408:
// per sink block 64*accstruct bytes of default memory plus 64*3*FLOAT +
// (4+FLOAT)*WIDTH + 4 bytes of write-combined memory, plus WIDTH source
// blocks of 64*3*FLOAT + 8 bytes.
nf_status nf::sic_limits(int out_kind, int cpd, uint64_t max_buffer_bytes, nf_gpu_limits *lim) {
    const float acc_bytes = out_kind == NF_OUT_FLOAT4 ? 16.f : 12.f;
    float src_wc = sizeof(float) * 3 * NFBLOCK + 8.0f;
    float sink_wc = sizeof(float) * 3 * NFBLOCK + (4.0f + sizeof(float)) * REF_WIDTH + 4.0f;
    float sink_def = acc_bytes * NFBLOCK;
    float total = sink_def + sink_wc + REF_WIDTH * src_wc;
    double blocks = ((double)max_buffer_bytes - 1e5) / total;
    if (!(blocks >= 1.0) || blocks > (double)INT32_MAX / REF_WIDTH) {
        set_error("nf_gpu_setup: buffer budget out of range");
        return NF_EINVAL;
    }
    lim->max_sink_blocks = (int)blocks;
    lim->max_source_blocks = REF_WIDTH * lim->max_sink_blocks;
    lim->max_sink_size = (size_t)NFBLOCK * lim->max_sink_blocks;
    lim->max_source_size = (size_t)NFBLOCK * lim->max_source_blocks;
    lim->max_nsink = lim->max_sink_blocks;
    lim->max_nsource = lim->max_nsink;
    if (lim->max_nsink <= 2 * cpd || lim->max_nsource <= (2 + REF_WIDTH) * cpd) {
        set_error("nf_gpu_setup: MaxNSink too small for this cpd (GPUControl.cu:407-408)");
        return NF_EINVAL;
    }
    return NF_OK;
}

extern "C" nf_status nf_gpu_setup(nf_ctx *ctx, int cpd, uint64_t max_buffer_bytes, int ngpu,
                                  int buffers_per_device, int use_pinned, nf_gpu_limits *limits) {
    if (!ctx || !limits || ngpu < 1 || buffers_per_device < 1 || cpd < 1) {
        set_error("nf_gpu_setup: bad argument");
        return NF_EINVAL;
    }
    if (ctx->sic) {  // GPUSetup runs once (GPUControl.cu:364)
        *limits = ctx->sic->limits;
        return NF_OK;
    }
    int ndev = 0;
    nf_status st = nf_get_ngpu(&ndev);
    if (st != NF_OK) return st;
    if (ngpu > ndev) {
        set_error("nf_gpu_setup: more GPUs requested than present");
        return NF_EINVAL;
    }
    nf_gpu_limits lim{};
    st = sic_limits(ctx->cfg.out_kind, cpd, max_buffer_bytes, &lim);
    if (st != NF_OK) return st;
    auto *S = new nf_ctx::Sic;
    S->limits = lim;
    S->cpd = cpd;
    // UsePinnedGPUMemory < 0: pin when the problem is large (GPUControl.cu:431-432)
    bool pinned = use_pinned < 0 ? lim.max_sink_blocks >= 10000 : use_pinned != 0;
    ctx->sic = S;
    for (int g = 0; g < ngpu * buffers_per_device; g++) {
        auto b = std::make_unique<SicBuffer>();
        b->index = g;
        b->device = ngpu == 1 ? ctx->device : g % ngpu;
        b->pinned = pinned;
        cudaError_t e = cudaSetDevice(b->device);
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaEventCreate(&b->ev0);
        if (e == cudaSuccess) e = cudaEventCreate(&b->ev1);
        if (e != cudaSuccess) {
            nf_status s2 = cuda_fail(e, "nf_gpu_setup");
            S->buffers.push_back(std::move(b));
            nf_sic_shutdown(ctx);
            return s2;
        }
        S->buffers.push_back(std::move(b));
    }
    for (auto &b : S->buffers) S->workers.emplace_back(worker_main, ctx, b.get());
    cudaSetDevice(ctx->device);
    *limits = lim;
    return NF_OK;
}

extern "C" nf_status nf_gpu_reset(nf_ctx *ctx) {
    if (!ctx) {
        set_error("nf_gpu_reset: null context");
        return NF_EINVAL;
    }
    nf_sic_shutdown(ctx);
    return NF_OK;
}

extern "C" nf_status nf_sic_execute(nf_ctx *ctx, const nf_sic_desc *sic, int jlow, int jhigh,
                                    int blocking, volatile int *completion) {
    if (!ctx || !sic || !completion) {
        set_error("nf_sic_execute: null argument");
        return NF_EINVAL;
    }
    if (!ctx->sic) {
        set_error("nf_sic_execute: nf_gpu_setup has not run");
        return NF_EINVAL;
    }
    nf_status st = check_desc(ctx, *sic, jlow, jhigh);
    if (st != NF_OK) return st;
    SicTask t;
    t.d = *sic;
    t.jlow = jlow;
    t.jhigh = jhigh;
    t.completion = completion;
    *completion = 0;
    if (blocking) {  // GPUExecute(blocking=1) runs on the caller's thread, buffer 0
        SicBuffer &b = *ctx->sic->buffers[0];
        {
            std::lock_guard<std::mutex> bl(b.mu);
            st = run_task(ctx, b, t);
        }
        finish(ctx, t, st);
        cudaSetDevice(ctx->device);
        return st;
    }
    {
        std::lock_guard<std::mutex> lk(ctx->sic->mu);
        ctx->sic->queue.push_back(t);
    }
    ctx->sic->cv.notify_one();
    return NF_OK;
}

extern "C" nf_status nf_sic_drain(nf_ctx *ctx, uint64_t timeout_ns) {
    if (!ctx) {
        set_error("nf_sic_drain: null context");
        return NF_EINVAL;
    }
    if (!ctx->sic) return NF_OK;
    auto *S = ctx->sic;
    std::unique_lock<std::mutex> lk(S->mu);
    bool ok = S->idle.wait_for(lk, std::chrono::nanoseconds(timeout_ns),
                               [&] { return S->queue.empty() && S->active == 0; });
    if (!ok) {
        set_error("nf_sic_drain: SICs still in flight at the timeout");
        return NF_ETIMEDOUT;
    }
    if (!S->error.empty()) {
        set_error(S->error);
        S->error.clear();
        return NF_EDEVICE;
    }
    return NF_OK;
}

extern "C" nf_status nf_sic_timing(nf_ctx *ctx, double *kernel_ms, uint64_t *sics,
                                   uint64_t *pairs, int reset) {
    if (!ctx) {
        set_error("nf_sic_timing: null context");
        return NF_EINVAL;
    }
    double ms = 0.0;
    uint64_t n = 0, p = 0;
    if (ctx->sic) {
        std::lock_guard<std::mutex> lk(ctx->sic->mu);
        ms = ctx->sic->kernel_ms;
        n = ctx->sic->sics;
        p = ctx->sic->pairs;
        if (reset) {
            ctx->sic->kernel_ms = 0.0;
            ctx->sic->sics = ctx->sic->pairs = 0;
        }
    }
    if (kernel_ms) *kernel_ms = ms;
    if (sics) *sics = n;
    if (pairs) *pairs = p;
    return NF_OK;
}
