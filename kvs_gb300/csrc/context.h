// context.h -- host-side state of libkvsmc shared by api.cu and batch.cu.
#pragma once
#include <atomic>
#include <cstdint>
#include <functional>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/kvsmc.h"
#include "mc_internal.h"

struct kvsmc_volume {
    kvsmc::VolumeView view;
    void* dev = nullptr;        // owned device allocation
    size_t bytes = 0;
    cudaEvent_t ev = nullptr;   // comes with dev: behind the last copy or pass that a call left running on it
    bool ev_own = true;         // ev stands on the owner's own stream, or on none
    int device = 0;             // the device it lies on
    kvsmc_context* owner = nullptr;   // the context that allocated it
    // read or written by work that no call of the owner's waits for (a plan's
    // replays, a captured update's, a server's workers, another context): its block
    // is not kept when it is freed
    std::atomic<bool> lent{false};
    bool has_minmax = false;
    double vmin = 0.0, vmax = 0.0;
    // parts of the same allocation: the brick min/max table (the streaming
    // kernels' empty-space skip; null for volumes that they do not take), written
    // by the pass that every copy into such a volume ends with, and the values'
    // range, where that pass has run (range_ready); otherwise the range is taken
    // when it is first asked for, into the asking context's memory
    kvsmc::IngestOut* range = nullptr;
    bool range_ready = false;
    float2* bricks = nullptr;
    bool bricks_valid = false;
};

struct kvsmc_context {
    int device = 0;
    int num_sms = 0;
    cudaStream_t own_stream = nullptr;
    cudaStream_t stream = nullptr;
    void* scratch = nullptr;     // grow-only device arena for per-call intermediates
    size_t scratch_bytes = 0;
    void* out_arena = nullptr;   // grow-only device outputs of the host call
    void* arena2 = nullptr;      // grow-only second arena (vertex normals' triangle lists)
    size_t arena2_bytes = 0;
    void* arena3 = nullptr;      // grow-only third arena (a batch's shared streaming count)
    size_t arena3_bytes = 0;
    void* arena4 = nullptr;      // grow-only fourth arena (grouped shared-vertex requests' count arrays)
    size_t arena4_bytes = 0;
    void* arena5 = nullptr;      // grow-only fifth arena (their per-triangle normals)
    size_t arena5_bytes = 0;
    size_t out_bytes = 0;
    kvsmc_volume* host_vol = nullptr;  // staging volume of the host call
    uint64_t* h_small = nullptr; // pinned: small read-backs (totals, min/max, status)
    void* h_stage = nullptr;     // pinned: staging of work tables sent to the device
    size_t h_stage_bytes = 0;
    uint64_t launches = 0;
    int path = 0;                // 0: streaming kernels where eligible, 1: gather kernels only
    // plane-wait poll limits of the streaming count / emit kernels (kvsmc_set_wait_limit)
    uint32_t wait_polls[2] = {kvsmc::kStreamWaitPolls, kvsmc::kStreamWaitPolls};
    uint64_t list_limit = ~0ull;   // entries that a pair list may have (kvsmc_set_list_limit)
    kvsmc::Profiler* prof = nullptr;
    // freed volumes' device blocks, kept for the next volumes (cudaMalloc and
    // cudaFree of a new field's 83 MB a frame cost 350 us): at most
    // kSpareBlocks blocks of kSpareBytes in all, given back when an
    // allocation fails and with the context
    struct Spare { void* p; size_t bytes; cudaEvent_t ev; };
    std::vector<Spare> spare;
    std::mutex spare_mutex;
    void* dense = nullptr;       // staging of host volumes whose rows are padded (at most kDenseStage)
    size_t dense_bytes = 0;
    // the last pass that reads it: on own_stream, or behind dense_ev
    bool dense_own = true;
    cudaEvent_t dense_ev = nullptr;
    std::vector<kvsmc::KernelFit> fits;   // launch shapes of the kernels launched so far
    std::string last_error;
    // auxiliary streams for launches that may run side by side (created on first use)
    static constexpr int kAux = 6;
    cudaStream_t aux[kAux] = {};
    cudaEvent_t fork_ev = nullptr;
    cudaEvent_t join_ev[kAux] = {};
    bool aux_ready = false;
    // copy stream of the host calls: results leave while later parts are
    // written (created on first use), one event per emit part
    cudaStream_t copy_stream = nullptr;
    static constexpr int kParts = 16;
    cudaEvent_t part_ev[kParts] = {};
    int* d_flag = nullptr;       // device word for checks of export calls (created on first use)
    int* h_flag = nullptr;       // pinned copy of it
    // export staging: two device record buffers, two pinned host buffers (grow-only)
    uint8_t* stl_dbuf[2] = {};
    uint8_t* stl_hbuf[2] = {};
    size_t stl_buf_bytes = 0;
    cudaEvent_t stl_ev[2] = {};
    // ASCII text of the STL writer: two device, two pinned buffers (grow-only)
    char* txt_dbuf[2] = {};
    char* txt_hbuf[2] = {};
    size_t txt_bytes = 0;
    // streaming launch shapes: the tuning table, or one forced shape
    std::vector<kvsmc_tune_entry> tuning;
    bool tune_forced = false;
    kvsmc_tune_choice tune_force{};
};

namespace kvsmc {
Profiler* profiler_create();
void profiler_destroy(Profiler* p);
}  // namespace kvsmc

namespace kvsmc_host {

kvsmc_status fail(kvsmc_context* ctx, kvsmc_status st, const char* fmt, ...);
inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }
inline kvsmc::Launch launch_of(kvsmc_context* ctx)
{
    kvsmc::Launch L{ctx->stream, ctx->num_sms, &ctx->launches, ctx->prof};
    L.wait_polls[0] = ctx->wait_polls[0];
    L.wait_polls[1] = ctx->wait_polls[1];
    L.fits = &ctx->fits;
    return L;
}
kvsmc_status ensure_scratch(kvsmc_context* ctx, size_t bytes);
kvsmc_status ensure_stage(kvsmc_context* ctx, size_t bytes);
kvsmc_status volume_minmax(kvsmc_context* ctx, kvsmc_volume* v);
bool equal_ref(double a, double b);
kvsmc::Classifier make_classifier(double iso);
void narrow_thresholds(double iso, float& f_thr, long long& i_thr);

// Bump allocator over an arena (256-byte aligned pieces).
struct Carve {
    char* base;
    size_t off = 0;
    template <typename P> P* take(size_t bytes)
    {
        P* p = reinterpret_cast<P*>(base + off);
        off = align_up(off + bytes, 256);
        return p;
    }
};

// One request of a batch after host-side planning.
struct Item {
    kvsmc_volume* vol = nullptr;
    kvsmc_params params{};
    double vmin = 0, vmax = 0;
    bool extracted = true;
    float* d_coords = nullptr;
    uint64_t coords_cap = 0;
    float* d_normals = nullptr;
    uint64_t normals_cap = 0;
    uint32_t* d_conn = nullptr;
    uint64_t conn_cap = 0;
    bool emit = false;           // write outputs (false: count only)
    void* h_coords = nullptr;    // host outputs from the allocator (host calls)
    void* h_normals = nullptr;
    void* h_conn = nullptr;
    kvsmc_sizes sizes{};
    kvsmc_status status = KVSMC_OK;
};

// A volume's device block: from the context's spare blocks, or a new one.
constexpr size_t kSpareBytes = (size_t)1 << 30;
constexpr size_t kSpareBlocks = 4;
kvsmc_status block_alloc(kvsmc_context* ctx, size_t bytes, kvsmc_volume* v);
// Give a volume's block back: kept for the next volumes of ctx once nothing
// reads it any more, or freed (ctx null, lent, or too large).
void block_free(kvsmc_context* ctx, kvsmc_volume* v);
// A call of ctx reads the volume.
inline void volume_use(const kvsmc_context* ctx, kvsmc_volume* v)
{
    if (v->owner != ctx) v->lent = true;
}
// Free every spare block (whether there were any).
bool block_release(kvsmc_context* ctx);

// cudaMalloc that frees the spare blocks before it gives up.
cudaError_t device_malloc_bytes(kvsmc_context* ctx, void** p, size_t bytes);
template <typename P> cudaError_t device_malloc(kvsmc_context* ctx, P** p, size_t bytes)
{
    void* q = nullptr;
    const cudaError_t e = device_malloc_bytes(ctx, &q, bytes);
    *p = static_cast<P*>(q);
    return e;
}

// Shape a volume and its allocation (kept when large enough).
kvsmc_status volume_alloc(kvsmc_context* ctx, kvsmc_dtype dtype, uint32_t nx, uint32_t ny, uint32_t nz,
                          kvsmc_volume* v);
// Dense values into the volume's layout, with its brick table and range.
constexpr size_t kDenseStage = (size_t)64 << 20;
constexpr size_t kStageRow = 8192;   // bytes of a row up to which volumes without a table are staged
kvsmc_status volume_copy_in(kvsmc_context* ctx, kvsmc_volume* v, const void* src, bool on_device);
void volume_destroy(kvsmc_context* ctx, kvsmc_volume* v);

// A resident volume of the given shape with uninitialised values (row-padded
// like the uploads); the caller fills it and then calls volume_bricks.
kvsmc_status volume_create(kvsmc_context* ctx, kvsmc_dtype dtype, uint32_t nx, uint32_t ny, uint32_t nz,
                           kvsmc_volume** out);

// The values that a caller wrote into a volume on the context's stream are all
// enqueued: its brick min/max table, if it has one, and with it its range.
kvsmc_status volume_bricks(kvsmc_context* ctx, kvsmc_volume* v);

// Run fn(i, stream) for i < n side by side on the context's auxiliary streams,
// forked from and joined back into `origin` (also inside a stream capture).
cudaError_t fan_out(kvsmc_context* ctx, cudaStream_t origin, size_t n,
                    const std::function<cudaError_t(size_t, cudaStream_t)>& fn);

// Decide min/max (MapperBase::setRange, the volume's cache or a preset) and
// the Math::Equal early exit; fills it.vmin/vmax/extracted and clears sizes.
kvsmc_status prepare(kvsmc_context* ctx, Item& it);

// The streaming launch shape for a volume under the context's tuning (zero
// fields resolved by the built-in rules).
kvsmc_tune_choice stream_shape(const kvsmc_context* ctx, const kvsmc::VolumeView& v);

// Requests the streaming kernels can take (duplicated mode, 8/16-bit and
// float32 data, finite isolevel, width <= 4096 cells).
bool stream_eligible(const kvsmc_context* ctx, const Item& it);
// The same volume and isolevel conditions, whatever the mode (the streaming
// count of a shared-vertex request).
bool stream_volume_eligible(const kvsmc_context* ctx, const Item& it);
// The same for all ten value types: the 32/64-bit integer and double volumes
// take the streaming layout too, one isolevel per pass (mc_wide.cu).  (Plans
// and the server take the narrow types only.)
bool any_stream_eligible(const kvsmc_context* ctx, const Item& it);
bool dup_stream_eligible(const kvsmc_context* ctx, const Item& it);
// Whether a count alone (nothing is emitted) goes by cells through the gather
// kernels.  8/16-bit and float32 volumes: a shared-vertex request that is counted
// by itself, where the streaming count, whose time is its crossed pairs' with
// vertices, is slower on smooth and crowded volumes alike (us by cells / smooth /
// every cell crossed, float32: 17 x 500 x 500 165 / 196 / 329, 129^3 54 / 71 / 84,
// 200^3 81 / 91 / 139; smaller ones 17 x 100 x 100 96 / 60 / 72, larger ones 201 x
// 300 x 300 142 / 116 / 228).  32/64-bit integers and doubles, with `together` the
// call's duplicated-mode requests on such volumes: the streaming count costs 48 us
// before it reads anything, 34 by cells, and its vertices a pass of their own;
// it reads a volume once and counts several requests in one launch.  Measured
// (us by cells / streaming): 128^3 doubles 48 / 63, 200^3 95 / 82, 512^3 927 /
// 475; 128^3 32-bit 46 / 54, 200^3 70 / 65; 64-bit integers 46 / 63 and at 512^3
// 446 / 450; two requests at 128^3 85 / 65; with vertices 128^3 67 / 106 and
// 55 / 88, 300^3 372 / 378, 420^3 928 / 723 (64-bit integers 773 / 807 at 512^3).
// Rows of few cells leave most lanes idle: 17 x 400 x 400 doubles 107 / 165,
// 2 x 1000 x 1000 406 / 717.  Several requests on them are one launch all the
// same, and one of them takes 0.7 us a thousand rows there, by cells 30 us and
// more the shorter the rows: of 16 requests one takes (doubles) 33 x 100 x 100
// 51 / 11, 33 x 300 x 300 64 / 64, 33 x 500 x 500 112 / 167, 2 x 300 x 300 123 /
// 63, 2 x 500 x 500 186 / 165; 32-bit 2 x 500 x 500 165 / 83, 3 x 700 x 900 236 / 227.
bool count_by_cells(const kvsmc::VolumeView& v, int mode, size_t together);
// Count (and, for items with emit set, emit) all eligible items together.
kvsmc_status stream_run(kvsmc_context* ctx, std::vector<Item*>& items);

}  // namespace kvsmc_host

#define KVSMC_CUDA(ctx, call)                                                                              \
    do {                                                                                                   \
        cudaError_t e_ = (call);                                                                           \
        if (e_ != cudaSuccess)                                                                             \
            return kvsmc_host::fail(ctx, e_ == cudaErrorMemoryAllocation ? KVSMC_ERR_OUT_OF_MEMORY         \
                                                                         : KVSMC_ERR_CUDA,                 \
                                    "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
    } while (0)
