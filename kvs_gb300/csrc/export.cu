// export.cu -- binary STL serialisation of a device triangle mesh.
//
// The records are what kvs::PolygonExporter<kvs::Stl>::exec
// (Source/Core/Visualization/Exporter/PolygonExporter.cpp:78-176) and
// kvs::Stl::write_binary (Source/Core/FileFormat/STL/Stl.cpp:490-540) write:
// per triangle its normal (3 floats), its three vertices (9 floats) and two
// zero bytes, 50 bytes, little-endian, after an 84-byte header (80 bytes
// "Generated by KVS" zero-padded, the uint32 triangle count).  Shared-vertex
// meshes are expanded through their connections; with vertex normals the
// triangle's normal is (n0 + n1 + n2) / 3 in float, in that order
// (PolygonExporter.cpp:133-152, kvs::Vector3 operator+ and operator/).
//
// A warp's work is a tile of 64 consecutive triangles, two per lane: their
// records are 100 bytes, 25 whole words, so they are composed from registers
// with 25 word stores at an odd stride, free of bank conflicts, and a tile's
// 3,200 bytes leave by one bulk shared-to-global copy.  Duplicated meshes with
// 16-byte aligned arrays arrive through a ring of two tiles a warp (TMA bulk
// copies, mbarrier completion): 16 warps an SM keep 98 KB in flight and none
// waits for another.  Shared-vertex meshes (gathers through the connections),
// unaligned arrays and the last partial tile load straight into registers.
// Bound by HBM: 48 bytes read and 50 written per triangle of a duplicated
// mesh.  4,000,037 triangles: 75.6 us with CTA-wide tiles of
// 256 and half-word stores, 68.6 us, 86% of the copy rate (three or four tiles
// a ring: 68.6 to 69.6); 661 triangles, in one launch: 30 -> 18 us a call.
#include <cstdio>
#include <cstring>
#include <vector>

#include "context.h"
#include "tma.cuh"

namespace kvsmc {

namespace {

constexpr uint32_t kStlTile = 64;   // triangles
constexpr uint32_t kStlRecord = 50;
constexpr uint32_t kStlPollLimit = 1u << 22;
constexpr unsigned FULL = 0xffffffffu;

constexpr int kStlStages = 2;
constexpr int kStlThreads = 256;

// Warp shared memory: composed records of two tiles and, for bulk loads, the
// ring of input tiles.
struct alignas(16) StlOut {
    uint32_t rec[2][kStlTile * kStlRecord / 4];
};
struct alignas(16) StlIn {
    float c[kStlStages][kStlTile * 9];
    float n[kStlStages][kStlTile * 3];
    uint64_t bar[kStlStages];
};

// Two triangles' 24 floats (each 3 of the normal, 9 of the corners) as 25
// record words: the first record's 48 bytes and two zero bytes, the second's
// shifted by half a word.
__device__ __forceinline__ void stl_compose(uint32_t* r, const float* f)
{
    uint32_t before = 0;
#pragma unroll
    for (int i = 0; i < 12; ++i) r[i] = __float_as_uint(f[i]);
#pragma unroll
    for (int i = 0; i < 12; ++i) {
        const uint32_t w = __float_as_uint(f[12 + i]);
        r[12 + i] = __funnelshift_l(before, w, 16);
        before = w;
    }
    r[24] = before >> 16;
}

// The lane's two triangles (t, t + 1; those below ntri) straight from memory.
template <int MODE>
__device__ __forceinline__ void stl_load(const float* __restrict__ coords, const float* __restrict__ normals,
                                         const uint32_t* __restrict__ conn, uint64_t nverts, uint64_t t, uint64_t ntri,
                                         int* bad_index, float* f)
{
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        float* g = f + 12 * h;
        const uint64_t tri = t + h;
        if (tri >= ntri) {
#pragma unroll
            for (int k = 0; k < 12; ++k) g[k] = 0.0f;
            continue;
        }
        if (MODE != KVSMC_SHARED_VERTEX_NORMAL) {
#pragma unroll
            for (int k = 0; k < 3; ++k) g[k] = __ldg(normals + 3 * tri + k);
        }
        if (MODE == KVSMC_DUP_POLYGON_NORMAL) {
#pragma unroll
            for (int k = 0; k < 9; ++k) g[3 + k] = __ldg(coords + 9 * tri + k);
            continue;
        }
        uint64_t v[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            v[k] = __ldg(conn + 3 * tri + k);
            if (v[k] >= nverts) {
                atomicExch(bad_index, 1);
                v[k] = 0;
            }
        }
#pragma unroll
        for (int k = 0; k < 9; ++k) g[3 + k] = __ldg(coords + 3 * v[k / 3] + k % 3);
        if (MODE == KVSMC_SHARED_VERTEX_NORMAL) {
            // ( normal0 + normal1 + normal2 ) / 3.0f, component by component
#pragma unroll
            for (int k = 0; k < 3; ++k)
                g[k] = __fdiv_rn(__fadd_rn(__fadd_rn(__ldg(normals + 3 * v[0] + k), __ldg(normals + 3 * v[1] + k)),
                                           __ldg(normals + 3 * v[2] + k)), 3.0f);
        }
    }
}

// Compose a tile's records in `rec` (no bulk store reads it any more) and
// send them: a whole tile by one bulk store of lane 0, a partial one by the
// lanes.  dst is 16-byte aligned.
__device__ __forceinline__ void stl_send(uint32_t* rec, const float* f, uint8_t* dst, uint32_t ntris, unsigned lane)
{
    stl_compose(rec + 25 * lane, f);
    if (ntris == kStlTile) {
        fence_proxy_async();   // the records, written by this thread, are read by the async proxy
        __syncwarp();
        if (lane == 0) {
            bulk_copy_s2g(dst, rec, kStlTile * kStlRecord);
            bulk_commit();
        }
        return;
    }
    __syncwarp();
    const uint32_t bytes = kStlRecord * ntris;
    for (uint32_t i = lane; i < bytes / 16; i += 32)
        reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(rec)[i];
    for (uint32_t i = bytes / 16 * 8 + lane; i < bytes / 2; i += 32)
        reinterpret_cast<uint16_t*>(dst)[i] = reinterpret_cast<const uint16_t*>(rec)[i];
    __syncwarp();
}

template <int MODE>
__global__ void __launch_bounds__(kStlThreads)
    k_stl_direct(const float* __restrict__ coords, const float* __restrict__ normals,
                 const uint32_t* __restrict__ conn, uint64_t nverts, uint64_t ntri, uint8_t* __restrict__ out,
                 int* __restrict__ bad_index)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    StlOut& O = reinterpret_cast<StlOut*>(smem_raw)[warp];
    const uint64_t tiles = (ntri + kStlTile - 1) / kStlTile, warps = (uint64_t)gridDim.x * (kStlThreads / 32);
    uint32_t b = 0;
    for (uint64_t tile = (uint64_t)blockIdx.x * (kStlThreads / 32) + warp; tile < tiles; tile += warps, b ^= 1u) {
        const uint64_t t0 = tile * kStlTile;
        float f[24];
        stl_load<MODE>(coords, normals, conn, nverts, t0 + 2 * lane, ntri, bad_index, f);
        if (lane == 0) bulk_wait_read<1>();   // rec[b] was sent two tiles ago
        __syncwarp();
        stl_send(O.rec[b], f, out + kStlRecord * t0, (uint32_t)(ntri - t0 < kStlTile ? ntri - t0 : kStlTile), lane);
    }
    if (lane == 0) bulk_wait<0>();
}

// A duplicated mesh; coords, normals, out 16-byte aligned.  status: set to 2
// when a load did not complete within the poll limit (the warp then drains its
// own copies and stops).
__global__ void __launch_bounds__(kStlThreads)
    k_stl_ring(const float* __restrict__ coords, const float* __restrict__ normals, uint64_t ntri,
               uint8_t* __restrict__ out, int* __restrict__ status)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr int kWarps = kStlThreads / 32;
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    StlIn& I = reinterpret_cast<StlIn*>(smem_raw)[warp];
    StlOut& O = reinterpret_cast<StlOut*>(smem_raw + kWarps * sizeof(StlIn))[warp];
    const uint64_t full = ntri / kStlTile, warps = (uint64_t)gridDim.x * kWarps;
    const uint64_t first = (uint64_t)blockIdx.x * kWarps + warp;
    auto issue = [&](uint64_t tile, int s) {
        mbar_arrive_expect_tx(&I.bar[s], kStlTile * 12 * sizeof(float));
        bulk_copy_g2s(I.c[s], coords + kStlTile * 9 * tile, kStlTile * 9 * sizeof(float), &I.bar[s]);
        bulk_copy_g2s(I.n[s], normals + kStlTile * 3 * tile, kStlTile * 3 * sizeof(float), &I.bar[s]);
    };
    if (lane == 0) {
        for (int s = 0; s < kStlStages; ++s) mbar_init(&I.bar[s], 1);
        fence_barrier_init();
        for (int s = 0; s < kStlStages; ++s)
            if (first + s * warps < full) issue(first + s * warps, s);
    }
    __syncwarp();
    uint32_t ph = 0, pending = 0;   // per stage: parity of its next completion; a load is in flight
    for (int s = 0; s < kStlStages; ++s)
        if (first + s * warps < full) pending |= 1u << s;
    int s = 0;
    uint32_t b = 0;
    for (uint64_t tile = first; tile < full; tile += warps) {
        const bool ok = mbar_wait(&I.bar[s], (ph >> s) & 1u, kStlPollLimit);
        if (!__all_sync(FULL, ok)) {
            if (lane == 0) atomicExch(status, 2);
            break;
        }
        ph ^= 1u << s;
        pending &= ~(1u << s);
        float f[24];
        const float2* c2 = reinterpret_cast<const float2*>(I.c[s] + 18 * lane);
        const float2* n2 = reinterpret_cast<const float2*>(I.n[s] + 6 * lane);
        float c[18], n[6];
#pragma unroll
        for (int k = 0; k < 9; ++k) { c[2 * k] = c2[k].x; c[2 * k + 1] = c2[k].y; }
#pragma unroll
        for (int k = 0; k < 3; ++k) { n[2 * k] = n2[k].x; n[2 * k + 1] = n2[k].y; }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int k = 0; k < 3; ++k) f[12 * h + k] = n[3 * h + k];
#pragma unroll
            for (int k = 0; k < 9; ++k) f[12 * h + 3 + k] = c[9 * h + k];
        }
        __syncwarp();   // the stage is read
        const uint64_t next = tile + kStlStages * warps;
        if (next < full) {
            if (lane == 0) {
                fence_proxy_async();
                issue(next, s);
            }
            pending |= 1u << s;
        }
        if (lane == 0) bulk_wait_read<1>();   // rec[b] was sent two tiles ago
        __syncwarp();
        stl_send(O.rec[b], f, out + kStlTile * kStlRecord * tile, kStlTile, lane);
        b ^= 1u;
        s = s + 1 < kStlStages ? s + 1 : 0;
    }
    if (full * kStlTile < ntri && full % warps == first) {   // the last partial tile
        float f[24];
        stl_load<KVSMC_DUP_POLYGON_NORMAL>(coords, normals, nullptr, 0, full * kStlTile + 2 * lane, ntri, status, f);
        if (lane == 0) bulk_wait_read<0>();
        __syncwarp();
        stl_send(O.rec[0], f, out + kStlTile * kStlRecord * full, (uint32_t)(ntri - full * kStlTile), lane);
    }
    if (lane == 0) {
        // after a timeout: the loads still in flight land (bounded) before the warp leaves
        for (int q = 0; q < kStlStages; ++q)
            if ((pending >> q) & 1u) mbar_wait(&I.bar[q], (ph >> q) & 1u, kStlPollLimit);
        bulk_wait<0>();
    }
}

}  // namespace

// out is 16-byte aligned.
cudaError_t launch_stl_records(const float* coords, const float* normals, const uint32_t* conn, uint64_t nverts,
                               uint64_t ntri, int mode, uint8_t* out, int* bad_index, const Launch& L)
{
    if (ntri == 0) return cudaSuccess;
    if (reinterpret_cast<uintptr_t>(out) & 15u) return cudaErrorInvalidValue;
    const bool ring = mode == KVSMC_DUP_POLYGON_NORMAL &&
                      ((reinterpret_cast<uintptr_t>(coords) | reinterpret_cast<uintptr_t>(normals)) & 15u) == 0;
    const void* kern = ring ? reinterpret_cast<const void*>(k_stl_ring)
                     : mode == KVSMC_DUP_POLYGON_NORMAL
                         ? reinterpret_cast<const void*>(k_stl_direct<KVSMC_DUP_POLYGON_NORMAL>)
                     : mode == KVSMC_SHARED_POLYGON_NORMAL
                         ? reinterpret_cast<const void*>(k_stl_direct<KVSMC_SHARED_POLYGON_NORMAL>)
                         : reinterpret_cast<const void*>(k_stl_direct<KVSMC_SHARED_VERTEX_NORMAL>);
    constexpr int warps = kStlThreads / 32;
    const size_t smem = warps * (sizeof(StlOut) + (ring ? sizeof(StlIn) : 0));
    int per_sm = 0;
    cudaError_t e = kernel_fit(L, kern, kStlThreads, smem, &per_sm, true);
    if (e != cudaSuccess) return e;
    const uint64_t tiles = (ntri + kStlTile - 1) / kStlTile, need = (tiles + warps - 1) / warps;
    const uint64_t resident = (uint64_t)(per_sm > 0 ? per_sm : 1) * (uint64_t)L.num_sms;
    void* direct[] = {&coords, &normals, &conn, &nverts, &ntri, &out, &bad_index};
    void* tma[] = {&coords, &normals, &ntri, &out, &bad_index};
    prof_begin(L, "stl_records");
    e = cudaLaunchKernel(kern, dim3((unsigned)(need < resident ? need : resident)), dim3(kStlThreads),
                         ring ? tma : direct, smem, L.stream);
    prof_end(L);
    *L.counter += 1;
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace kvsmc

namespace {

using kvsmc_host::fail;

kvsmc_status check_mesh(kvsmc_context* ctx, int32_t mode, const float* d_coords, const float* d_normals,
                        const uint32_t* d_connections, uint64_t ntriangles)
{
    if (mode != KVSMC_DUP_POLYGON_NORMAL && mode != KVSMC_SHARED_POLYGON_NORMAL && mode != KVSMC_SHARED_VERTEX_NORMAL)
        return fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "stl: bad mode %d", (int)mode);
    if (ntriangles && (!d_coords || !d_normals || (mode != KVSMC_DUP_POLYGON_NORMAL && !d_connections)))
        return fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "stl: null mesh array");
    return KVSMC_OK;
}

}  // namespace

extern "C" {

kvsmc_status kvsmc_stl_records(kvsmc_context* ctx, int32_t mode, const float* d_coords, const float* d_normals,
                               const uint32_t* d_connections, uint64_t nvertices, uint64_t ntriangles, void* d_out)
{
    if (!ctx) return KVSMC_ERR_INVALID_ARGUMENT;
    kvsmc_status st = check_mesh(ctx, mode, d_coords, d_normals, d_connections, ntriangles);
    if (st) return st;
    if (ntriangles == 0) return KVSMC_OK;
    if (!d_out || (reinterpret_cast<uintptr_t>(d_out) & 15u))
        return fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "stl: output must be 16-byte aligned device memory");
    KVSMC_CUDA(ctx, cudaSetDevice(ctx->device));
    if (!ctx->d_flag) KVSMC_CUDA(ctx, kvsmc_host::device_malloc(ctx, &ctx->d_flag, sizeof(int)));
    int* bad = ctx->d_flag;
    KVSMC_CUDA(ctx, cudaMemsetAsync(bad, 0, sizeof(int), ctx->stream));
    KVSMC_CUDA(ctx, kvsmc::launch_stl_records(d_coords, d_normals, d_connections, nvertices, ntriangles, mode,
                                              static_cast<uint8_t*>(d_out), bad, kvsmc_host::launch_of(ctx)));
    KVSMC_CUDA(ctx, cudaMemcpyAsync(ctx->h_small, bad, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    KVSMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    int h_bad = 0;
    std::memcpy(&h_bad, ctx->h_small, sizeof(int));
    if (h_bad == 2) return fail(ctx, KVSMC_ERR_TIMEOUT, "stl: a shared-memory load did not complete");
    if (h_bad) return fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "stl: a connection index is >= nvertices");
    return KVSMC_OK;
}

kvsmc_status kvsmc_write_stl(kvsmc_context* ctx, const char* path, int32_t mode, const float* d_coords,
                             const float* d_normals, const uint32_t* d_connections, uint64_t nvertices,
                             uint64_t ntriangles)
{
    if (!ctx || !path) return KVSMC_ERR_INVALID_ARGUMENT;
    kvsmc_status st = check_mesh(ctx, mode, d_coords, d_normals, d_connections, ntriangles);
    if (st) return st;
    if (ntriangles > 0xffffffffull)
        return fail(ctx, KVSMC_ERR_TOO_LARGE, "stl: %llu triangles do not fit the format's 32-bit count",
                    (unsigned long long)ntriangles);
    KVSMC_CUDA(ctx, cudaSetDevice(ctx->device));
    // chunks of 2^20 triangles, double-buffered through the context's staging
    // buffers: chunk i is serialised and copied while chunk i - 1 is written
    const uint64_t chunk = 1ull << 20;
    const uint64_t nchunks = (ntriangles + chunk - 1) / chunk;
    if (nchunks) {
        const size_t bytes = (size_t)(ntriangles < chunk ? ntriangles : chunk) * kvsmc::kStlRecordBytes;
        if (bytes > ctx->stl_buf_bytes) {
            KVSMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
            for (int b = 0; b < 2; ++b) {
                if (ctx->stl_dbuf[b]) cudaFree(ctx->stl_dbuf[b]);
                if (ctx->stl_hbuf[b]) cudaFreeHost(ctx->stl_hbuf[b]);
                ctx->stl_dbuf[b] = nullptr;
                ctx->stl_hbuf[b] = nullptr;
            }
            ctx->stl_buf_bytes = 0;
            for (int b = 0; b < 2; ++b) {
                KVSMC_CUDA(ctx, kvsmc_host::device_malloc(ctx, &ctx->stl_dbuf[b], bytes));
                KVSMC_CUDA(ctx, cudaMallocHost(&ctx->stl_hbuf[b], bytes));
                if (!ctx->stl_ev[b]) KVSMC_CUDA(ctx, cudaEventCreateWithFlags(&ctx->stl_ev[b], cudaEventDisableTiming));
            }
            ctx->stl_buf_bytes = bytes;
        }
        if (!ctx->d_flag) KVSMC_CUDA(ctx, kvsmc_host::device_malloc(ctx, &ctx->d_flag, sizeof(int)));
        if (!ctx->h_flag) KVSMC_CUDA(ctx, cudaMallocHost(&ctx->h_flag, sizeof(int)));
        KVSMC_CUDA(ctx, cudaMemsetAsync(ctx->d_flag, 0, sizeof(int), ctx->stream));
    }
    FILE* f = std::fopen(path, "wb");
    if (!f) return fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "stl: cannot open %s", path);
    char header[84];
    std::memset(header, 0, sizeof header);
    std::snprintf(header, 80, "Generated by KVS");
    const uint32_t count = (uint32_t)ntriangles;
    std::memcpy(header + 80, &count, 4);   // little-endian host (x86-64, aarch64)
    bool ok = std::fwrite(header, 1, 84, f) == 84;
    const kvsmc::Launch L = kvsmc_host::launch_of(ctx);
    auto chunk_tris = [&](uint64_t i) { return (i + 1) * chunk <= ntriangles ? chunk : ntriangles - i * chunk; };
    cudaError_t e = cudaSuccess;
    for (uint64_t i = 0; i <= nchunks && e == cudaSuccess && ok; ++i) {
        if (i < nchunks) {
            const int b = (int)(i & 1);
            const uint64_t t0 = i * chunk, nt = chunk_tris(i);
            const float* c = mode == KVSMC_DUP_POLYGON_NORMAL ? d_coords + 9 * t0 : d_coords;
            const float* nrm = mode == KVSMC_SHARED_VERTEX_NORMAL ? d_normals : d_normals + 3 * t0;
            const uint32_t* cn = mode == KVSMC_DUP_POLYGON_NORMAL ? nullptr : d_connections + 3 * t0;
            // the host buffer of this parity was written out before (chunk i - 2)
            e = kvsmc::launch_stl_records(c, nrm, cn, nvertices, nt, mode, ctx->stl_dbuf[b], ctx->d_flag, L);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(ctx->stl_hbuf[b], ctx->stl_dbuf[b], nt * kvsmc::kStlRecordBytes,
                                    cudaMemcpyDeviceToHost, ctx->stream);
            if (e == cudaSuccess) e = cudaEventRecord(ctx->stl_ev[b], ctx->stream);
        }
        if (i > 0 && e == cudaSuccess) {
            const int b = (int)((i - 1) & 1);
            e = cudaEventSynchronize(ctx->stl_ev[b]);
            if (e == cudaSuccess) {
                const size_t nb = chunk_tris(i - 1) * kvsmc::kStlRecordBytes;
                ok = std::fwrite(ctx->stl_hbuf[b], 1, nb, f) == nb;
            }
        }
    }
    int was_bad = 0;
    if (e == cudaSuccess && nchunks) {
        e = cudaMemcpyAsync(ctx->h_flag, ctx->d_flag, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (e == cudaSuccess) was_bad = *ctx->h_flag;
    }
    const bool closed = std::fclose(f) == 0;
    if (e != cudaSuccess) {
        cudaStreamSynchronize(ctx->stream);
        return fail(ctx, KVSMC_ERR_CUDA, "stl: %s", cudaGetErrorString(e));
    }
    if (!ok || !closed) {
        cudaStreamSynchronize(ctx->stream);
        return fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "stl: writing %s failed", path);
    }
    if (was_bad == 2) return fail(ctx, KVSMC_ERR_TIMEOUT, "stl: a shared-memory load did not complete");
    if (was_bad) return fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "stl: a connection index is >= nvertices");
    return KVSMC_OK;
}

kvsmc_status kvsmc_write_stl_host(kvsmc_context* ctx, const char* path, int32_t mode, const float* coords,
                                  uint64_t ncoords, const float* normals, uint64_t nnormals,
                                  const uint32_t* connections, uint64_t nconnections)
{
    if (!ctx || !path) return KVSMC_ERR_INVALID_ARGUMENT;
    if (mode != KVSMC_DUP_POLYGON_NORMAL && mode != KVSMC_SHARED_POLYGON_NORMAL && mode != KVSMC_SHARED_VERTEX_NORMAL)
        return fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "stl: bad mode %d", (int)mode);
    const bool dup = mode == KVSMC_DUP_POLYGON_NORMAL;
    const uint64_t ntri = dup ? ncoords / 9 : nconnections / 3;
    const uint64_t nverts = ncoords / 3;
    const uint64_t need_normals = mode == KVSMC_SHARED_VERTEX_NORMAL ? 3 * nverts : 3 * ntri;
    if (nnormals < need_normals || (ntri && (!coords || !normals || (!dup && !connections))))
        return fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "stl: mesh arrays of inconsistent sizes");
    KVSMC_CUDA(ctx, cudaSetDevice(ctx->device));
    float* d_c = nullptr;
    float* d_n = nullptr;
    uint32_t* d_k = nullptr;
    cudaError_t e = cudaSuccess;
    if (ntri) {
        e = kvsmc_host::device_malloc(ctx, &d_c, ncoords * sizeof(float));
        if (e == cudaSuccess) e = kvsmc_host::device_malloc(ctx, &d_n, need_normals * sizeof(float));
        if (e == cudaSuccess && !dup) e = kvsmc_host::device_malloc(ctx, &d_k, 3 * ntri * sizeof(uint32_t));
        if (e == cudaSuccess) e = cudaMemcpyAsync(d_c, coords, ncoords * sizeof(float), cudaMemcpyHostToDevice, ctx->stream);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(d_n, normals, need_normals * sizeof(float), cudaMemcpyHostToDevice, ctx->stream);
        if (e == cudaSuccess && !dup)
            e = cudaMemcpyAsync(d_k, connections, 3 * ntri * sizeof(uint32_t), cudaMemcpyHostToDevice, ctx->stream);
    }
    kvsmc_status st = KVSMC_OK;
    if (e != cudaSuccess)
        st = fail(ctx, e == cudaErrorMemoryAllocation ? KVSMC_ERR_OUT_OF_MEMORY : KVSMC_ERR_CUDA, "stl: %s",
                  cudaGetErrorString(e));
    else
        st = kvsmc_write_stl(ctx, path, mode, d_c, d_n, d_k, nverts, ntri);
    cudaStreamSynchronize(ctx->stream);
    if (d_c) cudaFree(d_c);
    if (d_n) cudaFree(d_n);
    if (d_k) cudaFree(d_k);
    return st;
}

}  // extern "C"
