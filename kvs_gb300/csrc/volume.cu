// volume.cu -- resident volumes: their device blocks, and the one pass that
// lays a volume out (rows padded to 16 bytes), takes its brick min/max table
// and its value range (GetMinMaxValues, StructuredVolumeObject.cpp:66-111).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>
#include <mutex>

#include "context.h"

namespace kvsmc {

namespace {

// Order-preserving 64-bit keys of the values (a NaN is never given one).
template <typename T> __device__ __forceinline__ unsigned long long value_key(T v)
{
    if constexpr (sizeof(T) == 4 && T(0.5) != T(0)) {   // float
        const uint32_t b = __float_as_uint(v == 0.0f ? 0.0f : v);
        return b & 0x80000000u ? ~b : b | 0x80000000u;
    } else if constexpr (sizeof(T) == 8 && T(0.5) != T(0)) {   // double
        const unsigned long long b = (unsigned long long)__double_as_longlong(v == 0.0 ? 0.0 : v);
        return b >> 63 ? ~b : b | (1ull << 63);
    } else if constexpr (T(-1) < T(0)) {
        return (unsigned long long)(long long)v ^ (1ull << 63);
    } else {
        return (unsigned long long)v;
    }
}

template <typename T> __device__ __forceinline__ unsigned long long raw_bits(T v)
{
    unsigned long long r = 0;
    memcpy(&r, &v, sizeof v);
    return r;
}

template <typename T> struct Limits;
#define KVSMC_LIMITS(T, LO, HI)                                  \
    template <> struct Limits<T> {                               \
        __device__ static T lowest() { return LO; }              \
        __device__ static T highest() { return HI; }             \
    };
KVSMC_LIMITS(int8_t, -128, 127)
KVSMC_LIMITS(int16_t, -32768, 32767)
KVSMC_LIMITS(int32_t, (int32_t)0x80000000, 0x7fffffff)
KVSMC_LIMITS(long long, (long long)0x8000000000000000ull, 0x7fffffffffffffffll)
KVSMC_LIMITS(uint8_t, 0, 255)
KVSMC_LIMITS(uint16_t, 0, 65535)
KVSMC_LIMITS(uint32_t, 0u, 0xffffffffu)
KVSMC_LIMITS(unsigned long long, 0ull, ~0ull)
KVSMC_LIMITS(float, __int_as_float(0xff800000), __int_as_float(0x7f800000))
KVSMC_LIMITS(double, __longlong_as_double((long long)0xfff0000000000000ull), __longlong_as_double(0x7ff0000000000000ll))
#undef KVSMC_LIMITS

constexpr int kIngestThreads = 256;

// A CTA's share of the range: the smallest of its threads' keys (all ones: none)
// into `out`, and the volume's first value.
template <bool FLOAT, typename T>
__device__ __forceinline__ void range_out(unsigned long long klo, unsigned long long knhi, unsigned long long zero,
                                          const T* values, IngestOut* out)
{
    __shared__ unsigned long long s_lo[kIngestThreads / 32], s_nhi[kIngestThreads / 32], s_zero[kIngestThreads / 32];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        klo = min(klo, __shfl_xor_sync(0xffffffffu, klo, o));
        knhi = min(knhi, __shfl_xor_sync(0xffffffffu, knhi, o));
        if (FLOAT) zero = min(zero, __shfl_xor_sync(0xffffffffu, zero, o));
    }
    if (lane == 0) {
        s_lo[warp] = klo;
        s_nhi[warp] = knhi;
        s_zero[warp] = zero;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < kIngestThreads / 32; ++k) {
            klo = min(klo, s_lo[k]);
            knhi = min(knhi, s_nhi[k]);
            zero = min(zero, s_zero[k]);
        }
        // (most CTAs change nothing: a look saves their turns at the same word)
        if (klo < __ldcg(&out->lo)) atomicMin(&out->lo, klo);
        if (knhi < __ldcg(&out->nhi)) atomicMin(&out->nhi, knhi);
        if (FLOAT && zero != ~0ull) atomicMin(&out->zero, zero);
        if (blockIdx.x == 0) out->first = raw_bits(values[0]);
    }
}

// One warp per brick of 8 cell planes x 2 cell rows x 128 cells (9 x 3 x 129
// nodes; bricks share their border nodes), persistent over the bricks.  src
// (may be null): the values, dense; every node is written once into the
// padded layout by the brick that owns it.  Without src the values are read
// in place.  Each brick's min and max go to `bricks`, the range of all values to
// `out`.
//
// Each value is read once from HBM (a brick's border nodes again from L1/L2,
// 1.7 loads a node in all) and written once; a warp's 13 loads of one plane are
// in flight together.  No lane branches on where its nodes end (columns and rows
// past the last are the last one again), and zeros and NaN are looked at closer
// only where one comparison a value has found some: branches for every value
// made 73 instructions a value and 78 us.  83 MB of floats (301 x 256 x 270):
// now 48 us, 3.4 TB/s read and written together (a copy, a brick pass and a
// min/max scan took 72, 137 us and more).  Looking at every zero of a background
// made the pass up to a fifth slower than without zeros; only a brick's first
// one is looked at.
template <typename T, bool COPY>
__global__ void __launch_bounds__(kIngestThreads)
    k_ingest(VolumeView v, const T* __restrict__ src, uint32_t nbx, uint32_t nby, uint64_t nbricks,
             float2* __restrict__ bricks, IngestOut* __restrict__ out)
{
    constexpr bool kFloat = T(0.5) != T(0);
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    T* const dst = static_cast<T*>(const_cast<void*>(v.data));
    const uint32_t cx = v.nx - 1, cy = v.ny - 1, cz = v.nz - 1;
    const uint64_t rp = COPY ? v.nx : v.pitch, sp = COPY ? (uint64_t)v.nx * v.ny : v.slice;
    const T* const from = COPY ? src : dst;
    T lo = Limits<T>::highest(), hi = Limits<T>::lowest();   // over this thread's values, NaN apart
    unsigned long long zero = ~0ull;                          // (index << 1 | sign) of its zero of lowest index
    const uint64_t warps = (uint64_t)gridDim.x * (kIngestThreads / 32);
    for (uint64_t b = (uint64_t)blockIdx.x * (kIngestThreads / 32) + warp; b < nbricks; b += warps) {
        const uint32_t q = (uint32_t)(b / nbx), bx = (uint32_t)(b - (uint64_t)q * nbx);   // (below 2^32 brick rows)
        const uint32_t bz = q / nby, by = q - bz * nby;
        // (ends as a start and a length: a row may have 2^32 - 1 nodes)
        const uint32_t x0 = bx * kBrickCells, x1 = x0 + min(kBrickCells, cx - x0);
        const uint32_t y0 = 2 * by, y1 = y0 + min(2u, cy - y0);
        const uint32_t z0 = bz * kBrickPlanes, z1 = z0 + min((uint32_t)kBrickPlanes, cz - z0);
        // this lane's nodes of a row: x0 + lane + 32 i, and lane r < 3 the one past
        // the brick's 128 cells in row r (its own only at the end of the row).
        // Columns and rows past the last are the last one again: the same values
        // to the same places.
        const uint32_t wx = x1 - x0, wy = y1 - y0;
        const bool full = wx == kBrickCells, own4 = x1 == cx;
        uint32_t off[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) off[i] = min(lane + 32 * i, wx);
        const uint32_t r4 = min(lane, wy);   // (lanes 0 .. 2)
        T blo = Limits<T>::highest(), bhi = Limits<T>::lowest();   // NaN apart
        bool nan = false, met = false;   // (met: a zero)
        const T* in = from + (uint64_t)z0 * sp + (uint64_t)y0 * rp + x0;
        T* to = dst + (uint64_t)z0 * v.slice + (uint64_t)y0 * v.pitch + x0;
        const uint64_t in1 = wy ? rp : 0, in2 = wy == 2 ? 2 * rp : in1;
        const uint64_t to1 = wy ? v.pitch : 0, to2 = wy == 2 ? 2 * v.pitch : to1;
        for (uint32_t z = z0; z <= z1; ++z, in += sp, to += v.slice) {
            T w[3][4], e = T(0);
            const T* const in_row[3] = {in, in + in1, in + in2};
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int i = 0; i < 4; ++i) w[r][i] = full ? (in_row[r] + lane)[32 * i] : in_row[r][off[i]];
            if (lane < 3) e = (in + r4 * rp)[wx];
            bool special = false;   // a zero or a NaN among this lane's values
            auto take = [&](T val) {
                if constexpr (kFloat) {
                    blo = fminf(blo, val);
                    bhi = fmaxf(bhi, val);
                } else {
                    if (val < blo) blo = val;
                    if (val > bhi) bhi = val;
                }
                if constexpr (kFloat) special |= !(val < T(0) || val > T(0));
            };
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int i = 0; i < 4; ++i) take(w[r][i]);
            if (lane < 3) take(e);
            if constexpr (kFloat) {
                if (special) {
#pragma unroll
                    for (int r = 0; r < 3; ++r)
#pragma unroll
                        for (int i = 0; i < 4; ++i) nan |= w[r][i] != w[r][i];
                    nan |= e != e;
                    // among equal values the scan keeps the first: only zeros' signs
                    // show it.  A thread meets a brick's values in index order, so the
                    // brick's first zero will do (a warp's bricks do not come in order)
                    if (!met) {
                        auto look = [&](T val, uint32_t y, uint32_t x) {
                            if (met || val != T(0)) return;
                            met = true;
                            zero = min(zero, ((((unsigned long long)z * v.ny + y) * v.nx + x) << 1) |
                                                 (raw_bits(val) != 0 ? 1ull : 0ull));
                        };
#pragma unroll
                        for (int r = 0; r < 3; ++r) {
#pragma unroll
                            for (int i = 0; i < 4; ++i) look(w[r][i], y0 + ((uint32_t)r < wy ? (uint32_t)r : wy), x0 + off[i]);
                            if ((int)lane == r) look(e, y0 + r4, x1);
                        }
                    }
                }
            }
            if (COPY && (z - z0 < kBrickPlanes || z == cz)) {
                T* const to_row[3] = {to, to + to1, to + to2};
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    if (r == 2 && y1 != cy) continue;   // the next brick's
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (full) (to_row[r] + lane)[32 * i] = w[r][i];
                        else to_row[r][off[i]] = w[r][i];
                    }
                }
                if (own4 && lane < 3 && (r4 < 2 || y1 == cy)) (to + r4 * v.pitch)[wx] = e;
            }
        }
        if (blo < lo) lo = blo;
        if (bhi > hi) hi = bhi;
        // (values of these types are floats exactly)
        float a = (float)blo, c = (float)bhi;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a = fminf(a, __shfl_xor_sync(0xffffffffu, a, o));
            c = fmaxf(c, __shfl_xor_sync(0xffffffffu, c, o));
        }
        nan = __any_sync(0xffffffffu, nan);
        // a brick holding a NaN is never skipped
        if (lane == 0)
            bricks[b] = nan ? make_float2(__int_as_float(0xff800000), __int_as_float(0x7f800000)) : make_float2(a, c);
    }
    const bool any = lo <= hi;
    range_out<kFloat>(any ? value_key(lo) : ~0ull, any ? ~value_key(hi) : ~0ull, zero, from, out);
}

// One value of the range of a thread's values (see k_flat).  8-byte values by
// their keys: doubles compare at 1/58 of the integer rate.
template <typename T> struct RangeTake {
    static constexpr bool kFloat = T(0.5) != T(0);
    unsigned long long klo = ~0ull, knhi = ~0ull, zero = ~0ull;
    T lo = Limits<T>::highest(), hi = Limits<T>::lowest();
    __device__ __forceinline__ void take(T val, uint64_t index)
    {
        if constexpr (sizeof(T) == 8) {
            unsigned long long k = value_key(val);
            if constexpr (kFloat) {
                const unsigned long long u = raw_bits(val) << 1;
                if (u - 1 >= 0xffe0000000000000ull) {   // a zero or a NaN
                    if (u != 0) return;
                    zero = min(zero, (index << 1) | (raw_bits(val) != 0 ? 1ull : 0ull));
                }
            }
            klo = min(klo, k);
            knhi = min(knhi, ~k);
        } else {
            if (val < lo) lo = val;   // (false for a NaN)
            if (val > hi) hi = val;
            if constexpr (kFloat)
                if (val == T(0)) zero = min(zero, (index << 1) | (raw_bits(val) != 0 ? 1ull : 0ull));
        }
    }
    __device__ __forceinline__ void keys()
    {
        if (sizeof(T) < 8 && lo <= hi) {
            klo = value_key(lo);
            knhi = ~value_key(hi);
        }
    }
};

// The same for volumes without a brick table (32/64-bit integers, doubles, and
// shapes that the streaming kernels do not take: one node thick, or rows wider
// than theirs): their values in index order, a warp 256 at a time with its eight
// loads in flight, so that it does not matter how the volume is shaped.  By
// bricks, an update of 262144 rows of one double took 985 us and one of
// 256x256x512 doubles 1789; now 42, and 1290 (the copy: nobody asked for the
// range).  A kvsmc_volume_from_device of the latter and its range: 183 us.
constexpr uint32_t kFlatTile = 256;

template <typename T, bool COPY>
__global__ void __launch_bounds__(kIngestThreads)
    k_flat(VolumeView v, const T* __restrict__ src, uint64_t n, IngestOut* __restrict__ out)
{
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    T* const dst = static_cast<T*>(const_cast<void*>(v.data));
    const bool padded = v.pitch != v.nx;
    RangeTake<T> r;
    const uint64_t tiles = (n + kFlatTile - 1) / kFlatTile, warps = (uint64_t)gridDim.x * (kIngestThreads / 32);
    for (uint64_t t = (uint64_t)blockIdx.x * (kIngestThreads / 32) + warp; t < tiles; t += warps) {
        const uint64_t i0 = t * kFlatTile, row0 = padded ? i0 / v.nx : 0;
        const uint32_t left = v.nx - (uint32_t)(i0 - row0 * v.nx);   // of the tile's first row
        uint64_t at[kFlatTile / 32];
        T w[kFlatTile / 32];
#pragma unroll
        for (uint32_t k = 0; k < kFlatTile / 32; ++k) {
            const uint32_t j = lane + 32 * k;
            uint64_t row = row0;
            uint32_t col = v.nx - left + j;
            if (padded && j >= left) {   // of a later row
                const uint32_t q = (j - left) / v.nx;
                row += 1 + q;
                col = (j - left) - q * v.nx;
            }
            at[k] = padded ? row * v.pitch + col : i0 + j;
            if (i0 + j < n) w[k] = COPY ? src[i0 + j] : dst[at[k]];
        }
#pragma unroll
        for (uint32_t k = 0; k < kFlatTile / 32; ++k) {
            const uint64_t i = i0 + lane + 32 * k;
            if (i >= n) continue;
            if (COPY) dst[at[k]] = w[k];
            r.take(w[k], i);
        }
    }
    r.keys();
    range_out<RangeTake<T>::kFloat>(r.klo, r.knhi, r.zero, COPY ? src : dst, out);
}

}  // namespace

cudaError_t launch_ingest(const VolumeView& v, const void* src, float2* bricks, IngestOut* d_out, const Launch& L)
{
    cudaError_t e = cudaMemsetAsync(d_out, 0xff, sizeof *d_out, L.stream);
    if (e != cudaSuccess) return e;
    // bricks of `per` cells along an axis of n nodes (at least one; n may be 2^32 - 1)
    auto bricks_of = [](uint32_t n, uint32_t per) { return n < 2 ? 1u : (n - 2) / per + 1; };
    const uint32_t nbx = bricks_of(v.nx, kBrickCells), nby = bricks_of(v.ny, 2);
    const uint64_t nbricks = (uint64_t)nbx * nby * bricks_of(v.nz, (uint32_t)kBrickPlanes);
    const uint64_t n = (uint64_t)v.nx * v.ny * v.nz;
    const uint64_t warps = bricks ? nbricks : (n + kFlatTile - 1) / kFlatTile;   // one each, if they fit
    const uint64_t need = (warps + kIngestThreads / 32 - 1) / (kIngestThreads / 32), cap = (uint64_t)L.num_sms * 8;
    const unsigned grid = (unsigned)(need < cap ? need : cap);
#define KVSMC_FLAT(T)                                                                                    \
    if (src) k_flat<T, true><<<grid, kIngestThreads, 0, L.stream>>>(v, static_cast<const T*>(src), n, d_out); \
    else k_flat<T, false><<<grid, kIngestThreads, 0, L.stream>>>(v, nullptr, n, d_out);                  \
    break;
#define KVSMC_TABLE(T)                                                                                        \
    if (!bricks) { KVSMC_FLAT(T) }                                                                            \
    if (src)                                                                                                  \
        k_ingest<T, true><<<grid, kIngestThreads, 0, L.stream>>>(v, static_cast<const T*>(src), nbx, nby, nbricks, \
                                                                 bricks, d_out);                              \
    else                                                                                                      \
        k_ingest<T, false><<<grid, kIngestThreads, 0, L.stream>>>(v, nullptr, nbx, nby, nbricks, bricks, d_out);   \
    break;
    prof_begin(L, "ingest");
    switch (v.dtype) {
    case 0: KVSMC_TABLE(int8_t)
    case 1: KVSMC_TABLE(int16_t)
    case 2: KVSMC_FLAT(int32_t)
    case 3: KVSMC_FLAT(long long)
    case 4: KVSMC_TABLE(uint8_t)
    case 5: KVSMC_TABLE(uint16_t)
    case 6: KVSMC_FLAT(uint32_t)
    case 7: KVSMC_FLAT(unsigned long long)
    case 8: KVSMC_TABLE(float)
    case 9: KVSMC_FLAT(double)
    default: return cudaErrorInvalidValue;
    }
#undef KVSMC_TABLE
#undef KVSMC_FLAT
    prof_end(L);
    *L.counter += 1;
    return cudaGetLastError();
}

}  // namespace kvsmc

namespace kvsmc_host {

namespace {

// A key of value_key back to its value.
double key_value(int dtype, unsigned long long k)
{
    switch (dtype) {
    case KVSMC_F32: {
        const uint32_t b = (uint32_t)k & 0x80000000u ? (uint32_t)k & 0x7fffffffu : ~(uint32_t)k;
        float f;
        std::memcpy(&f, &b, sizeof f);
        return (double)f;
    }
    case KVSMC_F64: {
        const unsigned long long b = k >> 63 ? k & ~(1ull << 63) : ~k;
        double d;
        std::memcpy(&d, &b, sizeof d);
        return d;
    }
    case KVSMC_I8: case KVSMC_I16: case KVSMC_I32: case KVSMC_I64: return (double)(long long)(k ^ (1ull << 63));
    default: return (double)k;
    }
}

// GetMinMaxValues (StructuredVolumeObject.cpp:66-85) from the ingest pass's
// result: the scan starts at values[0], which a NaN there never leaves, and
// keeps the first of equal values (seen in the sign of a zero).
void decode_range(int dtype, const kvsmc::IngestOut& o, double& lo, double& hi)
{
    if (dtype == KVSMC_F32 || dtype == KVSMC_F64) {
        double first;
        if (dtype == KVSMC_F32) {
            float f;
            const uint32_t b = (uint32_t)o.first;
            std::memcpy(&f, &b, sizeof f);
            first = (double)f;
        } else {
            std::memcpy(&first, &o.first, sizeof first);
        }
        if (std::isnan(first) || o.lo == ~0ull) {
            lo = hi = first;
            return;
        }
    }
    lo = key_value(dtype, o.lo);
    hi = key_value(dtype, ~o.nhi);
    if (o.zero != ~0ull) {
        const double z = o.zero & 1ull ? -0.0 : 0.0;
        if (lo == 0.0) lo = z;
        if (hi == 0.0) hi = z;
    }
}

size_t table_bytes(const kvsmc::VolumeView& v)
{
    const int dt = v.dtype;
    const bool ok = (dt == KVSMC_I8 || dt == KVSMC_I16 || dt == KVSMC_U8 || dt == KVSMC_U16 || dt == KVSMC_F32) &&
                    v.nx > 1 && v.ny > 1 && v.nz > 1 && v.nx - 1 <= (uint32_t)kvsmc::kStreamMaxCells;
    return ok ? kvsmc::brick_count(v) * sizeof(float2) : 0;
}

}  // namespace

kvsmc_status block_alloc(kvsmc_context* ctx, size_t bytes, kvsmc_volume* v)
{
    {
        // a spare block at most a quarter larger than asked for
        std::lock_guard<std::mutex> lock(ctx->spare_mutex);
        size_t best = ctx->spare.size();
        for (size_t i = 0; i < ctx->spare.size(); ++i)
            if (ctx->spare[i].bytes >= bytes && ctx->spare[i].bytes <= bytes + bytes / 4 + (1 << 20) &&
                (best == ctx->spare.size() || ctx->spare[i].bytes < ctx->spare[best].bytes))
                best = i;
        if (best < ctx->spare.size()) {
            v->dev = ctx->spare[best].p;
            v->bytes = ctx->spare[best].bytes;
            v->ev = ctx->spare[best].ev;
            ctx->spare.erase(ctx->spare.begin() + (long)best);
            return KVSMC_OK;
        }
    }
    cudaEvent_t ev = nullptr;
    KVSMC_CUDA(ctx, cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    const cudaError_t e = device_malloc(ctx, &v->dev, bytes);
    if (e != cudaSuccess) {
        cudaEventDestroy(ev);
        v->dev = nullptr;
        KVSMC_CUDA(ctx, e);
    }
    v->bytes = bytes;
    v->ev = ev;
    return KVSMC_OK;
}

cudaError_t device_malloc_bytes(kvsmc_context* ctx, void** p, size_t bytes)
{
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation && ctx && block_release(ctx)) {
        cudaGetLastError();
        e = cudaMalloc(p, bytes);
    }
    return e;
}

bool block_release(kvsmc_context* ctx)
{
    std::lock_guard<std::mutex> lock(ctx->spare_mutex);
    const bool any = !ctx->spare.empty();
    for (const kvsmc_context::Spare& s : ctx->spare) {
        cudaFree(s.p);
        cudaEventDestroy(s.ev);
    }
    ctx->spare.clear();
    return any;
}

void block_free(kvsmc_context* ctx, kvsmc_volume* v)
{
    if (!v->dev) return;
    // cudaFree waits for all work on the device.  A block that is kept waits for
    // the work that may still read it: calls wait for their own, the event stands
    // behind what uploads and updates leave running, on whatever stream, and a
    // block that other work reads is not kept.  (A wait for the whole device
    // would do, but is refused while any thread captures a stream, and ends its
    // capture.)
    if (ctx && !v->lent && v->bytes <= kSpareBytes && cudaEventSynchronize(v->ev) == cudaSuccess) {
        std::lock_guard<std::mutex> lock(ctx->spare_mutex);
        size_t held = 0;
        for (const kvsmc_context::Spare& s : ctx->spare) held += s.bytes;
        while (!ctx->spare.empty() && (held + v->bytes > kSpareBytes || ctx->spare.size() >= kSpareBlocks)) {
            held -= ctx->spare.front().bytes;   // the oldest leaves
            cudaFree(ctx->spare.front().p);
            cudaEventDestroy(ctx->spare.front().ev);
            ctx->spare.erase(ctx->spare.begin());
        }
        ctx->spare.push_back({v->dev, v->bytes, v->ev});
    } else {
        cudaFree(v->dev);
        cudaEventDestroy(v->ev);
    }
    v->dev = nullptr;
    v->bytes = 0;
    v->ev = nullptr;
    v->ev_own = true;
}

kvsmc_status volume_alloc(kvsmc_context* ctx, kvsmc_dtype dtype, uint32_t nx, uint32_t ny, uint32_t nz,
                          kvsmc_volume* v)
{
    const size_t es = kvsmc::dtype_size(dtype);
    const uint64_t pitch = align_up(nx, 16 / es);
    v->view.nx = nx; v->view.ny = ny; v->view.nz = nz;
    v->view.dtype = dtype;
    v->view.pitch = pitch;
    v->view.slice = pitch * ny;
    v->has_minmax = false;
    v->range_ready = false;
    v->bricks_valid = false;
    // values and 256 bytes of slack | range record | brick table
    const size_t values = align_up((size_t)pitch * ny * nz * es + 256, 256);
    const size_t bytes = values + 256 + table_bytes(v->view);
    if (bytes > v->bytes) {
        block_free(ctx, v);
        kvsmc_status st = block_alloc(ctx, bytes, v);
        if (st) return st;
        v->device = ctx->device;
        v->owner = ctx;
    }
    v->view.data = v->dev;
    v->range = reinterpret_cast<kvsmc::IngestOut*>(static_cast<char*>(v->dev) + values);
    v->bricks = table_bytes(v->view) ? reinterpret_cast<float2*>(static_cast<char*>(v->dev) + values + 256) : nullptr;
    return KVSMC_OK;
}

kvsmc_status volume_bricks(kvsmc_context* ctx, kvsmc_volume* v)
{
    if (v->bricks) {
        KVSMC_CUDA(ctx, kvsmc::launch_ingest(v->view, nullptr, v->bricks, v->range, launch_of(ctx)));
        v->bricks_valid = true;
        v->range_ready = true;
    }
    // (without a table too: the pass that turned a file's bytes may still run)
    v->ev_own = v->owner == ctx && ctx->stream == ctx->own_stream;
    KVSMC_CUDA(ctx, cudaEventRecord(v->ev, ctx->stream));
    return KVSMC_OK;
}

kvsmc_status volume_copy_in(kvsmc_context* ctx, kvsmc_volume* v, const void* src, bool on_device)
{
    const size_t es = kvsmc::dtype_size(v->view.dtype);
    const size_t row = (size_t)v->view.nx * es;
    const size_t rows = (size_t)v->view.ny * v->view.nz;
    const size_t dense = row * rows;
    v->has_minmax = false;
    v->range_ready = false;
    // An update may be captured into a caller's graph: its replays come when the
    // caller likes, so it takes no part in the events, reads no buffer of the
    // context's, and the block is not kept when the volume is freed.
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &cap) != cudaSuccess) cudaGetLastError();
    const bool captured = cap != cudaStreamCaptureStatusNone;
    // what the context's own stream ran comes first there without an event
    const bool own = ctx->stream == ctx->own_stream;
    if (captured) v->lent = true;
    else if (!(own && v->ev_own && v->owner == ctx))   // (an update on another stream comes first)
        KVSMC_CUDA(ctx, cudaStreamWaitEvent(ctx->stream, v->ev, 0));
    const void* from = nullptr;   // values the ingest pass copies (null: they are in place)
    if (on_device) {
        // read in place of a copy where the kernel can: device memory of this
        // GPU, aligned to the value type (a copy takes any address)
        cudaPointerAttributes a;
        if ((reinterpret_cast<uintptr_t>(src) % es) == 0 && cudaPointerGetAttributes(&a, src) == cudaSuccess &&
            a.type == cudaMemoryTypeDevice && a.device == ctx->device)
            from = src;
        else
            cudaGetLastError();
    } else if (v->view.pitch != v->view.nx && dense <= kDenseStage && !captured &&
               (v->bricks || row <= kStageRow)) {
        // rows that are padded on the device: one dense copy into a staging
        // buffer, padded by the ingest pass (a row-by-row copy of 99-node rows
        // of 16-bit values ran at 6 GB/s: 2.1 MB in 340 us; where no table asks for a
        // pass anyway, long rows are faster by themselves: 512 rows of 4097 doubles
        // 131 us staged, 105, of 1001 49, 50).  The last pass that
        // reads the buffer may be on another stream (kvsmc_set_stream): the copy
        // waits for it
        if (!ctx->dense_ev) KVSMC_CUDA(ctx, cudaEventCreateWithFlags(&ctx->dense_ev, cudaEventDisableTiming));
        if (!own && ctx->dense_own) KVSMC_CUDA(ctx, cudaEventRecord(ctx->dense_ev, ctx->own_stream));
        if (dense > ctx->dense_bytes) {
            if (own && ctx->dense_own) KVSMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
            else KVSMC_CUDA(ctx, cudaEventSynchronize(ctx->dense_ev));
            if (ctx->dense) cudaFree(ctx->dense);
            ctx->dense = nullptr;
            ctx->dense_bytes = 0;
            const size_t want = align_up(dense, 1 << 20);
            KVSMC_CUDA(ctx, device_malloc(ctx, &ctx->dense, want));
            ctx->dense_bytes = want;
        }
        if (!(own && ctx->dense_own)) KVSMC_CUDA(ctx, cudaStreamWaitEvent(ctx->stream, ctx->dense_ev, 0));
        KVSMC_CUDA(ctx, cudaMemcpyAsync(ctx->dense, src, dense, cudaMemcpyHostToDevice, ctx->stream));
        from = ctx->dense;
    }
    if (!from) {
        const cudaMemcpyKind kind = on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
        if (v->view.pitch == v->view.nx)
            KVSMC_CUDA(ctx, cudaMemcpyAsync(v->dev, src, dense, kind, ctx->stream));
        else
            KVSMC_CUDA(ctx, cudaMemcpy2DAsync(v->dev, v->view.pitch * es, src, row, row, rows, kind, ctx->stream));
    }
    // values that are in place already and need no table: their range is taken
    // when it is first asked for (an update with a preset one never does)
    v->bricks_valid = false;
    if (from || v->bricks) {
        KVSMC_CUDA(ctx, kvsmc::launch_ingest(v->view, from, v->bricks, v->range, launch_of(ctx)));
        v->bricks_valid = v->bricks != nullptr;
        v->range_ready = true;
    }
    if (captured) return KVSMC_OK;
    v->ev_own = own && v->owner == ctx;
    KVSMC_CUDA(ctx, cudaEventRecord(v->ev, ctx->stream));
    if (from && from == ctx->dense) {
        ctx->dense_own = own;
        if (!own) KVSMC_CUDA(ctx, cudaEventRecord(ctx->dense_ev, ctx->stream));
    }
    return KVSMC_OK;
}

kvsmc_status volume_minmax(kvsmc_context* ctx, kvsmc_volume* v)
{
    if (v->has_minmax) return KVSMC_OK;
    volume_use(ctx, v);
    kvsmc::IngestOut* range = v->range;
    if (!v->range_ready) {
        // a pass of its own, into the context's memory: another context may ask for
        // the same volume's range at the same time
        if (kvsmc_status st = ensure_scratch(ctx, sizeof(kvsmc::IngestOut))) return st;
        range = static_cast<kvsmc::IngestOut*>(ctx->scratch);
        KVSMC_CUDA(ctx, kvsmc::launch_ingest(v->view, nullptr, nullptr, range, launch_of(ctx)));
    }
    KVSMC_CUDA(ctx, cudaMemcpyAsync(ctx->h_small, range, sizeof(kvsmc::IngestOut), cudaMemcpyDeviceToHost, ctx->stream));
    KVSMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    kvsmc::IngestOut o;
    std::memcpy(&o, ctx->h_small, sizeof o);
    decode_range(v->view.dtype, o, v->vmin, v->vmax);
    v->has_minmax = true;
    return KVSMC_OK;
}

void volume_destroy(kvsmc_context* ctx, kvsmc_volume* v)
{
    block_free(ctx && ctx->device == v->device ? ctx : nullptr, v);
    delete v;
}

}  // namespace kvsmc_host
