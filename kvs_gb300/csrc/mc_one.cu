// mc_one.cu -- the count pass for groups of one isolevel, every value type.
//
// Most calls ask for one isosurface, and for one the threshold masks of the
// general count (mc_stream.cu: a bucket lookup per node, a loop over the
// isolevels of every cell) are not needed: a node is one compare, a lane's
// nine nodes of a staged row are nine bits, the cells that the isolevel
// crosses are three logic operations on the four rows' bits, and only where
// some lane has such a cell are the cases formed (an 8 x 8 bit transpose) and
// their triangles looked up.  Tasks, units, ring and outputs are the general
// count's: a chunk of cell planes, R cell rows, a segment of 256 / R cells,
// lane l on 8 cells of row l / (32 / R); one u16 triangle count per unit and
// (LIST) the unit's crossed cells in the pair list.
#include <cuda_runtime.h>

#include "mc_internal.h"
#include "tma.cuh"

namespace kvsmc {

namespace {

constexpr int kOneThreads = 256;
constexpr int kOneWarps = kOneThreads / 32;
constexpr unsigned FULL = 0xffffffffu;

__device__ uint8_t d_one_ntri[256] = MC_NTRI_INIT;

__host__ __device__ __forceinline__ size_t one_align(size_t v) { return (v + 127) / 128 * 128; }

// One compare per value: the classifier's threshold in the cheapest form.
template <typename T> struct Above {
    int t;   // 8/16-bit integers
    __device__ explicit Above(const Classifier& c)
        : t(c.i_thr > 0x7fffffffll ? 0x7fffffff : (c.i_thr < -0x7fffffffll ? -0x7fffffff : (int)c.i_thr))
    {
    }
    __device__ bool operator()(T v) const { return (int)v > t; }
};
template <> struct Above<float> {
    float t;
    __device__ explicit Above(const Classifier& c) : t(c.f_thr) {}
    __device__ bool operator()(float v) const { return v > t; }
};
#define KVSMC_ABOVE_WIDE(T)                                              \
    template <> struct Above<T> {                                        \
        Classifier c;                                                    \
        __device__ explicit Above(const Classifier& k) : c(k) {}         \
        __device__ bool operator()(T v) const { return above(c, v); }    \
    };
KVSMC_ABOVE_WIDE(int32_t)
KVSMC_ABOVE_WIDE(uint32_t)
KVSMC_ABOVE_WIDE(long long)
KVSMC_ABOVE_WIDE(unsigned long long)
KVSMC_ABOVE_WIDE(double)
#undef KVSMC_ABOVE_WIDE

// The 9 bits "above" of nodes 0 .. 8 of a staged row (16-byte shared loads).
template <typename T> __device__ __forceinline__ uint32_t row_bits(const T* p, const Above<T>& ab)
{
    constexpr int kVec = 16 / sizeof(T) < 8 ? 16 / sizeof(T) : 8;   // values per load
    struct alignas(kVec * sizeof(T)) Vec { T v[kVec]; };
    uint32_t m = 0;
#pragma unroll
    for (int g = 0; g < 8 / kVec; ++g) {
        const Vec w = reinterpret_cast<const Vec*>(p)[g];
#pragma unroll
        for (int i = 0; i < kVec; ++i) m |= ab(w.v[i]) ? 1u << (g * kVec + i) : 0u;
    }
    return m | (ab(p[8]) ? 1u << 8 : 0u);
}

template <typename T, int R, bool LIST>
__global__ void __launch_bounds__(kOneThreads)
    k_count_one(const StreamGroup* __restrict__ groups, int ngroups, uint64_t ntasks,
                const StreamIso* __restrict__ isos, uint16_t* __restrict__ unit_counts, int* __restrict__ status,
                unsigned long long* __restrict__ next_task, uint32_t wait_polls, PairList pl)
{
    constexpr int LPR = 32 / R;                     // lanes per cell row
    constexpr uint32_t SEG = kStreamSegCells / R;   // cells per row segment
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint8_t s_ntri[256];
    const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    s_ntri[tid] = d_one_ntri[tid];
    __syncthreads();   // the only CTA-wide barrier
    const uint32_t row_elems = groups[0].seg_elems;
    const uint32_t plane_elems = (R + 1) * row_elems;
    unsigned char* wbase = smem_raw + (size_t)warp * (128 + one_align((size_t)3 * plane_elems * sizeof(T)));
    uint64_t* bar = reinterpret_cast<uint64_t*>(wbase);
    T* ring = reinterpret_cast<T*>(wbase + 128);
    if (lane == 0) {
        for (int b = 0; b < 3; ++b) mbar_init(&bar[b], 1);
        fence_barrier_init();
    }
    __syncwarp();
    const uint32_t half = lane / LPR, xl = (lane % LPR) * 8;   // this lane's row of the task and first cell
    uint64_t lcur = 0, lend = 0;   // this warp's entries of the pair list
    bool lfull = false;
    uint32_t ph = 0;   // per ring buffer: parity of its next completion
    int gi = 0;
    for (;;) {
        unsigned long long tk = 0;
        if (lane == 0) tk = atomicAdd(next_task, 1ull);
        const uint64_t task = __shfl_sync(FULL, tk, 0);
        if (task >= ntasks) break;
        while (gi + 1 < ngroups && task >= groups[gi + 1].task_begin) ++gi;   // (tasks come in increasing order)
        const StreamGroup& G = groups[gi];
        const Above<T> ab(isos[G.iso_begin].cls);
        const uint32_t local = (uint32_t)(task - G.task_begin);
        const uint32_t cx = G.vol.nx - 1, cy = G.vol.ny - 1, cz = G.vol.nz - 1, wpr = G.wpr;
        const uint64_t pitch = G.vol.pitch, slice = G.vol.slice;
        const uint32_t cyr = (cy + R - 1) / R;
        const uint32_t q = local / wpr, seg = local - q * wpr;
        const uint32_t zc = q / cyr, y = (q - zc * cyr) * R;
        const uint32_t z0 = zc * G.zchunk;
        const uint32_t z1 = z0 + G.zchunk < cz ? z0 + G.zchunk : cz;   // cell planes [z0, z1)
        // empty space: a brick whose node range lies on one side of the threshold
        const float2* bricks = G.bricks;
        const uint32_t nby = (cy + 1) / 2, brick_wpr = G.brick_wpr;
        const float thr = isos[G.iso_begin].f.f_thr;
        auto brick_empty = [&](uint32_t z) -> bool {
            const float2* row = bricks + ((uint64_t)(z / kBrickPlanes) * nby + (y >> 1)) * brick_wpr;
            float2 mm = row[R == 2 ? seg : 2 * seg];
            if (R == 1 && 2 * seg + 1 < brick_wpr) {   // a 256-cell segment spans two bricks
                const float2 m1 = row[2 * seg + 1];
                mm.x = fminf(mm.x, m1.x);
                mm.y = fmaxf(mm.y, m1.y);
            }
            return (mm.x > thr) == (mm.y > thr);
        };
        if (bricks) {
            bool all_empty = true;
            for (uint32_t z = z0; z < z1 && all_empty; z = (z / kBrickPlanes + 1) * kBrickPlanes)
                all_empty = brick_empty(z);
            if (all_empty) continue;   // (counts and pair numbers are zeroed before the pass)
        }
        const uint32_t nplanes = z1 - z0 + 1;
        const uint32_t nrows = y + R + 1 <= G.vol.ny ? R + 1 : G.vol.ny - y;   // node rows staged per plane
        const uint64_t xoff = (uint64_t)seg * SEG;
        const uint64_t avail = (pitch - xoff) * sizeof(T);
        const uint32_t row_bytes = (uint32_t)(avail < G.seg_copy_bytes ? avail : G.seg_copy_bytes);
        const T* src0 = static_cast<const T*>(G.vol.data) + (uint64_t)z0 * slice + (uint64_t)y * pitch + xoff;
        auto issue = [&](uint32_t i) {
            const uint32_t b = i % 3u;
            T* dst = ring + b * plane_elems;
            const T* src = src0 + (uint64_t)i * slice;
            mbar_arrive_expect_tx(&bar[b], nrows * row_bytes);
            for (uint32_t r = 0; r < nrows; ++r) bulk_copy_g2s(dst + r * row_elems, src + r * pitch, row_bytes, &bar[b]);
        };
        auto acquire = [&](uint32_t i) -> bool {
            const uint32_t b = i % 3u;
            const bool ok = mbar_wait(&bar[b], (ph >> b) & 1u, wait_polls);
            if (ok) ph ^= 1u << b;
            return ok;
        };
        __syncwarp();   // the previous task's reads of the ring are done
        if (lane == 0) {
            fence_proxy_async();
            for (uint32_t i = 0; i < nplanes && i < 3; ++i) issue(i);
        }
        const bool row_ok = y + half < cy;
        // the lane's unit and (isolevel, unit) counter at plane z0 (the group's
        // fields are read once per task: the stores below could alias them)
        const uint32_t plane_units = cy * wpr;
        const uint64_t unit0 = ((uint64_t)z0 * cy + y + half) * wpr + seg;
        uint16_t* const ucount = unit_counts + G.unit_base + unit0;
        uint16_t* upairs = LIST ? pl.unit_pairs + G.pair_base + unit0 : nullptr;
        uint32_t* ulist = LIST ? pl.unit_list + G.pair_base + unit0 : nullptr;
        // this lane's cells inside the volume, as a mask
        const int lim = row_ok ? (int)cx - (int)((uint32_t)xoff + xl) : 0;
        const uint32_t inside = lim >= 8 ? 0xffu : (lim <= 0 ? 0u : (1u << lim) - 1u);
        auto plane_bits = [&](uint32_t i, uint32_t& r0, uint32_t& r1) {
            const T* p = ring + (i % 3u) * plane_elems + half * row_elems + xl;
            r0 = row_bits<T>(p, ab);
            r1 = row_bits<T>(p + row_elems, ab);
        };
        uint32_t a0 = 0, a1 = 0;   // plane z: rows y + half and the next
        bool have_a = false, brick_skip = false, dead = false;
        uint32_t acq = 0, issued = 0;
        for (uint32_t z = z0; z < z1; ++z) {
            const uint32_t s = z - z0;
            bool ok = true;
            while (ok && acq <= s + 1) {
                ok = acquire(acq);
                if (ok) ++acq;
            }
            if (__any_sync(FULL, !ok)) {
                if (lane == 0) atomicExch(status, 1);
                dead = true;
                issued = s + 3 < nplanes ? s + 3 : nplanes;
                break;
            }
            if (bricks && (s == 0 || z % kBrickPlanes == 0)) brick_skip = brick_empty(z);
            if (brick_skip) {
                have_a = false;
            } else {
                if (!have_a) plane_bits(s, a0, a1);
                uint32_t b0, b1;
                plane_bits(s + 1, b0, b1);
                const uint32_t o = a0 | a1 | b0 | b1, n = a0 & a1 & b0 & b1;
                uint32_t act = (o | (o >> 1)) & ~(n & (n >> 1)) & inside;   // the crossed cells
                if (__any_sync(FULL, act != 0)) {
                    const uint32_t m = __popc(act);
                    uint16_t* entry = nullptr;
                    if (LIST) {
                        uint32_t inc = m;
#pragma unroll
                        for (int d = 1; d < 32; d <<= 1) {
                            const uint32_t t = __shfl_up_sync(FULL, inc, d);
                            if (lane >= (unsigned)d) inc += t;
                        }
                        const uint32_t npairs = __shfl_sync(FULL, inc, 31);
                        if (lcur + npairs > lend) {
                            const uint32_t want = npairs > pl.run ? npairs : pl.run;
                            unsigned long long at = 0;
                            if (lane == 0) at = atomicAdd(pl.cursor, (unsigned long long)want);
                            lcur = __shfl_sync(FULL, at, 0);
                            lend = lcur + want;
                            if (lend > pl.cap && !lfull) {
                                lfull = true;
                                if (lane == 0) atomicExch(pl.overflow, 1);
                            }
                        }
                        entry = lfull ? nullptr : pl.list + lcur + (inc - m);
                        const uint32_t before = R == 1 ? 0u : __shfl_sync(FULL, inc, LPR - 1);
                        if (lane % LPR == 0 && row_ok) {
                            const uint32_t b = half ? before : 0u;
                            upairs[(uint64_t)s * plane_units] = (uint16_t)((R == 1 || half ? npairs : before) - b);
                            ulist[(uint64_t)s * plane_units] = (uint32_t)lcur + b;
                        }
                        lcur += npairs;
                    }
                    // byte k of the word: case bit k of the 8 cells (corners 0:(x,y,z)
                    // 1:(x+1,y,z) 2:(x+1,y+1,z) 3:(x,y+1,z), 4..7 the same at z+1); the
                    // transpose makes byte i cell i's case
                    uint64_t cw = (uint64_t)((a0 & 0xffu) | ((a0 >> 1) << 8) | ((a1 >> 1) << 16) | (a1 << 24)) |
                                  ((uint64_t)((b0 & 0xffu) | ((b0 >> 1) << 8) | ((b1 >> 1) << 16) | (b1 << 24)) << 32);
                    uint64_t tt = (cw ^ (cw >> 7)) & 0x00AA00AA00AA00AAull;
                    cw ^= tt ^ (tt << 7);
                    tt = (cw ^ (cw >> 14)) & 0x0000CCCC0000CCCCull;
                    cw ^= tt ^ (tt << 14);
                    tt = (cw ^ (cw >> 28)) & 0x00000000F0F0F0F0ull;
                    cw ^= tt ^ (tt << 28);
                    uint32_t tris = 0;
                    while (act) {
                        const uint32_t i = __ffs(act) - 1;
                        act &= act - 1;
                        tris += s_ntri[(uint32_t)(cw >> (8 * i)) & 0xffu];
                        if (LIST && entry) *entry++ = (uint16_t)(xl + i);
                    }
                    __syncwarp();
                    uint32_t sum;
                    if (R == 1) {
                        sum = __reduce_add_sync(FULL, tris);
                    } else {
                        sum = tris;
#pragma unroll
                        for (int d = LPR / 2; d > 0; d >>= 1) sum += __shfl_xor_sync(FULL, sum, d);
                    }
                    if (lane % LPR == 0 && row_ok && sum)
                        ucount[(uint64_t)s * plane_units] = (uint16_t)sum;
                }
                a0 = b0;
                a1 = b1;
                have_a = true;
            }
            // plane z is consumed: refill its buffer with plane z + 3
            __syncwarp();
            if (lane == 0 && s + 3 < nplanes) {
                fence_proxy_async();
                issue(s + 3);
            }
        }
        if (dead) {
            // wait (bounded, by its own limit) for the copies still in flight, then stop
            for (uint32_t i = acq; i < issued; ++i) {
                const uint32_t b = i % 3u;
                if (mbar_wait(&bar[b], (ph >> b) & 1u, 1u << 16)) ph ^= 1u << b;
            }
            break;
        }
    }
}

}  // namespace

#define KVSMC_ONE_SWITCH(DT, ...)                                    \
    switch (DT) {                                                    \
    case 0: { using T = int8_t; __VA_ARGS__; } break;                \
    case 1: { using T = int16_t; __VA_ARGS__; } break;               \
    case 2: { using T = int32_t; __VA_ARGS__; } break;               \
    case 3: { using T = long long; __VA_ARGS__; } break;             \
    case 4: { using T = uint8_t; __VA_ARGS__; } break;               \
    case 5: { using T = uint16_t; __VA_ARGS__; } break;              \
    case 6: { using T = uint32_t; __VA_ARGS__; } break;              \
    case 7: { using T = unsigned long long; __VA_ARGS__; } break;    \
    case 8: { using T = float; __VA_ARGS__; } break;                 \
    case 9: { using T = double; __VA_ARGS__; } break;                \
    default: return cudaErrorInvalidValue;                           \
    }

cudaError_t launch_count_one(int dtype, int rows, const StreamGroup* d_groups, int ngroups, uint64_t ntasks,
                             const StreamIso* d_isos, uint16_t* d_unit_counts, int* d_status,
                             unsigned long long* d_next_task, const Launch& L, const PairList* list)
{
    if (ntasks == 0) return cudaSuccess;
    if (rows != 1 && rows != 2) return cudaErrorInvalidValue;
    const size_t smem = (size_t)kOneWarps *
                        (128 + one_align(3 * (size_t)(rows + 1) * stream_row_elems(dtype, rows) * dtype_size(dtype)));
    const uint64_t need = (ntasks + kOneWarps - 1) / kOneWarps;
    KVSMC_ONE_SWITCH(dtype, {
        auto kern = rows == 1 ? (list ? k_count_one<T, 1, true> : k_count_one<T, 1, false>)
                              : (list ? k_count_one<T, 2, true> : k_count_one<T, 2, false>);
        int per_sm = 0;
        const cudaError_t e = kernel_fit(L, reinterpret_cast<const void*>(kern), kOneThreads, smem, &per_sm, true);
        if (e != cudaSuccess) return e;
        if (list && per_sm > kListWarpsPerSm / kOneWarps) per_sm = kListWarpsPerSm / kOneWarps;
        const uint64_t resident = (uint64_t)(per_sm > 0 ? per_sm : 1) * (uint64_t)L.num_sms;
        prof_begin(L, "count_one");
        kern<<<(unsigned)(need < resident ? need : resident), kOneThreads, smem, L.stream>>>(
            d_groups, ngroups, ntasks, d_isos, d_unit_counts, d_status, d_next_task, L.wait_polls[0],
            list ? *list : PairList{});
        prof_end(L);
    });
    *L.counter += 1;
    return cudaGetLastError();
}

}  // namespace kvsmc
