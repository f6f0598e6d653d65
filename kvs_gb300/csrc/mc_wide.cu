// mc_wide.cu -- the classifying emit of 32/64-bit integer and double volumes
// (duplicated mode): for counts whose pair list overflowed or had no room.
// (The count is mc_one.cu's, the emit over listed pairs mc_pairs.cu's.)
//
// A warp task is a streaming cell task with one row per task: a chunk of cell
// planes, one cell row, a 256-cell segment, the two node rows of each node
// plane arriving in the warp's three-buffer ring through bulk copies.  Lane l
// owns cells 8 l .. 8 l + 7.  One isolevel per group: each node is classified
// by one integer compare (Classifier), the 8 cells' cases come out of four
// 9-bit row masks by an 8 x 8 bit transpose, and the upper plane's masks are
// the next step's lower ones.  A step's triangles are spread over the lanes,
// one lane a triangle, its vertices by the FP64 sequence (201 x 173 x 187
// doubles, 488 k triangles: 175 us; over listed pairs 81 us).
#include <cuda_runtime.h>

#include "mc_internal.h"
#include "tma.cuh"

namespace kvsmc {

namespace {

constexpr int kWideThreads = 256;
constexpr int kWideWarps = kWideThreads / 32;
constexpr unsigned FULL = 0xffffffffu;

__constant__ uint64_t c_w_tri[256] = MC_TRI_PACKED_INIT;
__constant__ uint8_t c_w_ntri[256] = MC_NTRI_INIT;
__constant__ uint8_t c_w_edge[12] = MC_EDGE_PACKED_INIT;

__host__ __device__ __forceinline__ size_t w_align(size_t v) { return (v + 127) / 128 * 128; }

template <typename T>
__global__ void __launch_bounds__(kWideThreads)
    k_wide(const StreamGroup* __restrict__ groups, int ngroups, uint64_t ntasks, const StreamIso* __restrict__ isos,
           const uint16_t* __restrict__ unit_counts, const uint32_t* __restrict__ unit_offsets,
           const uint64_t* __restrict__ plane_base, int* __restrict__ status,
           unsigned long long* __restrict__ next_task, uint32_t wait_polls, uint64_t task0,
           const uint64_t* __restrict__ totals, const int* __restrict__ only_if)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint64_t s_tri[256];
    __shared__ uint8_t s_ntri[256];
    __shared__ uint8_t s_edge[16];
    const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    for (unsigned c = tid; c < 256; c += blockDim.x) {
        s_tri[c] = c_w_tri[c];
        s_ntri[c] = c_w_ntri[c];
        if (c < 12) s_edge[c] = c_w_edge[c];
    }
    // the only CTA-wide barrier (an emit whose count gave up writes nothing)
    if (__syncthreads_or(*status != 0 || (only_if && *only_if == 0))) return;
    const uint32_t row_elems = groups[0].seg_elems;
    const size_t plane_elems = 2 * (size_t)row_elems;
    unsigned char* wbase = smem_raw + (size_t)warp * (128 + w_align(3 * plane_elems * sizeof(T)));
    uint64_t* bar = reinterpret_cast<uint64_t*>(wbase);
    T* ring = reinterpret_cast<T*>(wbase + 128);
    if (lane == 0) {
        for (int b = 0; b < 3; ++b) mbar_init(&bar[b], 1);
        fence_barrier_init();
    }
    __syncwarp();
    uint32_t ph = 0;   // per ring buffer: parity of its next completion
    int gi = 0;
    for (;;) {
        unsigned long long tk = 0;
        if (lane == 0) tk = atomicAdd(next_task, 1ull);
        const uint64_t task = task0 + __shfl_sync(FULL, tk, 0);
        if (task >= ntasks) break;
        while (gi + 1 < ngroups && task >= groups[gi + 1].task_begin) ++gi;   // (tasks come in increasing order)
        const StreamGroup& G = groups[gi];
        if (G.skip_emit) continue;
        const StreamIso& I = isos[G.iso_begin];
        float* const out_c = I.coords;
        float* const out_n = I.normals;
        const uint64_t cap = I.cap_tris;
        if (!out_c || (totals && totals[G.iso_begin] > cap)) continue;   // not written at all
        const Classifier cls = I.cls;
        const uint64_t local = task - G.task_begin;
        const uint32_t cx = G.vol.nx - 1, cy = G.vol.ny - 1, cz = G.vol.nz - 1, wpr = G.wpr;
        const uint64_t pitch = G.vol.pitch, slice = G.vol.slice;
        const T* vol = static_cast<const T*>(G.vol.data);
        const uint32_t seg = (uint32_t)(local % wpr);
        const uint32_t y = (uint32_t)((local / wpr) % cy);
        const uint32_t zc = (uint32_t)(local / ((uint64_t)wpr * cy));
        const uint32_t z0 = zc * G.zchunk;
        const uint32_t z1 = z0 + G.zchunk < cz ? z0 + G.zchunk : cz;   // cell planes [z0, z1)
        const uint32_t nplanes = z1 - z0 + 1;
        const uint64_t xoff = (uint64_t)seg * kStreamSegCells;
        const uint64_t avail = (pitch - xoff) * sizeof(T);
        const uint32_t row_bytes = (uint32_t)(avail < G.seg_copy_bytes ? avail : G.seg_copy_bytes);
        auto issue = [&](uint32_t i) {
            const int b = (int)(i % 3u);
            T* dst = ring + (size_t)b * plane_elems;
            const T* src = vol + (uint64_t)(z0 + i) * slice + (uint64_t)y * pitch + xoff;
            mbar_arrive_expect_tx(&bar[b], 2 * row_bytes);
            for (uint32_t r = 0; r < 2; ++r) bulk_copy_g2s(dst + r * row_elems, src + r * pitch, row_bytes, &bar[b]);
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
        uint32_t acq = 0, issued = 0;
        bool dead = false;
        const int lim = (int)cx - (int)((uint32_t)xoff + 8 * lane);   // this lane's cells inside the row (if < 8)
        auto unit_of = [&](uint32_t zz) -> uint64_t { return G.unit_base + ((uint64_t)zz * cy + y) * wpr + seg; };
        const uint64_t first_plane = plane_base[I.plane_index];
        auto unit_first = [&](uint32_t zz) -> uint64_t {
            return plane_base[I.plane_index + zz] - first_plane + unit_offsets[unit_of(zz)];
        };
        // the unit's triangles and first triangle, loaded one step ahead
        uint32_t next_count = unit_counts[unit_of(z0)];
        uint64_t next_first = unit_first(z0);
        uint32_t ma = 0;        // rows y, y + 1 of plane z: this lane's 9 nodes above (bits 0-8, 16-24)
        bool have_a = false;
        auto row_mask = [&](const T* p) -> uint32_t {
            uint32_t m = 0;
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                m |= (above(cls, p[k]) ? 1u : 0u) << k;
                m |= (above(cls, p[row_elems + k]) ? 1u : 0u) << (16 + k);
            }
            return m;
        };
        for (uint32_t z = z0; z < z1; ++z) {
            const uint32_t st = z - z0;
            const uint32_t count_now = next_count;
            const uint64_t tbase = next_first;
            if (z + 1 < z1) {
                next_count = unit_counts[unit_of(z + 1)];
                next_first = unit_first(z + 1);
            }
            bool ok = true;
            while (ok && acq <= st + 1) {
                ok = acquire(acq);
                if (ok) ++acq;
            }
            if (__any_sync(FULL, !ok)) {
                if (lane == 0) atomicExch(status, 1);
                dead = true;
                issued = st + 3 < nplanes ? st + 3 : nplanes;
                break;
            }
            if (count_now == 0) {
                have_a = false;
            } else {
                const T* a = ring + (size_t)(st % 3u) * plane_elems + 8 * lane;
                const T* b = ring + (size_t)((st + 1) % 3u) * plane_elems + 8 * lane;
                if (!have_a) ma = row_mask(a);
                const uint32_t mb = row_mask(b);
                const uint32_t a0 = ma & 0x1ffu, a1 = ma >> 16, b0 = mb & 0x1ffu, b1 = mb >> 16;
                ma = mb;
                have_a = true;
                // byte k of the word: case bit k of the 8 cells (corners 0:(x,y,z)
                // 1:(x+1,y,z) 2:(x+1,y+1,z) 3:(x,y+1,z), 4..7 the same at z+1); the
                // transpose makes byte i cell i's case
                uint64_t cw = (uint64_t)((a0 & 0xffu) | ((a0 >> 1) << 8) | ((a1 >> 1) << 16) | ((a1 & 0xffu) << 24)) |
                              ((uint64_t)((b0 & 0xffu) | ((b0 >> 1) << 8) | ((b1 >> 1) << 16) | ((b1 & 0xffu) << 24))
                               << 32);
                uint64_t tt = (cw ^ (cw >> 7)) & 0x00AA00AA00AA00AAull;
                cw ^= tt ^ (tt << 7);
                tt = (cw ^ (cw >> 14)) & 0x0000CCCC0000CCCCull;
                cw ^= tt ^ (tt << 14);
                tt = (cw ^ (cw >> 28)) & 0x00000000F0F0F0F0ull;
                cw ^= tt ^ (tt << 28);
                if (lim < 8) cw &= lim <= 0 ? 0ull : (~0ull >> (64 - 8 * lim));   // cells past the row: none
                uint32_t n = 0;
                if (cw != 0 && cw != ~0ull) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) n += s_ntri[(uint32_t)(cw >> (8 * i)) & 0xffu];
                }
                {
                    uint32_t inc = n;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t t = __shfl_up_sync(FULL, inc, o);
                        if (lane >= (unsigned)o) inc += t;
                    }
                    const uint32_t total = __shfl_sync(FULL, inc, 31);
                    for (uint32_t q0 = 0; q0 < total; q0 += 32) {
                        // triangle q: of the first lane whose inclusive count exceeds it
                        const uint32_t q = q0 + lane;
                        uint32_t lo = 0;
#pragma unroll
                        for (int s = 4; s >= 0; --s) {
                            const uint32_t mid = lo + (1u << s) - 1u;
                            if (__shfl_sync(FULL, inc, mid) <= q) lo = mid + 1;
                        }
                        const uint32_t owner = lo < 32 ? lo : 31;
                        uint32_t r = q - __shfl_sync(FULL, inc - n, owner);
                        const uint64_t ocw = __shfl_sync(FULL, cw, owner);
                        if (q >= total) continue;
                        uint32_t ci = 0;
#pragma unroll
                        for (int i = 0; i < 7; ++i) {
                            const uint32_t nt = s_ntri[(uint32_t)(ocw >> (8 * i)) & 0xffu];
                            if (ci == (uint32_t)i && r >= nt) { r -= nt; ci = i + 1; }
                        }
                        const uint64_t pk = s_tri[(uint32_t)(ocw >> (8 * ci)) & 0xffu] >> (12 * r);
                        const uint32_t xl = 8 * owner + ci;
                        const uint64_t t = tbase + q;
                        if (t >= cap) continue;
                        float3 v[3];
#pragma unroll
                        for (int e = 0; e < 3; ++e) {
                            const unsigned ep = s_edge[(uint32_t)(pk >> (4 * e)) & 15u];
                            const unsigned c0 = ep & 7u, c1 = ep >> 3, d = c0 ^ c1;
                            auto at = [&](unsigned c) -> double {
                                const uint32_t buf = (st + (c >> 2)) % 3u;
                                return to_double(ring[buf * plane_elems + ((c >> 1) & 1u) * row_elems + xl + (c & 1u)]);
                            };
                            const uint32_t x = (uint32_t)xoff + xl;
                            v[e] = interpolate_exact_axis(I.ip, at(c0), at(c1), __uint2float_rn(x + (c0 & 1u)),
                                               __uint2float_rn(y + ((c0 >> 1) & 1u)), __uint2float_rn(z + (c0 >> 2)),
                                               __uint2float_rn(x + (c1 & 1u)), __uint2float_rn(y + ((c1 >> 1) & 1u)),
                                               __uint2float_rn(z + (c1 >> 2)), d == 1u ? 0 : (d == 2u ? 1 : 2));
                        }
                        float* o = out_c + 9 * t;
#pragma unroll
                        for (int e = 0; e < 3; ++e) { o[3 * e] = v[e].x; o[3 * e + 1] = v[e].y; o[3 * e + 2] = v[e].z; }
                        const float3 nn = tri_normal(v[0], v[1], v[2]);
                        float* p = out_n + 3 * t;
                        p[0] = nn.x; p[1] = nn.y; p[2] = nn.z;
                    }
                }
            }
            // plane z is consumed: refill its buffer with plane z + 3
            __syncwarp();
            if (lane == 0 && st + 3 < nplanes) {
                fence_proxy_async();
                issue(st + 3);
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

#define KVSMC_WIDE_SWITCH(DT, ...)                                   \
    switch (DT) {                                                    \
    case 2: { using T = int32_t; __VA_ARGS__; } break;               \
    case 3: { using T = long long; __VA_ARGS__; } break;             \
    case 6: { using T = uint32_t; __VA_ARGS__; } break;              \
    case 7: { using T = unsigned long long; __VA_ARGS__; } break;    \
    case 9: { using T = double; __VA_ARGS__; } break;                \
    default: return cudaErrorInvalidValue;                           \
    }

cudaError_t launch_wide(int dtype, const StreamGroup* d_groups, int ngroups, uint64_t ntasks,
                        const StreamIso* d_isos, const uint16_t* d_unit_counts, const uint32_t* d_unit_offsets,
                        const uint64_t* d_plane_base, int* d_status, unsigned long long* d_next_task, const Launch& L,
                        uint64_t task0, const uint64_t* d_totals, const int* d_only_if)
{
    const size_t smem =
        (size_t)kWideWarps * (128 + w_align(3 * 2 * stream_row_elems(dtype, 1) * dtype_size(dtype)));
    const uint64_t need = (ntasks - task0 + kWideWarps - 1) / kWideWarps;
    KVSMC_WIDE_SWITCH(dtype, {
        auto kern = k_wide<T>;
        int per_sm = 0;
        const cudaError_t e = kernel_fit(L, reinterpret_cast<const void*>(kern), kWideThreads, smem, &per_sm, true);
        if (e != cudaSuccess) return e;
        const uint64_t resident = (uint64_t)(per_sm > 0 ? per_sm : 1) * (uint64_t)L.num_sms;
        prof_begin(L, "wide_emit");
        kern<<<(unsigned)(need < resident ? need : resident), kWideThreads, smem, L.stream>>>(
            d_groups, ngroups, ntasks, d_isos, d_unit_counts, d_unit_offsets, d_plane_base, d_status, d_next_task,
            L.wait_polls[1], task0, d_totals, d_only_if);
        prof_end(L);
    });
    *L.counter += 1;
    return cudaGetLastError();
}

}  // namespace kvsmc
