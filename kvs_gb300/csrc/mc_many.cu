// mc_many.cu -- the count pass for several isolevels of a volume at once
// (8/16-bit and float32 values): triangles per (unit, isolevel) and, with a
// list, the active (cell, isolevel) pairs for mc_pairs.cu and mc_connect.cu.
//
// Tasks, units and threshold masks are the streaming kernels' (mc_stream.cu,
// mc_thermo.cuh): a warp walks a chunk of cell planes of R cell rows, lane l on
// 8 cells; each node's mask has bit k set when it is above isolevel k, and a
// cell's active isolevels are OR & ~AND of its corners' masks.  What is new
// against counting in the lanes' own loops (one divergent pass per pair: its
// case code, a table read and a shared atomic):
//   * the new plane's masks also go to shared memory, so a pair's case code can
//     be formed by any lane;
//   * the lanes only list their pairs (cell, isolevel) in a per-warp buffer;
//     the pairs are then taken 32 at a time, one per lane: the eight mask bits,
//     the triangle count, and one addition per distinct (row, isolevel) of the
//     round (__match_any_sync and bit-sliced ballots), no atomics; only steps
//     where all lanes have many pairs keep the lanes' loops;
//   * the same 32 entries go to the global list as one coalesced store;
//   * a staged plane's values are not needed once its masks are formed, so two
//     buffers a warp suffice, and the next copies start before the pairs are
//     worked on.
// Bound by instruction issue (70% busy) and shared-memory latency, and above all
// it must not spill: 32 warps an SM at 64 registers took 1500 and 2312 us below,
// 24 at 80 take 1210 and 1887, with the lower plane's masks read back from
// shared memory and the task's addresses kept there.  640x704x600 f32, 16
// isolevels: 1532 us with the lanes' loops, 1210 us; 1024x768x640 u16, 4
// isolevels: 2735 -> 1887 us.
//
// NODES: the shared-vertex modes' vertices per node unit too (plane, node row,
// 256-node segment; those whose node segments are their cell segments).  A
// node's cut edges are its cell's lower ones, so a pair adds them to its key
// beside its triangles; the last cell of a row, the last row and the last plane
// add the nodes behind them.
#include <cuda_runtime.h>

#include "mc_internal.h"
#include "mc_tables.h"
#include "mc_thermo.cuh"
#include "tma.cuh"

namespace kvsmc {

namespace {

constexpr int kManyThreads = 256;
constexpr int kManyWarps = kManyThreads / 32;
// Listed pairs per warp at a time.  A lane's pairs lie side by side, so where
// every cell has several a short buffer is filled by one or two lanes at a time:
// 16 isolevels of noise, 150^3: 6910 us a call with 128 entries, 5820 with 1024.
constexpr uint32_t kManyBuf = 1024;
// Pairs a step from which the lanes' own loops are looked at.
constexpr uint32_t kManyCrowd = 512;
constexpr unsigned FULL = 0xffffffffu;

__device__ uint8_t d_many_ntri[256] = MC_NTRI_INIT;   // per reference case

__host__ __device__ __forceinline__ size_t many_align(size_t v) { return (v + 127) / 128 * 128; }

// Mask rows: SEG + 1 nodes and padding to 16 bytes.
template <int R> constexpr uint32_t kMaskRow = 256 / R + 8;

template <typename T, int R> struct alignas(16) ManyWarp {
    uint16_t mask[2][R + 1][kMaskRow<R>];   // node masks of the lower and the upper plane (plane & 1)
    uint16_t buf[kManyBuf];                 // cell in the warp (8 bits) | isolevel << 8
    // [row][isolevel]: triangles | vertices << 16 of the current units; with
    // vertices (R = 1) 16 + k: those of the node units past the last cell row,
    // past the last cell plane and past both, 10 bits each
    uint32_t cnt[32];
    uint64_t bar[2];
    uint16_t* counts;                       // the task's counters, pair numbers, list entries and node counters
    uint16_t* pairs;
    uint32_t* list;
    uint32_t* nodes;
    ThermoTables<T> th;
};

template <typename T, int R, bool LIST, bool NODES>
__global__ void __launch_bounds__(kManyThreads, 3)
    k_count_many(const StreamGroup* __restrict__ groups, int ngroups, uint64_t ntasks,
                 const StreamIso* __restrict__ isos, uint16_t* __restrict__ unit_counts, int* __restrict__ status,
                 unsigned long long* __restrict__ next_task, uint32_t wait_polls, PairList pl,
                 uint32_t* __restrict__ node_counts)
{
    static_assert(!NODES || R == 1, "node units are one row");
    constexpr int LPR = 32 / R;                     // lanes per cell row
    constexpr uint32_t SEG = kStreamSegCells / R;   // cells per row segment
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint8_t s_tab[256];   // by corner code: triangles | the lower node's cut edges << 3
    const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    s_tab[tid] = (uint8_t)(d_many_ntri[code_to_case(tid)] |
                           ((((tid ^ (tid >> 4)) & 1u) + ((tid ^ (tid >> 1)) & 1u) + ((tid ^ (tid >> 2)) & 1u)) << 3));
    __syncthreads();   // the only CTA-wide barrier
    const uint32_t row_elems = groups[0].seg_elems;
    const uint32_t plane_elems = (R + 1) * row_elems;
    const size_t wstride = many_align(sizeof(ManyWarp<T, R>)) + many_align((size_t)2 * plane_elems * sizeof(T));
    ManyWarp<T, R>& W = *reinterpret_cast<ManyWarp<T, R>*>(smem_raw + (size_t)warp * wstride);
    T* ring = reinterpret_cast<T*>(smem_raw + (size_t)warp * wstride + many_align(sizeof(ManyWarp<T, R>)));
    if (lane == 0) {
        mbar_init(&W.bar[0], 1);
        mbar_init(&W.bar[1], 1);
        fence_barrier_init();
    }
    W.cnt[lane] = 0;
    __syncwarp();
    const uint32_t half = lane / LPR, xl = (lane % LPR) * 8;   // this lane's row of the task and first cell
    const unsigned lt = (1u << lane) - 1u;
    uint32_t lcur = 0, lend = 0;   // this warp's entries of the pair list (less than 2^31 while it is not full)
    bool lfull = false;
    uint32_t ph = 0;   // per ring buffer: parity of its next completion
    int gi = 0, gcur = -1;
    for (;;) {
        unsigned long long tk = 0;
        if (lane == 0) tk = atomicAdd(next_task, 1ull);
        const uint64_t task = __shfl_sync(FULL, tk, 0);
        if (task >= ntasks) break;
        while (gi + 1 < ngroups && task >= groups[gi + 1].task_begin) ++gi;   // (tasks come in increasing order)
        const StreamGroup& G = groups[gi];
        const int niso = G.niso;
        const float bs = G.bs, bo = G.bo;
        const uint32_t local = (uint32_t)(task - G.task_begin);
        const uint32_t cx = G.vol.nx - 1, cy = G.vol.ny - 1, cz = G.vol.nz - 1, wpr = G.wpr;
        const uint64_t pitch = G.vol.pitch, slice = G.vol.slice;
        const uint32_t cyr = (cy + R - 1) / R;
        const uint32_t rq = local / wpr, seg = local - rq * wpr;
        const uint32_t zc = rq / cyr, y = (rq - zc * cyr) * R;
        const uint32_t z0 = zc * G.zchunk;
        const uint32_t z1 = z0 + G.zchunk < cz ? z0 + G.zchunk : cz;   // cell planes [z0, z1)
        if (gi != gcur) {
            __syncwarp();
            float t = 0.0f;
            if (lane < (unsigned)niso) t = isos[G.iso_begin + lane].f.f_thr;
            thermo_build(W.th, t, niso, bs, bo, lane);
            gcur = gi;
        }
        // empty space: a brick whose node min and max have the same mask
        const float2* bricks = G.bricks;
        const uint32_t nby = (cy + 1) / 2, brick_wpr = G.brick_wpr;
        auto brick_empty = [&](uint32_t z) -> bool {
            const float2* row = bricks + ((uint64_t)(z / kBrickPlanes) * nby + (y >> 1)) * brick_wpr;
            float2 mm = row[R == 2 ? seg : 2 * seg];
            if (R == 1 && 2 * seg + 1 < brick_wpr) {   // a 256-cell segment spans two bricks
                const float2 m1 = row[2 * seg + 1];
                mm.x = fminf(mm.x, m1.x);
                mm.y = fmaxf(mm.y, m1.y);
            }
            return thermo_rank(W.th, bs, bo, mm.x) == thermo_rank(W.th, bs, bo, mm.y);
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
            T* dst = ring + (i & 1u) * plane_elems;
            const T* src = src0 + (uint64_t)i * slice;
            mbar_arrive_expect_tx(&W.bar[i & 1u], nrows * row_bytes);
            for (uint32_t r = 0; r < nrows; ++r)
                bulk_copy_g2s(dst + r * row_elems, src + r * pitch, row_bytes, &W.bar[i & 1u]);
        };
        auto acquire = [&](uint32_t i) -> bool {
            const bool ok = mbar_wait(&W.bar[i & 1u], (ph >> (i & 1u)) & 1u, wait_polls);
            if (ok) ph ^= 1u << (i & 1u);
            return ok;
        };
        uint32_t issued = nplanes < 2 ? nplanes : 2;   // planes whose copies were started
        __syncwarp();   // the previous task's reads of the ring are done
        if (lane == 0) {
            fence_proxy_async();
            for (uint32_t i = 0; i < issued; ++i) issue(i);
        }
        const bool row_ok = y + half < cy;
        // where the task's counters at plane z0 and row y lie (in shared memory: the
        // loop below has no registers to spare)
        const uint32_t plane_units = cy * wpr;
        if (lane == 0) {
            const uint64_t unit0 = ((uint64_t)z0 * cy + y) * wpr + seg;
            W.counts = unit_counts + G.unit_base + unit0 * (uint32_t)niso;
            if (LIST) {
                W.pairs = pl.unit_pairs + G.pair_base + unit0;
                W.list = pl.unit_list + G.pair_base + unit0;
            }
            if (NODES)
                W.nodes = G.node_units ? node_counts + G.node_base + ((uint64_t)z0 * G.vol.ny + y) * wpr + seg : nullptr;
        }
        // lane 16 h + k: the counter of isolevel k in row y + h
        const uint32_t ch = lane >> 4, ck = lane & 15u;
        const bool my_count = ch < (uint32_t)R && ck < (uint32_t)niso && y + ch < cy;
        const bool last_row = y + 1 == cy;
        const int lim = row_ok ? (int)cx - (int)((uint32_t)xoff + xl) : 0;   // this lane's cells inside the volume (if < 8)
        // masks of plane i's nodes into its mask rows: each lane's 8 in rows half
        // and half + 1 (left in P0, P1 too), a lane per row for the node behind the
        // last cell
        auto plane_masks = [&](uint32_t i, uint32_t* P0, uint32_t* P1) {
            const T* p = ring + (i & 1u) * plane_elems;
            uint16_t* m = W.mask[i & 1u][0];
            row_masks<T, 8>(p + half * row_elems, xl, W.th, bs, bo, P0);
            *reinterpret_cast<uint4*>(m + half * kMaskRow<R> + xl) = make_uint4(P0[0], P0[1], P0[2], P0[3]);
            row_masks<T, 8>(p + (half + 1) * row_elems, xl, W.th, bs, bo, P1);
            if (half == R - 1)
                *reinterpret_cast<uint4*>(m + R * kMaskRow<R> + xl) = make_uint4(P1[0], P1[1], P1[2], P1[3]);
            if (lane <= (unsigned)R)
                m[lane * kMaskRow<R> + SEG] = (uint16_t)thermo_mask(W.th, bs, bo, (float)p[lane * row_elems + SEG]);
        };
        bool dead = false, pa_valid = false, brick_skip = false;
        uint32_t acq = 0;
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
                break;
            }
            if (bricks && (s == 0 || z % kBrickPlanes == 0)) brick_skip = brick_empty(z);
            uint32_t PB0[4], PB1[4];
            if (!brick_skip) {
                if (!pa_valid) plane_masks(s, PB0, PB1);
                plane_masks(s + 1, PB0, PB1);
            }
            // plane z's values are consumed, and plane z + 1's once their masks are
            // formed: refill their buffers with planes z + 2 and z + 3
            __syncwarp();
            {
                uint32_t upto = brick_skip ? s + 3 : s + 4;
                if (upto > nplanes) upto = nplanes;
                if (lane == 0 && issued < upto) {
                    fence_proxy_async();
                    for (uint32_t i = issued; i < upto; ++i) issue(i);
                }
                issued = upto > issued ? upto : issued;
            }
            if (brick_skip) {
                pa_valid = false;
                continue;
            }
            // per cell: the isolevels whose threshold lies between its lowest and
            // highest corner (thermometer codes: OR = the highest, AND = the lowest)
            uint32_t act[4], m = 0;
            {
                // (plane z's masks come back from shared memory: carried in registers
                // they made the compiler spill)
                const uint16_t* ma = W.mask[s & 1u][half] + xl;
                const uint16_t* mb = W.mask[(s + 1) & 1u][half] + xl;
                const uint4 A0 = *reinterpret_cast<const uint4*>(ma);
                const uint4 A1 = *reinterpret_cast<const uint4*>(ma + kMaskRow<R>);
                const uint32_t a0 = ma[8], a1 = ma[kMaskRow<R> + 8], b0 = mb[8], b1 = mb[kMaskRow<R> + 8];
                const uint32_t co[5] = {A0.x | A1.x | PB0[0] | PB1[0], A0.y | A1.y | PB0[1] | PB1[1],
                                        A0.z | A1.z | PB0[2] | PB1[2], A0.w | A1.w | PB0[3] | PB1[3], a0 | a1 | b0 | b1};
                const uint32_t ca[5] = {A0.x & A1.x & PB0[0] & PB1[0], A0.y & A1.y & PB0[1] & PB1[1],
                                        A0.z & A1.z & PB0[2] & PB1[2], A0.w & A1.w & PB0[3] & PB1[3], a0 & a1 & b0 & b1};
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    const uint32_t o = co[w] | __funnelshift_r(co[w], co[w + 1], 16);
                    const uint32_t a = ca[w] & __funnelshift_r(ca[w], ca[w + 1], 16);
                    act[w] = o & ~a;
                    if (lim < 8) act[w] &= (2 * w < lim ? 0xffffu : 0u) | (2 * w + 1 < lim ? 0xffff0000u : 0u);
                    m += __popc(act[w]);
                }
            }
            pa_valid = true;
            uint32_t inc = m;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t t = __shfl_up_sync(FULL, inc, d);
                if (lane >= (unsigned)d) inc += t;
            }
            const uint32_t npairs = __shfl_sync(FULL, inc, 31);
            if (npairs == 0) continue;
            if (LIST) {
                if (lcur + npairs > lend) {
                    const uint32_t want = npairs > pl.run ? npairs : pl.run;
                    unsigned long long at = 0;
                    if (lane == 0) at = atomicAdd(pl.cursor, (unsigned long long)want);
                    at = __shfl_sync(FULL, at, 0);
                    lcur = (uint32_t)at;
                    lend = lcur + want;
                    if (at + want > pl.cap && !lfull) {
                        lfull = true;
                        if (lane == 0) atomicExch(pl.overflow, 1);
                    }
                }
                // each of the step's R units: its pairs, its first entry
                const uint32_t before = R == 1 ? 0u : __shfl_sync(FULL, inc, LPR - 1);
                if (lane % LPR == 0 && row_ok) {
                    const uint32_t b = half ? before : 0u;
                    const uint64_t u = (uint64_t)s * plane_units + half * wpr;
                    W.pairs[u] = (uint16_t)((R == 1 || half ? npairs : before) - b);
                    W.list[u] = lcur + b;
                }
            }
            const uint32_t my_first = inc - m;
            // the vertices of a pair's nodes behind the last row and plane
            auto far_nodes = [&](uint32_t code, uint32_t k, bool last) {
                auto cut = [&](int i, int j) -> uint32_t { return ((code >> i) ^ (code >> j)) & 1u; };
                uint32_t v = 0;
                if (last_row) v += cut(1, 5) + cut(1, 3) + (last ? cut(5, 7) : 0u);
                if (z + 1 == cz) v += (cut(2, 6) + cut(2, 3) + (last ? cut(6, 7) : 0u)) << 10;
                if (last_row && z + 1 == cz) v += cut(3, 7) << 20;
                if (v) atomicAdd(&W.cnt[16 + k], v);
            };
            // this lane's pairs (cell order, then isolevel) that fall into the buffer
            auto fill = [&](uint32_t fill0) {
                if (!m || my_first >= fill0 + kManyBuf || my_first + m <= fill0) return;
                uint32_t slot = my_first - fill0;   // (wraps below the window)
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    uint32_t am = (act[i >> 1] >> (16 * (i & 1))) & 0xffffu;
                    while (am) {
                        const uint32_t k = __ffs(am) - 1;
                        am &= am - 1;
                        if (slot < kManyBuf) W.buf[slot] = (uint16_t)((lane * 8 + i) | (k << 8));
                        ++slot;
                    }
                }
            };
            // crowded, and evenly: the lanes' own loops with a shared atomic a pair (14
            // instructions an iteration) take less than rounds of 32 pairs (60 each).
            // The noise's count alone: 1430 us by rounds, 288
            const bool crowded = npairs >= kManyCrowd && __reduce_max_sync(FULL, m) < npairs / 10;
            if (crowded) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    uint32_t am = (act[i >> 1] >> (16 * (i & 1))) & 0xffffu;
                    if (!am) continue;
                    const uint32_t x = xl + i;
                    const uint16_t* a = W.mask[s & 1u][half] + x;
                    const uint16_t* b = W.mask[(s + 1) & 1u][half] + x;
                    const uint32_t w0 = a[0] | ((uint32_t)a[1] << 16), w2 = b[0] | ((uint32_t)b[1] << 16);
                    a += kMaskRow<R>;
                    b += kMaskRow<R>;
                    const uint32_t w1 = a[0] | ((uint32_t)a[1] << 16), w3 = b[0] | ((uint32_t)b[1] << 16);
                    const bool last = NODES && xoff + x == cx - 1;
                    do {
                        const uint32_t k = __ffs(am) - 1;
                        am &= am - 1;
                        const uint32_t code = case_code(w0, w1, w2, w3, k), tab = s_tab[code];
                        uint32_t v = tab & 7u;
                        if (NODES) {
                            v += (tab >> 3) << 16;
                            if (last) v += ((((code >> 4) ^ (code >> 5)) & 1u) + (((code >> 4) ^ (code >> 6)) & 1u)) << 16;
                            if (last_row || z + 1 == cz) far_nodes(code, k, last);
                        }
                        atomicAdd(&W.cnt[half * 16 + k], v);
                    } while (am);
                }
                __syncwarp();
                for (uint32_t fill0 = 0; LIST && fill0 < npairs; fill0 += kManyBuf) {
                    fill(fill0);
                    __syncwarp();
                    for (uint32_t e = lane; e < kManyBuf && fill0 + e < npairs && !lfull; e += 32) {
                        const uint32_t v = W.buf[e];
                        pl.list[(uint64_t)lcur + fill0 + e] = (uint16_t)(((v & 0xffu) & (SEG - 1)) | (v & 0xff00u));
                    }
                    __syncwarp();
                }
            }
            for (uint32_t fill0 = 0; !crowded && fill0 < npairs; fill0 += kManyBuf) {
                fill(fill0);
                __syncwarp();
                const uint32_t nfill = npairs - fill0 < kManyBuf ? npairs - fill0 : kManyBuf;
                for (uint32_t r0 = 0; r0 < nfill; r0 += 32) {
                    const bool has = r0 + lane < nfill;
                    const uint32_t e = has ? W.buf[r0 + lane] : 0u;
                    const uint32_t h = R == 1 ? 0u : (e & 0xffu) / SEG, x = (e & 0xffu) & (SEG - 1), k = e >> 8;
                    if (LIST && has && !lfull) pl.list[(uint64_t)lcur + fill0 + r0 + lane] = (uint16_t)(x | (k << 8));
                    // corner code: bit r: row r's node x, bit 4 + r: its node x + 1
                    const uint16_t* a = W.mask[s & 1u][h] + x;
                    const uint16_t* b = W.mask[(s + 1) & 1u][h] + x;
                    const uint32_t w0 = a[0] | ((uint32_t)a[1] << 16), w2 = b[0] | ((uint32_t)b[1] << 16);
                    a += kMaskRow<R>;
                    b += kMaskRow<R>;
                    const uint32_t w1 = a[0] | ((uint32_t)a[1] << 16), w3 = b[0] | ((uint32_t)b[1] << 16);
                    const uint32_t code = case_code(w0, w1, w2, w3, k);
                    const uint32_t tab = has ? s_tab[code] : 0u, nt = tab & 7u;
                    const uint32_t key = R == 1 ? k : h * 16 + k;
                    const uint32_t grp = __match_any_sync(FULL, has ? key : 32u + lane);
                    uint32_t sum = 0;
#pragma unroll
                    for (int bit = 0; bit < 3; ++bit)
                        sum += (uint32_t)__popc(__ballot_sync(FULL, (nt >> bit) & 1u) & grp) << bit;
                    if (NODES) {
                        // the cut edges of the cell's lower node, and in the row's last cell
                        // of the node behind it
                        uint32_t nv = tab >> 3;
                        const bool last = has && xoff + x == cx - 1;
                        if (last) nv += (((code >> 4) ^ (code >> 5)) & 1u) + (((code >> 4) ^ (code >> 6)) & 1u);
#pragma unroll
                        for (int bit = 0; bit < 3; ++bit)
                            sum += (uint32_t)__popc(__ballot_sync(FULL, (nv >> bit) & 1u) & grp) << (16 + bit);
                        if (has && (last_row || z + 1 == cz)) far_nodes(code, k, last);
                    }
                    if (has && (grp & lt) == 0) W.cnt[key] += sum;   // one lane per distinct key
                    __syncwarp();
                }
            }
            lcur += npairs;
            if (my_count) {
                W.counts[((uint64_t)s * plane_units + ch * wpr) * (uint32_t)niso + ck] = (uint16_t)W.cnt[lane];
                if (NODES && W.nodes) {
                    const uint64_t plane_nodes = (uint64_t)G.vol.ny * wpr;
                    uint32_t* n = W.nodes + ck * G.node_units + s * plane_nodes;
                    const uint32_t v = W.cnt[16 + lane];
                    n[0] = W.cnt[lane] >> 16;
                    if (last_row) n[wpr] = v & 0x3ffu;
                    if (z + 1 == cz) n[plane_nodes] = (v >> 10) & 0x3ffu;
                    if (last_row && z + 1 == cz) n[plane_nodes + wpr] = v >> 20;
                }
            }
            __syncwarp();
            W.cnt[lane] = 0;
            __syncwarp();
        }
        if (dead) {
            // wait (bounded, by its own limit) for the copies still in flight, then stop
            for (uint32_t i = acq; i < issued; ++i)
                if (mbar_wait(&W.bar[i & 1u], (ph >> (i & 1u)) & 1u, 1u << 16)) ph ^= 1u << (i & 1u);
            break;
        }
    }
}

}  // namespace

#define KVSMC_MANY_SWITCH(DT, ...)                      \
    switch (DT) {                                       \
    case 0: { using T = int8_t; __VA_ARGS__; } break;   \
    case 1: { using T = int16_t; __VA_ARGS__; } break;  \
    case 4: { using T = uint8_t; __VA_ARGS__; } break;  \
    case 5: { using T = uint16_t; __VA_ARGS__; } break; \
    case 8: { using T = float; __VA_ARGS__; } break;    \
    default: return cudaErrorInvalidValue;              \
    }

cudaError_t launch_count_many(int dtype, int rows, const StreamGroup* d_groups, int ngroups, uint64_t ntasks,
                              const StreamIso* d_isos, uint16_t* d_unit_counts, int* d_status,
                              unsigned long long* d_next_task, const Launch& L, int ctas_per_sm, const PairList* list,
                              uint32_t* d_node_counts)
{
    if (ntasks == 0) return cudaSuccess;
    if (rows != 1 && (rows != 2 || d_node_counts)) return cudaErrorInvalidValue;
    const uint64_t need = (ntasks + kManyWarps - 1) / kManyWarps;
    KVSMC_MANY_SWITCH(dtype, {
        const size_t smem = kManyWarps * (many_align(rows == 1 ? sizeof(ManyWarp<T, 1>) : sizeof(ManyWarp<T, 2>)) +
                                          many_align(2 * (size_t)(rows + 1) * stream_row_elems(dtype, rows) * sizeof(T)));
        auto kern = d_node_counts ? (list ? k_count_many<T, 1, true, true> : k_count_many<T, 1, false, true>)
                    : rows == 1   ? (list ? k_count_many<T, 1, true, false> : k_count_many<T, 1, false, false>)
                                  : (list ? k_count_many<T, 2, true, false> : k_count_many<T, 2, false, false>);
        int per_sm = 0;
        const cudaError_t e = kernel_fit(L, reinterpret_cast<const void*>(kern), kManyThreads, smem, &per_sm, true);
        if (e != cudaSuccess) return e;
        if (ctas_per_sm > 0 && ctas_per_sm < per_sm) per_sm = ctas_per_sm;
        if (list && per_sm > kListWarpsPerSm / kManyWarps) per_sm = kListWarpsPerSm / kManyWarps;
        const uint64_t resident = (uint64_t)(per_sm > 0 ? per_sm : 1) * (uint64_t)L.num_sms;
        prof_begin(L, "count_many");
        kern<<<(unsigned)(need < resident ? need : resident), kManyThreads, smem, L.stream>>>(
            d_groups, ngroups, ntasks, d_isos, d_unit_counts, d_status, d_next_task, L.wait_polls[0],
            list ? *list : PairList{}, d_node_counts);
        prof_end(L);
    });
    *L.counter += 1;
    return cudaGetLastError();
}

}  // namespace kvsmc
