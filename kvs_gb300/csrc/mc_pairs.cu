// mc_pairs.cu -- the emit pass over listed cells: the count pass has already
// found every active (cell, isolevel) pair and listed it, so the triangles
// are written without classifying the volume again.
//
// The count writes, per unit (z, y, segment), its pairs in (cell, isolevel)
// order as 16-bit entries (cell in the segment | isolevel << 8) somewhere in
// one list, with the unit's first entry and their number.  A warp task here
// is a block of up to 32 consecutive units of one cell plane: lane u takes
// unit u's descriptor, a warp scan makes one index space of the block's
// pairs, and they are taken 32 at a time, one per lane, whatever unit they
// belong to.  Consecutive units' triangles of one isolevel are consecutive in
// its output, so an isolevel's position is its first unit's offset plus a
// running count.  Per round:
//   * each lane reads its cell's 8 corner values from the volume (L1/L2: a
//     cell's neighbours share its sectors), forms the corner code by 8
//     compares and leaves the values in a shared table, 9 words a cell, so that
//     the lanes of one cell reading its corners meet in different banks;
//   * lanes of the same isolevel are grouped with __match_any_sync, bit-sliced
//     ballots give each pair's output position;
//   * one lane per (pair, used edge) interpolates a vertex (the FP32
//     certificate of mc_interp.cuh) into a pool, one lane per (pair, triangle)
//     reads its three and writes the triangle.
// The rounds are full up to a block's last one (the re-classifying emit took
// the pairs of one 256-cell segment at a time: 6 of 32 lanes with one
// isolevel on smooth data), nothing waits for staged planes, and without the
// ring and the masks 32 warps are resident on an SM instead of 16.  What
// bounds it is the issue of about 1200 instructions a round and the latency of
// shuffles and shared memory between them (24 warps kept the issue slots 66%
// busy; DRAM writes are a third of its time).  So a pair's cell, code, isolevel
// and vertex base are one word, its output place and first triangle another (a
// task writes less than 2^16 triangles, so places are counted from the task's
// start and the isolevels' 64-bit addresses are formed once per task), and an
// edge's corners and axis are one byte of one table.  640x704x600 f32, 16
// isolevels: 3810 -> 3550 us (40% of the 9 GB it writes at the copy rate);
// 1024x768x640 u16, 4 isolevels: 2519 -> 2255 us.  Of that, a round's list
// entries read a round ahead: 3630 -> 3550 and 2276 -> 2255; 48 uneven volumes
// 846 -> 805.
#include <cuda_runtime.h>

#include "mc_emit.cuh"
#include "mc_internal.h"
#include "mc_interp.cuh"
#include "mc_pairs.cuh"
#include "tma.cuh"

#ifndef KVSMC_PAIRS_CTAS
#define KVSMC_PAIRS_CTAS 4
#endif

namespace kvsmc {

namespace {

__device__ PairTables d_pair_tables = make_pair_tables();

// An isolevel's constants: what a vertex needs is three 16-byte reads.  err is
// infinite where the certificate does not apply (it then decides nothing).
struct alignas(16) PairIso {
    float ih, il, err, vmin;
    float vmax, mc[3];
    float sc[3], thr;
    float* coords;
    float* normals;
    uint64_t cap_tris;
    uint64_t pad;
};
static_assert(sizeof(PairIso) == 80, "lanes of different isolevels meet in different banks");

struct alignas(16) PairOut {
    float* coords;
    float* normals;
};

template <typename V> struct alignas(16) PairWarp {
    PairIso ic[kStreamMaxIso];
    float4 pv[kPairVerts];     // vertex pool: x, y, z, unused (one 16-byte access per vertex)
    PairOut out[kStreamMaxIso];   // per isolevel: where the task's triangles go
    uint32_t room[kStreamMaxIso]; // and how many of them may be written
    V cv[32][9];               // corner values of the round's cells (9: a cell's corners in different banks)
    uint32_t add[32];          // per isolevel: triangles of the round
};

template <typename T>
__global__ void __launch_bounds__(kPairThreads, KVSMC_PAIRS_CTAS)
    k_emit_pairs(const StreamGroup* __restrict__ groups, int ngroups, uint64_t ntasks,
                 const StreamIso* __restrict__ isos, PairList pl, const uint32_t* __restrict__ unit_offsets,
                 const uint64_t* __restrict__ plane_base, int* __restrict__ status,
                 unsigned long long* __restrict__ next_task, uint32_t wait_polls, uint64_t task0,
                 const uint64_t* __restrict__ totals)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar;
    PairTables& TB = *reinterpret_cast<PairTables*>(smem_raw);
    const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    using V = typename PairValue<T>::type;
    PairWarp<V>& W = reinterpret_cast<PairWarp<V>*>(smem_raw + sizeof(PairTables))[warp];
    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_barrier_init();
        mbar_arrive_expect_tx(&bar, sizeof(PairTables));
        bulk_copy_g2s(&TB, &d_pair_tables, sizeof(PairTables), &bar);
    }
    W.add[lane] = 0;
    // nothing to write at when the count gave up or its list overflowed (the
    // caller then runs the re-classifying emit)
    const bool stop = __syncthreads_or(*status != 0 || *pl.overflow != 0);
    const bool ok = mbar_wait(&bar, 0, wait_polls);
    if (!__syncthreads_and(ok) || stop) {
        if (tid == 0) {
            if (!stop) atomicExch(status, 1);
            mbar_wait(&bar, 0, 1u << 16);   // the copy lands before the CTA leaves
        }
        return;
    }
    const unsigned lt = (1u << lane) - 1u;
    int gi = 0, gcur = -1;
    bool live = true;
    for (;;) {
        unsigned long long tk = 0;
        if (lane == 0) tk = atomicAdd(next_task, 1ull);
        const uint64_t task = task0 + __shfl_sync(FULL, tk, 0);
        if (task >= ntasks) break;
        while (gi + 1 < ngroups && task >= groups[gi + 1].etask_begin) ++gi;   // (tasks come in increasing order)
        const StreamGroup& G = groups[gi];
        if (G.skip_emit) continue;
        const int niso = G.niso, iso_begin = G.iso_begin;
        if (gi != gcur) {
            __syncwarp();
            if (lane < (unsigned)niso) {
                const StreamIso& I = isos[iso_begin + lane];
                PairIso& c = W.ic[lane];
                c.ih = I.f.ih;
                c.il = I.f.il;
                c.err = I.f.lean_ok ? I.f.iso_err : __int_as_float(0x7f800000);
                c.vmin = I.f.vmin_f;
                c.vmax = I.f.vmax_f;
                c.thr = I.f.f_thr;
                for (int a = 0; a < 3; ++a) { c.mc[a] = I.ip.min_coord[a]; c.sc[a] = I.ip.scale[a]; }
                // a request that does not fit its outputs is not written at all
                c.coords = totals && totals[iso_begin + (int)lane] > I.cap_tris ? nullptr : I.coords;
                c.normals = I.normals;
                c.cap_tris = I.cap_tris;
            }
            live = __any_sync(FULL, lane < (unsigned)niso && W.ic[lane & 15u].coords != nullptr);
            gcur = gi;
        }
        if (!live) continue;
        const uint32_t local = (uint32_t)(task - G.etask_begin);
        const uint32_t z = local / G.eblocks, u0 = (local - z * G.eblocks) * G.eblock;   // first unit in the plane
        const PairBlock B = pair_block(G, pl, z, u0, G.eblock, lane);
        if (B.npairs == 0) continue;
        // per isolevel: where the task's first triangle goes and how many fit
        __syncwarp();
        if (lane < (unsigned)niso) {
            const uint64_t pi = isos[iso_begin + lane].plane_index;
            const uint64_t at = plane_base[pi + z] - plane_base[pi] +
                                unit_offsets[G.unit_base + ((uint64_t)z * ((G.vol.ny - 1) * G.wpr) + u0) * niso + lane];
            const PairIso& c = W.ic[lane];
            W.out[lane] = PairOut{c.coords + 9 * at, c.normals + 3 * at};
            W.room[lane] = !c.coords || c.cap_tris <= at ? 0u
                           : c.cap_tris - at < 0xffffu ? (uint32_t)(c.cap_tris - at) : 0xffffu;
        }
        __syncwarp();
        uint32_t run = 0;   // lane k: the task's triangles of isolevel k so far (at most 32 * 256 * 5)
        const uint64_t pitch = G.vol.pitch, slice = G.vol.slice;
        const T* vz = static_cast<const T*>(G.vol.data) + (uint64_t)z * slice;
        const float fz = __uint2float_rn(z);
        uint32_t taken = 0;
        // the round's list entries, read a round ahead
        uint32_t next_x, next_y, next_e = 0;
        auto fetch = [&](uint32_t p0) {
            const uint32_t at = pair_entry(B, p0 + lane, next_x, next_y);
            if (p0 + lane < B.npairs) next_e = pl.list[at];
        };
        fetch(0);
        for (uint32_t r0 = 0; r0 < B.npairs; r0 += taken) {
            // ---- one pair per lane, as many as the vertex pool holds
            bool has = r0 + lane < B.npairs;
            uint32_t x = next_x;
            const uint32_t y = next_y;
            uint32_t k = 0, code = 0;
            if (has) {
                x += next_e & 0xffu;
                k = next_e >> 8;
                code = pair_corners<T, V>(vz + (uint64_t)y * pitch + x, pitch, slice, W.cv[lane], [&](T v) -> bool {
                    if constexpr (kPairFast<T>) return (float)v > W.ic[k].thr;
                    else return above(isos[iso_begin].cls, v);   // (one isolevel per group)
                });
            }
            const float fy = __uint2float_rn(y);   // (rows below 2^24: exact)
            const uint32_t cnt = has ? TB.counts[code] : 0u;
            const uint32_t ne0 = cnt >> 3;
            uint32_t vpre = 0;
#pragma unroll
            for (int bit = 0; bit < 4; ++bit)
                vpre += (uint32_t)__popc(__ballot_sync(FULL, (ne0 >> bit) & 1u) & lt) << bit;
            has = has && vpre + ne0 <= (uint32_t)kPairVerts;   // a suffix of lanes waits
            taken = (uint32_t)__popc(__ballot_sync(FULL, has));
            const uint32_t nv = __shfl_sync(FULL, vpre + ne0, taken - 1);
            if (r0 + taken < B.npairs) fetch(r0 + taken);
            const uint32_t nt = has ? cnt & 7u : 0u;
            const uint32_t pe = x | (k << 12) | (code << 16) | (vpre << 24);   // (x < 4096; vpre < kPairVerts)
            // output position of the pair's first triangle: its isolevel's running
            // count plus the triangles of the earlier lanes of that isolevel
            const uint32_t grp = niso == 1 ? __ballot_sync(FULL, has) : __match_any_sync(FULL, has ? k : 32u + lane);
            uint32_t pre = 0, gtot = 0, tpre = 0, ntr = 0;
#pragma unroll
            for (int bit = 0; bit < 3; ++bit) {
                const uint32_t bm = __ballot_sync(FULL, (nt >> bit) & 1u);
                pre += (uint32_t)__popc(bm & grp & lt) << bit;
                gtot += (uint32_t)__popc(bm & grp) << bit;
                tpre += (uint32_t)__popc(bm & lt) << bit;
                ntr += (uint32_t)__popc(bm) << bit;
            }
            const uint32_t ot = __shfl_sync(FULL, run, k) + pre + (tpre << 16);   // (both below 2^16)
            if (niso == 1) {
                run += ntr;
            } else {
                if (has && (31 - __clz(grp)) == (int)lane) W.add[k] = gtot;
                __syncwarp();
                run += W.add[lane];
                W.add[lane] = 0;
            }
            __syncwarp();   // the corner values are there
            // ---- vertices: one (pair, used edge) per lane.  Item j's pair: the
            // pairs' first items as bits of one word (every pair has items), so
            // the pair is the number of first items up to j
            uint32_t seen = 0;
            for (uint32_t j0 = 0; j0 < nv; j0 += 32) {
                const uint32_t j = j0 + lane;
                const bool hv = j < nv;
                const uint32_t starts = __reduce_or_sync(FULL, has && vpre - j0 < 32u ? 1u << (vpre - j0) : 0u);
                const uint32_t q = seen + (uint32_t)__popc(starts & (lt | (1u << lane))) - 1u;
                seen += (uint32_t)__popc(starts);
                const uint32_t qe = __shfl_sync(FULL, pe, q);
                const float qy = __shfl_sync(FULL, fy, q);
                const uint32_t ed = TB.edges[(qe >> 16) & 255u][hv ? j - (qe >> 24) : 0u];
                const uint32_t c0 = ed & 7u, c1 = (ed >> 3) & 7u;
                const int axis = (int)(ed >> 6);
                const V va = W.cv[q][c0], vb = W.cv[q][c1];
                const uint32_t qx = qe & 0xfffu, qk = (qe >> 12) & 15u;
                // corner coordinates: integers below 2^24, exact as floats
                const float ax = __uint2float_rn(qx + (c0 & 1u)), ay = __fadd_rn(qy, (c0 & 2u) ? 1.0f : 0.0f);
                const float az = __fadd_rn(fz, (c0 & 4u) ? 1.0f : 0.0f);
                const bool up = c1 > c0;
                float3 v;
                if constexpr (kPairFast<T>) {
                    const float a = axis == 0 ? ax : (axis == 1 ? ay : az);
                    const float4* ic = reinterpret_cast<const float4*>(&W.ic[qk]);
                    const float4 i0 = ic[0], i1 = ic[1], i2 = ic[2];
                    FastIso f;
                    f.ih = i0.x;
                    f.il = i0.y;
                    f.iso_err = i0.z;
                    f.vmin_f = i0.w;
                    f.vmax_f = i1.x;
                    f.lean_ok = 1;
                    float r;
                    const bool good = fast_axis_lean<(sizeof(T) < 4)>(va, vb, a, up, f, r);
                    v.x = __fmul_rn(__fadd_rn(axis == 0 ? r : ax, i1.y), i2.x);
                    v.y = __fmul_rn(__fadd_rn(axis == 1 ? r : ay, i1.z), i2.y);
                    v.z = __fmul_rn(__fadd_rn(axis == 2 ? r : az, i1.w), i2.z);
                    if (hv && !good) {   // (about one in 10^5) the exact FP64 sequence
                        const StreamIso& I = isos[iso_begin + qk];
                        v = edge_vertex_axis(I.f, I.ip.min_coord, I.ip.scale, I.ip, va, vb, ax, ay, az, axis,
                                             __fadd_rn(a, up ? 1.0f : -1.0f));
                    }
                } else {
                    const float d = up ? 1.0f : -1.0f;
                    v = interpolate_exact_axis(isos[iso_begin].ip, va, vb, ax, ay, az, axis == 0 ? __fadd_rn(ax, d) : ax,
                                               axis == 1 ? __fadd_rn(ay, d) : ay, axis == 2 ? __fadd_rn(az, d) : az, axis);
                }
                if (hv) W.pv[j] = make_float4(v.x, v.y, v.z, 0.0f);
            }
            __syncwarp();
            // ---- triangles: one (pair, triangle) per lane, table order
            seen = 0;
            for (uint32_t j0 = 0; j0 < ntr; j0 += 32) {
                const uint32_t j = j0 + lane;
                const bool ht = j < ntr;
                const uint32_t starts = __reduce_or_sync(FULL, has && tpre - j0 < 32u ? 1u << (tpre - j0) : 0u);
                const uint32_t q = seen + (uint32_t)__popc(starts & (lt | (1u << lane))) - 1u;
                seen += (uint32_t)__popc(starts);
                const uint32_t qe = __shfl_sync(FULL, pe, q);
                const uint32_t qo = __shfl_sync(FULL, ot, q);
                if (ht) {
                    const uint32_t t = j - (qo >> 16), o = (qo & 0xffffu) + t, qk = (qe >> 12) & 15u;
                    const uint32_t sl = (uint32_t)(TB.tri_slots[(qe >> 16) & 255u] >> (12 * t));
                    const float4* pv = W.pv + (qe >> 24);
                    const float4 fa = pv[sl & 15u], fb = pv[(sl >> 4) & 15u], fc = pv[(sl >> 8) & 15u];
                    const float3 A = make_float3(fa.x, fa.y, fa.z), B = make_float3(fb.x, fb.y, fb.z);
                    const float3 C = make_float3(fc.x, fc.y, fc.z);
                    if (o < W.room[qk]) {
                        const PairOut to = W.out[qk];
                        store_triangle(to.coords + 9 * o, to.normals + 3 * o, A, B, C, tri_normal(A, B, C));
                    }
                }
            }
            __syncwarp();
        }
    }
}

}  // namespace

cudaError_t launch_emit_pairs(int dtype, const StreamGroup* d_groups, int ngroups, uint64_t ntasks,
                              const StreamIso* d_isos, const PairList& list, const uint32_t* d_unit_offsets,
                              const uint64_t* d_plane_base, int* d_status, unsigned long long* d_next_task,
                              const Launch& L, uint64_t task0, const uint64_t* d_totals)
{
    if (ntasks <= task0) return cudaSuccess;
    const uint64_t need = (ntasks - task0 + kPairWarps - 1) / kPairWarps;
    const void* kern = nullptr;
    size_t smem = sizeof(PairTables);
#define KVSMC_PAIR_CASE(CODE, T)                                                     \
    case CODE:                                                                       \
        kern = reinterpret_cast<const void*>(k_emit_pairs<T>);                       \
        smem += kPairWarps * sizeof(PairWarp<typename PairValue<T>::type>);          \
        break;
    switch (dtype) {
        KVSMC_PAIR_CASE(0, int8_t)
        KVSMC_PAIR_CASE(1, int16_t)
        KVSMC_PAIR_CASE(2, int32_t)
        KVSMC_PAIR_CASE(3, long long)
        KVSMC_PAIR_CASE(4, uint8_t)
        KVSMC_PAIR_CASE(5, uint16_t)
        KVSMC_PAIR_CASE(6, uint32_t)
        KVSMC_PAIR_CASE(7, unsigned long long)
        KVSMC_PAIR_CASE(8, float)
        KVSMC_PAIR_CASE(9, double)
    default: break;
    }
#undef KVSMC_PAIR_CASE
    if (!kern) return cudaErrorInvalidValue;
    int per_sm = 0;
    cudaError_t e = kernel_fit(L, kern, kPairThreads, smem, &per_sm);
    if (e != cudaSuccess) return e;
    const uint64_t resident = (uint64_t)(per_sm > 0 ? per_sm : 1) * (uint64_t)L.num_sms;
    uint32_t polls = L.wait_polls[1];
    PairList pl = list;
    void* args[] = {&d_groups, &ngroups, &ntasks, &d_isos, &pl, &d_unit_offsets, &d_plane_base, &d_status,
                    &d_next_task, &polls, &task0, &d_totals};
    prof_begin(L, "stream_emit");
    e = cudaLaunchKernel(kern, dim3((unsigned)(need < resident ? need : resident)), dim3(kPairThreads), args, smem,
                         L.stream);
    prof_end(L);
    *L.counter += 1;
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace kvsmc
