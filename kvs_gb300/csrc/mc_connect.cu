// mc_connect.cu -- the shared-vertex modes over listed pairs: calculate_isopoints
// (MarchingCubes.cpp:366-446), connect_isopoints (:456-521) and the vertex
// normals (:569-605) from the crossed cells that the count pass listed.
//
// Tasks, blocks and rounds are mc_pairs.cu's.  In the connection pass a round's vertex items (one per
// (pair, used edge), 4 to 5 a pair) each read the rank word of the edge's lower
// node, which gives the vertex id, and have the vertex itself by interpolating
// it again from the corner values at hand (the same certified bits; a read of
// it would depend on the id's and cost another trip to L2; the few that the
// certificate cannot decide, and the wide types, are read).  The triangle items
// take ids and positions from the pool.
//
// Vertex normals are sums of the triangles' normals in triangle order.  An edge
// has at most four cells around it, in z, y, x order, and a cell's triangles
// are consecutive, so the order is known from where a cell lies: the vertex
// items write each cell's first triangle and which of its triangles use the
// edge (at most 5) to the vertex's slot of that cell, no atomics, no sort, and
// the sum walks the four slots.  (Every case uses all of its cut edges, so a
// slot is written for each cell there is.)
//
// Bound by latency: three dependent trips (list entry, corner values, rank
// word) with 24 warps an SM; 32 (64 registers, and less L1) take 771 us, 24
// 745.  385x320x352 f32, 8 isolevels with vertex normals: classifying
// connection pass 857 us, then lists by atomics 332 and sorted sums 303; now
// 727 and 242 (745 before a round's list entries were read a round ahead).
#include <cuda_runtime.h>

#include "mc_device.cuh"
#include "mc_emit.cuh"
#include "mc_internal.h"
#include "mc_interp.cuh"
#include "mc_pairs.cuh"
#include "mc_slots.cuh"
#include "tma.cuh"

namespace kvsmc {

namespace {

constexpr PairTables h_conn_tables = make_pair_tables();

constexpr bool every_cut_edge_is_used()
{
    for (int c = 0; c < 256; ++c)
        for (int e = 0; e < (h_conn_tables.counts[c] >> 3); ++e)
            if (!h_conn_tables.users[c][e]) return false;
    for (int c = 0; c < 256; ++c) {   // and the used ones are the cut ones
        int cut = 0;
        for (int e = 0; e < 12; ++e) {
            const int c0 = h_edge[e] & 7, c1 = h_edge[e] >> 3;
            // corner dx + 2 dy + 4 dz -> bit of the corner code
            const int b0 = (c0 >> 1) | ((c0 & 1) << 2), b1 = (c1 >> 1) | ((c1 & 1) << 2);
            cut += ((c >> b0) ^ (c >> b1)) & 1;
        }
        if (cut != (h_conn_tables.counts[c] >> 3)) return false;
    }
    return true;
}
static_assert(every_cut_edge_is_used(), "a vertex has a slot written by each of its cells");

__device__ PairTables d_conn_tables = make_pair_tables();

// A request's constants, 144 bytes apart: lanes of different requests reading
// one field meet in different banks.
struct __align__(16) ConnConst {
    FastIso f;
    float mc[3], sc[3];
    uint64_t ntri;
    const uint4* rank;
    const float* coords;
    uint32_t* connections;
    float* tri_out;
    float4* tri4;
    uint2* slots;
    uint32_t nvert, enabled, pad[6];
};
static_assert(sizeof(ConnConst) == 144, "bank stride");

template <typename V> struct alignas(16) ConnWarp {
    float4 pv[kPairVerts];          // vertex pool: x, y, z, id
    V cv[32][9];                    // corner values of the round's cells
    uint64_t first[kStreamMaxIso];  // per isolevel: the task's first triangle
    uint32_t add[32];               // per isolevel: triangles of the round
};

template <typename T>
__global__ void __launch_bounds__(kPairThreads, 3)
    k_connect_pairs(const StreamGroup* __restrict__ groups, const StreamIso* __restrict__ isos,
                    const __grid_constant__ ConnTable conn, PairList pl, const uint32_t* __restrict__ unit_offsets,
                    const uint64_t* __restrict__ plane_base, uint64_t ntasks, uint32_t words_per_row,
                    int* __restrict__ status, unsigned long long* __restrict__ next_task, uint32_t wait_polls)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ ConnConst s_iso[kStreamMaxIso];
    PairTables& TB = *reinterpret_cast<PairTables*>(smem_raw);
    const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    using V = typename PairValue<T>::type;
    ConnWarp<V>& W = reinterpret_cast<ConnWarp<V>*>(smem_raw + sizeof(PairTables))[warp];
    const StreamGroup& G = groups[0];
    const uint32_t niso = (uint32_t)G.niso;
    const int iso_begin = G.iso_begin;
    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_barrier_init();
        mbar_arrive_expect_tx(&bar, sizeof(PairTables));
        bulk_copy_g2s(&TB, &d_conn_tables, sizeof(PairTables), &bar);
    }
    if (tid < niso) {
        const StreamIso& I = isos[iso_begin + tid];
        const ConnIso& c = conn.iso[tid];
        ConnConst& k = s_iso[tid];
        k.f = I.f;
        for (int a = 0; a < 3; ++a) { k.mc[a] = I.ip.min_coord[a]; k.sc[a] = I.ip.scale[a]; }
        k.ntri = c.ntri;
        k.rank = c.rank;
        k.coords = c.coords;
        k.connections = c.connections;
        k.tri_out = c.tri_out;
        k.tri4 = c.tri4;
        k.slots = c.slots;
        k.nvert = (uint32_t)c.nvert;
        k.enabled = c.enabled;
    }
    W.add[lane] = 0;
    // the node emit gave up (its rank words and vertices are not all there), or
    // the list is not complete
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
    const uint32_t ny = G.vol.ny;
    const uint64_t pitch = G.vol.pitch, slice = G.vol.slice;
    for (;;) {
        unsigned long long tk = 0;
        if (lane == 0) tk = atomicAdd(next_task, 1ull);
        const uint64_t task = __shfl_sync(FULL, tk, 0);
        if (task >= ntasks) break;
        const uint32_t z = (uint32_t)task / G.eblocks, u0 = ((uint32_t)task - z * G.eblocks) * G.eblock;
        const PairBlock B = pair_block(G, pl, z, u0, G.eblock, lane);
        if (B.npairs == 0) continue;
        __syncwarp();
        if (lane < niso) {
            const uint64_t pi = isos[iso_begin + lane].plane_index;
            W.first[lane] = plane_base[pi + z] - plane_base[pi] +
                            unit_offsets[G.unit_base + ((uint64_t)z * ((ny - 1) * G.wpr) + u0) * niso + lane];
        }
        __syncwarp();
        uint32_t run = 0;   // lane k: the task's triangles of isolevel k so far (at most 32 * 256 * 5)
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
                    if constexpr (kPairFast<T>) return (float)v > s_iso[k].f.f_thr;
                    else return above(isos[iso_begin].cls, v);   // (one isolevel per group)
                });
            }
            const bool on = has && s_iso[k].enabled;
            const uint32_t cnt = on ? TB.counts[code] : 0u;
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
            const bool item = has && ne0 != 0;   // (a pair of a request that is not written has none)
            const uint32_t pe = x | (k << 12) | (code << 16) | (vpre << 24);   // (x < 4096; vpre < kPairVerts)
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
            // lanes with items in lane order: item j's pair is the number of
            // first items up to j, counted among them
            const uint32_t items = __ballot_sync(FULL, item);
            const bool gaps = (uint32_t)__popc(items) != taken;
            // ---- vertices: one (pair, used edge) per lane
            uint32_t seen = 0;
            for (uint32_t j0 = 0; j0 < nv; j0 += 32) {
                const uint32_t j = j0 + lane;
                const bool hv = j < nv;
                const uint32_t starts = __reduce_or_sync(FULL, item && vpre - j0 < 32u ? 1u << (vpre - j0) : 0u);
                uint32_t q = seen + (uint32_t)__popc(starts & (lt | (1u << lane))) - 1u;
                seen += (uint32_t)__popc(starts);
                if (gaps) q = nth_set_bit(items, q) & 31u;
                const uint32_t qe = __shfl_sync(FULL, pe, q);
                const uint32_t qy = __shfl_sync(FULL, y, q);
                const uint32_t qo = __shfl_sync(FULL, ot, q);
                const uint32_t qcode = (qe >> 16) & 255u, r = hv ? j - (qe >> 24) : 0u;
                const uint32_t ed = TB.edges[qcode][r];
                const uint32_t nd = ed & (ed >> 3) & 7u;   // the lower corner: bits of both
                const uint32_t axis = ed >> 6;
                const uint32_t qk = (qe >> 12) & 15u;
                const ConnConst& I = s_iso[qk];
                const uint32_t lx = (qe & 0xfffu) + (nd & 1u), ly = qy + ((nd >> 1) & 1u), lz = z + (nd >> 2);
                if (hv) {
                    const uint4 R = __ldg(I.rank + ((uint64_t)lz * ny + ly) * words_per_row + (lx >> 5));
                    const V va = W.cv[q][nd], vb = W.cv[q][nd | (1u << axis)];
                    const float ax = __uint2float_rn(lx), ay = __uint2float_rn(ly);
                    const float az = __fadd_rn(fz, (nd & 4u) ? 1.0f : 0.0f);
                    float3 v = make_float3(0.0f, 0.0f, 0.0f);
                    bool good = false;
                    if constexpr (kPairFast<T>) {
                        const float a = axis == 0 ? ax : (axis == 1 ? ay : az);
                        float w;
                        good = fast_axis_lean<(sizeof(T) < 4)>(va, vb, a, true, I.f, w);
                        v.x = __fmul_rn(__fadd_rn(axis == 0 ? w : ax, I.mc[0]), I.sc[0]);
                        v.y = __fmul_rn(__fadd_rn(axis == 1 ? w : ay, I.mc[1]), I.sc[1]);
                        v.z = __fmul_rn(__fadd_rn(axis == 2 ? w : az, I.mc[2]), I.sc[2]);
                    }
                    const uint32_t bit = lx & 31u, ltb = (1u << bit) - 1u;
                    uint32_t id = R.w + __popc(R.x & ltb) + __popc(R.y & ltb) + __popc(R.z & ltb);
                    if (axis >= 1) id += (R.x >> bit) & 1u;
                    if (axis >= 2) id += (R.y >> bit) & 1u;
                    if (id < I.nvert) {
                        if (!good) {
                            const float* c = I.coords + 3 * (uint64_t)id;
                            v = make_float3(c[0], c[1], c[2]);
                        }
                        if (I.slots) {
                            // the cell's place among the edge's four, in z, y, x order
                            const uint32_t at2 = axis == 0 ? nd >> 1 : (axis == 1 ? (nd & 1u) | ((nd >> 1) & 2u) : nd & 3u);
                            I.slots[4 * (uint64_t)id + (3u - at2)] =
                                make_uint2((uint32_t)W.first[qk] + (qo & 0xffffu), TB.users[qcode][r]);
                        }
                    }
                    W.pv[j] = make_float4(v.x, v.y, v.z, __uint_as_float(id));
                }
            }
            __syncwarp();
            // ---- triangles: one (pair, triangle) per lane, table order
            seen = 0;
            for (uint32_t j0 = 0; j0 < ntr; j0 += 32) {
                const uint32_t j = j0 + lane;
                const uint32_t starts = __reduce_or_sync(FULL, item && tpre - j0 < 32u ? 1u << (tpre - j0) : 0u);
                uint32_t q = seen + (uint32_t)__popc(starts & (lt | (1u << lane))) - 1u;
                seen += (uint32_t)__popc(starts);
                if (gaps) q = nth_set_bit(items, q) & 31u;
                const uint32_t qe = __shfl_sync(FULL, pe, q);
                const uint32_t qo = __shfl_sync(FULL, ot, q);
                if (j < ntr) {
                    const uint32_t t = j - (qo >> 16), qk = (qe >> 12) & 15u;
                    const uint32_t sl = (uint32_t)(TB.tri_slots[(qe >> 16) & 255u] >> (12 * t));
                    const float4* pv = W.pv + (qe >> 24);
                    const float4 fa = pv[sl & 15u], fb = pv[(sl >> 4) & 15u], fc = pv[(sl >> 8) & 15u];
                    const uint32_t ia = __float_as_uint(fa.w), ib = __float_as_uint(fb.w), ic = __float_as_uint(fc.w);
                    const ConnConst& I = s_iso[qk];
                    const uint64_t tt = W.first[qk] + (qo & 0xffffu) + t;
                    if (tt >= I.ntri || ia >= I.nvert || ib >= I.nvert || ic >= I.nvert) {
                        atomicExch(status, 2);   // never with consistent rank words; nothing is written out of range
                    } else {
                        uint32_t* o = I.connections + 3 * tt;
                        o[0] = ia; o[1] = ib; o[2] = ic;
                        const float3 n = tri_normal(make_float3(fa.x, fa.y, fa.z), make_float3(fb.x, fb.y, fb.z),
                                                    make_float3(fc.x, fc.y, fc.z));
                        if (I.tri4) {
                            I.tri4[tt] = make_float4(n.x, n.y, n.z, 0.0f);
                        } else if (I.tri_out) {
                            float* w = I.tri_out + 3 * tt;
                            w[0] = n.x; w[1] = n.y; w[2] = n.z;
                        }
                    }
                }
            }
            __syncwarp();
        }
    }
}

// calculate_isopoints (MarchingCubes.cpp:366-446) over listed pairs: the
// vertices and rank words that mc_snode.cu's kernels write, from the cells that
// the count found.  A node's cut edges make its cell (the one it is the lower
// corner of) a listed pair; the nodes behind the last cell of a row belong to
// that cell's item list, those of the last row and plane to tasks of their own,
// which walk the last cell row's or plane's pairs for the nodes at their far
// side.  So a task's pairs are its vertices in id order, and a round numbers
// them as the emit numbers triangles.  A round's pairs of one (unit, isolevel,
// 32-node word) collect the word's flags in shared memory; the first of them
// stores the word, with its own first vertex as the word's; a word that goes on
// in the next round gets the rest by atomics.
// 385x320x352 f32, 8 isolevels: 711 us classifying every node again, 291 us.
struct __align__(16) NodeConst {
    FastIso f;
    float mc[3], sc[3];
    float* coords;
    uint4* rank;
    uint2* slots;
    const uint64_t* offsets;
    uint64_t pad[3];
};
static_assert(sizeof(NodeConst) == 112, "bank stride");

template <typename V> struct alignas(16) NodeWarp {
    V cv[32][9];                    // corner values of the round's cells
    uint64_t first[kStreamMaxIso];  // per isolevel: the task's first vertex
    uint32_t add[kStreamMaxIso];    // per isolevel: vertices of the round,
    uint32_t last[kStreamMaxIso];   // and the word of its last pair so far
    uint32_t flags[32][3];          // per leading lane: the word's x, y, z flags
};

template <typename T>
__global__ void __launch_bounds__(kPairThreads, 4)
    k_nodes_pairs(const StreamGroup* __restrict__ groups, const StreamIso* __restrict__ isos,
                  const __grid_constant__ NodeTable nodes, PairList pl, uint64_t ntasks, uint32_t words_per_row,
                  int* __restrict__ status, unsigned long long* __restrict__ next_task)
{
    using V = typename PairValue<T>::type;
    __shared__ NodeConst s_iso[kStreamMaxIso];
    __shared__ NodeWarp<V> sw[kPairWarps];
    const unsigned tid = threadIdx.x, lane = tid & 31u;
    NodeWarp<V>& W = sw[tid >> 5];
    const StreamGroup& G = groups[0];
    const uint32_t niso = (uint32_t)G.niso;
    const int iso_begin = G.iso_begin;
    if (tid < niso) {
        const StreamIso& I = isos[iso_begin + tid];
        const NodeOut& o = nodes.iso[tid];
        NodeConst& k = s_iso[tid];
        k.f = I.f;
        for (int a = 0; a < 3; ++a) { k.mc[a] = I.ip.min_coord[a]; k.sc[a] = I.ip.scale[a]; }
        k.coords = o.coords;
        k.rank = o.rank;
        k.slots = o.slots;
        k.offsets = o.offsets;
    }
    if (__syncthreads_or(*status != 0 || *pl.overflow != 0)) return;   // the list is not complete
    const unsigned lt = (1u << lane) - 1u;
    const uint32_t nx = G.vol.nx, ny = G.vol.ny, nz = G.vol.nz, wpr = G.wpr;
    const uint64_t pitch = G.vol.pitch, slice = G.vol.slice;
    for (;;) {
        unsigned long long tk = 0;
        if (lane == 0) tk = atomicAdd(next_task, 1ull);
        const uint64_t task = __shfl_sync(FULL, tk, 0);
        if (task >= ntasks) break;
        // (node plane, block of units); the last block of a plane is the nodes
        // behind the last cell row, the last plane those behind the last cell plane
        const uint32_t per = G.eblocks + 1;
        const uint32_t zn = (uint32_t)task / per, e = (uint32_t)task - zn * per;
        const bool far_y = e == G.eblocks, far_z = zn == nz - 1;
        const uint32_t z = far_z ? zn - 1 : zn;   // cell plane
        const uint32_t u0 = far_y ? (ny - 2) * wpr : e * G.eblock;
        const PairBlock B = pair_block(G, pl, z, u0, far_y ? wpr : G.eblock, lane);
        if (B.npairs == 0) continue;
        const uint32_t row = (far_y ? 1u : 0u) | (far_z ? 2u : 0u);   // the node's row among the cell's four
        __syncwarp();
        if (lane < niso) {
            const uint64_t* off = s_iso[lane].offsets;
            W.first[lane] = s_iso[lane].coords ? off[((uint64_t)zn * ny + (u0 / wpr + (far_y ? 1u : 0u))) * wpr + u0 % wpr] - off[0] : 0;
            W.last[lane] = 0xffffffffu;
            W.add[lane] = 0;
        }
        __syncwarp();
        uint32_t run = 0;   // lane k: the task's vertices of isolevel k so far
        const T* vz = static_cast<const T*>(G.vol.data) + (uint64_t)z * slice;
        const float fz = __uint2float_rn(zn);
        uint32_t next_x, next_y, next_e = 0;
        auto fetch = [&](uint32_t p0) {
            const uint32_t at = pair_entry(B, p0 + lane, next_x, next_y);
            if (p0 + lane < B.npairs) next_e = pl.list[at];
        };
        fetch(0);
        for (uint32_t r0 = 0; r0 < B.npairs; r0 += 32) {
            // ---- one pair per lane
            bool has = r0 + lane < B.npairs;
            uint32_t x = next_x, y = next_y;
            uint32_t k = 0, cut = 0;
            if (has) {
                x += next_e & 0xffu;
                k = next_e >> 8;
                const uint32_t code = pair_corners<T, V>(vz + (uint64_t)y * pitch + x, pitch, slice, W.cv[lane],
                                                         [&](T v) -> bool {
                    if constexpr (kPairFast<T>) return (float)v > s_iso[k].f.f_thr;
                    else return above(isos[iso_begin].cls, v);   // (one isolevel per group)
                });
                has = s_iso[k].coords != nullptr;
                // the node's cut edges (code bit r: row r at x, 4 + r: at x + 1)
                const uint32_t n = code >> row, f = code >> (4 + row);
                cut = (n ^ f) & 1u;
                if (!far_y) cut |= ((n ^ (n >> 1)) & 1u) << 1;
                if (!far_z) cut |= ((n ^ (n >> 2)) & 1u) << 2;
                if (x + 2 == nx) {   // and those of the row's last node
                    if (!far_y) cut |= ((f ^ (f >> 1)) & 1u) << 3;
                    if (!far_z) cut |= ((f ^ (f >> 2)) & 1u) << 4;
                }
                if (!has) cut = 0;
            }
            if (r0 + 32 < B.npairs) fetch(r0 + 32);
            y += far_y ? 1u : 0u;   // the node's
            const uint32_t nv0 = (uint32_t)__popc(cut);
            const uint32_t kgrp = niso == 1 ? __ballot_sync(FULL, has) : __match_any_sync(FULL, has ? k : 32u + lane);
            uint32_t pre = 0, gtot = 0, vpre = 0, nv = 0;
#pragma unroll
            for (int bit = 0; bit < 3; ++bit) {
                const uint32_t bm = __ballot_sync(FULL, (nv0 >> bit) & 1u);
                pre += (uint32_t)__popc(bm & kgrp & lt) << bit;
                gtot += (uint32_t)__popc(bm & kgrp) << bit;
                vpre += (uint32_t)__popc(bm & lt) << bit;
                nv += (uint32_t)__popc(bm) << bit;
            }
            const uint32_t start = __shfl_sync(FULL, run, k) + pre;   // the pair's first vertex, from the task's
            // ---- rank words
            const uint32_t word = y * words_per_row + (x >> 5);   // (in the node plane)
            const uint32_t wgrp = __match_any_sync(FULL, has ? word : 0xffffffffu - lane) & kgrp;
            const int leader = __ffs(wgrp) - 1;
            W.flags[lane][0] = 0;
            W.flags[lane][1] = 0;
            W.flags[lane][2] = 0;
            __syncwarp();
            const bool split = (x & 31u) == 31u;   // the row's last node opens a word of its own
            if (has) {
                const uint32_t bit = 1u << (x & 31u);
#pragma unroll
                for (int a = 0; a < 3; ++a)
                    if ((cut >> a) & 1u) atomicOr(&W.flags[leader][a], bit);
                if ((cut >> 3) && !split) {
                    if (cut & 8u) atomicOr(&W.flags[leader][1], bit << 1);
                    if (cut & 16u) atomicOr(&W.flags[leader][2], bit << 1);
                }
            }
            __syncwarp();
            if (has && (int)lane == leader) {
                const NodeConst& I = s_iso[k];
                uint4* R = I.rank + (uint64_t)zn * ny * words_per_row + word;
                const uint32_t fx = W.flags[lane][0], fy = W.flags[lane][1], fz3 = W.flags[lane][2];
                if (W.last[k] != word) {
                    *R = make_uint4(fx, fy, fz3, (uint32_t)(W.first[k] + start));
                } else {   // begun in the round before
                    if (fx) atomicOr(&R->x, fx);
                    if (fy) atomicOr(&R->y, fy);
                    if (fz3) atomicOr(&R->z, fz3);
                }
            }
            if ((cut >> 3) && split)
                s_iso[k].rank[(uint64_t)zn * ny * words_per_row + word + 1] =
                    make_uint4(0, (cut >> 3) & 1u, cut >> 4, (uint32_t)(W.first[k] + start) + (uint32_t)__popc(cut & 7u));
            __syncwarp();   // the words before are read
            if (has && (31 - __clz(kgrp)) == (int)lane) {
                W.add[k] = gtot;
                W.last[k] = word;
            }
            __syncwarp();
            if (lane < kStreamMaxIso) {
                run += W.add[lane];
                W.add[lane] = 0;
            }
            __syncwarp();
            // ---- vertices: one per lane, from the corner values
            const uint32_t pe = x | (k << 12) | (cut << 16) | (vpre << 21);   // (x < 4096; vpre <= 160)
            const uint32_t items = __ballot_sync(FULL, nv0 != 0);
            uint32_t seen = 0;
            for (uint32_t j0 = 0; j0 < nv; j0 += 32) {
                const uint32_t j = j0 + lane;
                const uint32_t starts = __reduce_or_sync(FULL, nv0 && vpre - j0 < 32u ? 1u << (vpre - j0) : 0u);
                const uint32_t nth = seen + (uint32_t)__popc(starts & (lt | (1u << lane)));   // 1 ..
                seen += (uint32_t)__popc(starts);
                const uint32_t q = nth_set_bit(items, nth - 1u) & 31u;
                const uint32_t qe = __shfl_sync(FULL, pe, q), qy = __shfl_sync(FULL, y, q);
                const uint32_t qs = __shfl_sync(FULL, start, q);
                if (j < nv) {
                    const uint32_t r = j - (qe >> 21), qk = (qe >> 12) & 15u;
                    uint32_t m = (qe >> 16) & 31u;
#pragma unroll
                    for (uint32_t i = 0; i < 4; ++i)
                        if (i < r) m &= m - 1u;
                    const uint32_t ed = (uint32_t)__ffs(m) - 1u;          // 0 .. 2 the node's, 3, 4 the last node's y and z
                    const uint32_t far_x = ed >= 3u ? 1u : 0u, axis = ed - 2u * far_x;
                    const uint32_t c0 = far_x | ((row & 1u) << 1) | ((row & 2u) << 1);
                    const V va = W.cv[q][c0], vb = W.cv[q][c0 | (1u << axis)];
                    const uint32_t lx = (qe & 0xfffu) + far_x;
                    const float ax = __uint2float_rn(lx), ay = __uint2float_rn(qy);
                    const NodeConst& I = s_iso[qk];
                    float3 v;
                    bool good = false;
                    if constexpr (kPairFast<T>) {
                        const float a = axis == 0 ? ax : (axis == 1 ? ay : fz);
                        float w;
                        good = fast_axis_lean<(sizeof(T) < 4)>(va, vb, a, true, I.f, w);
                        v.x = __fmul_rn(__fadd_rn(axis == 0 ? w : ax, I.mc[0]), I.sc[0]);
                        v.y = __fmul_rn(__fadd_rn(axis == 1 ? w : ay, I.mc[1]), I.sc[1]);
                        v.z = __fmul_rn(__fadd_rn(axis == 2 ? w : fz, I.mc[2]), I.sc[2]);
                    }
                    if (!good) {   // the exact FP64 sequence
                        const float bx = axis == 0 ? __fadd_rn(ax, 1.0f) : ax, by = axis == 1 ? __fadd_rn(ay, 1.0f) : ay;
                        const float bz = axis == 2 ? __fadd_rn(fz, 1.0f) : fz;
                        if constexpr (kPairFast<T>)
                            v = edge_vertex_fast(isos[iso_begin + qk].ip, I.f, va, vb, ax, ay, fz, bx, by, bz, (int)axis);
                        else
                            v = interpolate_exact_axis(isos[iso_begin].ip, va, vb, ax, ay, fz, bx, by, bz, (int)axis);
                    }
                    const uint64_t id = W.first[qk] + qs + r;
                    float* o = I.coords + 3 * id;
                    o[0] = v.x; o[1] = v.y; o[2] = v.z;
                    if (I.slots) clear_face_slots(I.slots, id, lx, qy, zn, nx, ny, nz);
                }
            }
            __syncwarp();   // the corner values and first vertices are read
        }
    }
}

// One vertex per thread: the normals of its cells' triangles that use it, cell
// by cell, in triangle order.  A cell has one or two such triangles almost
// always, so those eight reads go out together; the others follow one by one.
__global__ void __launch_bounds__(256)
    k_vertex_slots(const uint2* __restrict__ slots, const float4* __restrict__ tri4, uint64_t ntri, uint64_t nvert,
                   float* __restrict__ normals)
{
    const uint64_t v = (uint64_t)blockIdx.x * 256 + threadIdx.x;
    if (v >= nvert) return;
    const uint4* s = reinterpret_cast<const uint4*>(slots + 4 * v);
    const uint4 lo = s[0], hi = s[1];
    const uint32_t first[4] = {lo.x, lo.z, hi.x, hi.z};
    uint32_t left[4] = {lo.y & 31u, lo.w & 31u, hi.y & 31u, hi.w & 31u};
    float4 n[4][2];
    bool is[4][2];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint64_t t = (uint64_t)first[c] + (uint32_t)(__ffs(left[c]) - 1);
            is[c][i] = left[c] != 0 && t < ntri;   // (an id past the last one: a pass before gave up)
            left[c] &= left[c] - 1u;
            if (is[c][i]) n[c][i] = __ldg(tri4 + t);
        }
    }
    float sx = 0.0f, sy = 0.0f, sz = 0.0f;
    auto add = [&](const float4& a) {
        sx = __fadd_rn(sx, a.x);
        sy = __fadd_rn(sy, a.y);
        sz = __fadd_rn(sz, a.z);
    };
#pragma unroll
    for (int c = 0; c < 4; ++c) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
            if (is[c][i]) add(n[c][i]);
        for (uint32_t m = left[c]; m; m &= m - 1u) {
            const uint64_t t = (uint64_t)first[c] + (uint32_t)(__ffs(m) - 1);
            if (t < ntri) add(__ldg(tri4 + t));
        }
    }
    normals[3 * v + 0] = sx;
    normals[3 * v + 1] = sy;
    normals[3 * v + 2] = sz;
}

size_t slots_align(size_t v) { return (v + 255) / 256 * 256; }

}  // namespace

cudaError_t launch_connect_pairs(const StreamGroup* d_group, const StreamIso* d_isos, const ConnTable& conn, int dtype,
                                 uint32_t words_per_row, const PairList& list, const uint32_t* unit_offsets,
                                 const uint64_t* plane_base, uint64_t ntasks, int* status,
                                 unsigned long long* next_task, const Launch& L)
{
    if (ntasks == 0) return cudaSuccess;
    const void* kern = nullptr;
    size_t smem = sizeof(PairTables);
#define KVSMC_CONN_CASE(CODE, T)                                                     \
    case CODE:                                                                       \
        kern = reinterpret_cast<const void*>(k_connect_pairs<T>);                    \
        smem += kPairWarps * sizeof(ConnWarp<typename PairValue<T>::type>);          \
        break;
    switch (dtype) {
        KVSMC_CONN_CASE(0, int8_t)
        KVSMC_CONN_CASE(1, int16_t)
        KVSMC_CONN_CASE(2, int32_t)
        KVSMC_CONN_CASE(3, long long)
        KVSMC_CONN_CASE(4, uint8_t)
        KVSMC_CONN_CASE(5, uint16_t)
        KVSMC_CONN_CASE(6, uint32_t)
        KVSMC_CONN_CASE(7, unsigned long long)
        KVSMC_CONN_CASE(8, float)
        KVSMC_CONN_CASE(9, double)
    default: break;
    }
#undef KVSMC_CONN_CASE
    if (!kern) return cudaErrorInvalidValue;
    int per_sm = 0;
    cudaError_t e = kernel_fit(L, kern, kPairThreads, smem, &per_sm);
    if (e != cudaSuccess) return e;
    const uint64_t need = (ntasks + kPairWarps - 1) / kPairWarps;
    const uint64_t resident = (uint64_t)(per_sm > 0 ? per_sm : 1) * (uint64_t)L.num_sms;
    uint32_t polls = L.wait_polls[1];
    PairList pl = list;
    ConnTable table = conn;
    void* args[] = {&d_group, &d_isos, &table, &pl, &unit_offsets, &plane_base, &ntasks, &words_per_row, &status,
                    &next_task, &polls};
    prof_begin(L, "connect_pairs");
    e = cudaLaunchKernel(kern, dim3((unsigned)(need < resident ? need : resident)), dim3(kPairThreads), args, smem,
                         L.stream);
    prof_end(L);
    *L.counter += 1;
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_nodes_pairs(const StreamGroup* d_group, const StreamIso* d_isos, const NodeTable& nodes, int dtype,
                               uint32_t words_per_row, const PairList& list, uint64_t ntasks, int* status,
                               unsigned long long* next_task, const Launch& L)
{
    if (ntasks == 0) return cudaSuccess;
    const void* kern = dtype == 0   ? reinterpret_cast<const void*>(k_nodes_pairs<int8_t>)
                       : dtype == 1 ? reinterpret_cast<const void*>(k_nodes_pairs<int16_t>)
                       : dtype == 4 ? reinterpret_cast<const void*>(k_nodes_pairs<uint8_t>)
                       : dtype == 5 ? reinterpret_cast<const void*>(k_nodes_pairs<uint16_t>)
                       : dtype == 8 ? reinterpret_cast<const void*>(k_nodes_pairs<float>)
                                    : nullptr;   // (the wide types' node units are not counted with their pairs)
    if (!kern) return cudaErrorInvalidValue;
    int per_sm = 0;
    cudaError_t e = kernel_fit(L, kern, kPairThreads, 0, &per_sm);
    if (e != cudaSuccess) return e;
    const uint64_t need = (ntasks + kPairWarps - 1) / kPairWarps;
    const uint64_t resident = (uint64_t)(per_sm > 0 ? per_sm : 1) * (uint64_t)L.num_sms;
    PairList pl = list;
    NodeTable table = nodes;
    void* args[] = {&d_group, &d_isos, &table, &pl, &ntasks, &words_per_row, &status, &next_task};
    prof_begin(L, "nodes_pairs");
    e = cudaLaunchKernel(kern, dim3((unsigned)(need < resident ? need : resident)), dim3(kPairThreads), args, 0, L.stream);
    prof_end(L);
    *L.counter += 1;
    return e != cudaSuccess ? e : cudaGetLastError();
}

size_t vertex_slots_bytes(uint64_t ntri, uint64_t nvert) { return slots_align(16 * ntri) + slots_align(32 * nvert); }

VertexSlots vertex_slots_carve(uint64_t ntri, uint64_t, void* scratch)
{
    char* p = static_cast<char*>(scratch);
    return VertexSlots{reinterpret_cast<float4*>(p), reinterpret_cast<uint2*>(p + slots_align(16 * ntri))};
}

cudaError_t launch_vertex_slots(const VertexSlots& v, uint64_t ntri, uint64_t nvert, float* normals, const Launch& L)
{
    if (nvert == 0) return cudaSuccess;
    prof_begin(L, "vertex_slots");
    k_vertex_slots<<<(unsigned)((nvert + 255) / 256), 256, 0, L.stream>>>(v.slots, v.tri4, ntri, nvert, normals);
    prof_end(L);
    *L.counter += 1;
    return cudaGetLastError();
}

}  // namespace kvsmc
