// mc_connect.cu -- connect_isopoints (MarchingCubes.cpp:456-521) and the vertex
// normals (:569-605) of the shared-vertex modes over listed pairs: the count
// pass has listed the crossed cells, the node emit has written vertices and
// rank words (mc_snode.cu).
//
// Tasks, blocks and rounds are mc_pairs.cu's.  A round's vertex items (one per
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
// 745 and 242.
#include <cuda_runtime.h>

#include "mc_device.cuh"
#include "mc_emit.cuh"
#include "mc_internal.h"
#include "mc_interp.cuh"
#include "mc_pairs.cuh"
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
        const PairBlock B = pair_block(G, pl, (uint32_t)task, lane);
        if (B.npairs == 0) continue;
        const uint32_t z = B.z;
        __syncwarp();
        if (lane < niso) {
            const uint64_t pi = isos[iso_begin + lane].plane_index;
            W.first[lane] = plane_base[pi + z] - plane_base[pi] +
                            unit_offsets[G.unit_base + ((uint64_t)z * ((ny - 1) * G.wpr) + B.u0) * niso + lane];
        }
        __syncwarp();
        uint32_t run = 0;   // lane k: the task's triangles of isolevel k so far (at most 32 * 256 * 5)
        const T* vz = static_cast<const T*>(G.vol.data) + (uint64_t)z * slice;
        const float fz = __uint2float_rn(z);
        uint32_t taken = 0;
        for (uint32_t r0 = 0; r0 < B.npairs; r0 += taken) {
            // ---- one pair per lane, as many as the vertex pool holds
            bool has = r0 + lane < B.npairs;
            uint32_t x, y;
            const uint32_t at = pair_entry(B, r0 + lane, x, y);
            uint32_t k = 0, code = 0;
            if (has) {
                const uint32_t e = pl.list[at];
                x += e & 0xffu;
                k = e >> 8;
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
                if (gaps) q = __fns(items, 0, (int)q + 1);
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
                if (gaps) q = __fns(items, 0, (int)q + 1);
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
