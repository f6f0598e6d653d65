// slice.cu -- kvs::SlicePlane on structured volumes, on the GPU.
//
// The reference (Source/Core/Visualization/Mapper/SlicePlane.cpp) runs
// marching cubes on the plane function p(x) = a x + b y + c z + d instead of
// the volume: a cell's case has bit k set iff p(corner k) > 0 in float
// (calculate_table_index, :802-818; substitute_plane_equation, :949-959,
// ((a x + b y) + c z) + d), triangles come from MarchingCubesTable in table
// order with vertices (e[i], e[i+2], e[i+1]) (:101-135), each vertex at
// (1 - r) v0 + r v1 with r = |p0 / (p1 - p0)| in float (interpolate_vertex,
// :986-995) then (v + min_coord) * scale; its colour is
// ColorMap::at(value) of the volume value interpolated with the same r in the
// value type's own arithmetic (interpolate_value, :1006-1031; ColorMap.cpp:
// 1043-1054, RGBColor::Mix, RGBColor(Vec3) rounding); one normal per triangle
// -((v2 - v0) x (v1 - v0)).  Cells in z, y, x order.
//
// Two passes over groups of consecutive cell rows (y, z), a warp per group (32
// rows, fewer where the plane runs along the rows): count (cases from the plane
// alone, only over the x-interval of a row's cells that the plane can cut,
// bounded conservatively), an exclusive scan of the groups' counts, emit (the group's cut cells gathered, then 32 at a time: a
// vertex per lane, a triangle per lane; the volume read only at the corners of
// cut edges).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "context.h"
#include "mc_emit.cuh"
#include "slice_common.cuh"
#include "mc_tables.h"

namespace kvsmc {

namespace {

// Case tables, laid out at compile time: per case the triangle corners as ranks
// among its used edges (4 bits each, table order), the used edges (corner A |
// corner B << 4; corner: dx + 2 dy + 4 dz) and triangles | edges << 4.
struct alignas(16) SliceTables {
    uint64_t slots[256];
    uint8_t edges[256][12];
    uint8_t counts[256];
};

constexpr uint64_t h_slice_tri[256] = MC_TRI_PACKED_INIT;
constexpr uint8_t h_slice_ntri[256] = MC_NTRI_INIT;
constexpr uint8_t h_slice_edge[12] = MC_EDGE_PACKED_INIT;

constexpr SliceTables make_slice_tables()
{
    SliceTables t{};
    for (int c = 0; c < 256; ++c) {
        int n = 0;
        uint64_t of[12] = {};
        for (int k = 0; k < 3 * (int)h_slice_ntri[c]; ++k) {
            const uint64_t e = (h_slice_tri[c] >> (4 * k)) & 15u;
            int r = 0;
            while (r < n && of[r] != e) ++r;
            if (r == n) {
                of[n] = e;
                t.edges[c][n++] = (uint8_t)((h_slice_edge[e] & 7u) | ((h_slice_edge[e] >> 3) << 4));
            }
            t.slots[c] |= (uint64_t)r << (4 * k);
        }
        t.counts[c] = (uint8_t)(h_slice_ntri[c] | (n << 4));
    }
    return t;
}

__device__ const SliceTables d_slice_tables = make_slice_tables();

constexpr int kSliceThreads = 128;
constexpr int kSliceWarps = kSliceThreads / 32;
constexpr uint32_t kSliceVerts = 192;   // vertices of a round
constexpr unsigned FULL = 0xffffffffu;

// The plane's signs at the four nodes (x, y.., z..) of a cell's face: bit r =
// above at rows (y, z), (y + 1, z), (y, z + 1), (y + 1, z + 1).
__device__ __forceinline__ uint32_t slice_signs(const SliceJob& j, uint32_t x, uint32_t y, uint32_t z)
{
    const float fx = __uint2float_rn(x), fy = __uint2float_rn(y), fz = __uint2float_rn(z);
    const float y1 = __uint2float_rn(y + 1), z1 = __uint2float_rn(z + 1);
    return (plane_at(j, fx, fy, fz) > 0.0f ? 1u : 0u) | (plane_at(j, fx, y1, fz) > 0.0f ? 2u : 0u) |
           (plane_at(j, fx, fy, z1) > 0.0f ? 4u : 0u) | (plane_at(j, fx, y1, z1) > 0.0f ? 8u : 0u);
}

// The case from the signs at x and at x + 1 (corners (x,y,z) 0:(0,0,0)
// 1:(1,0,0) 2:(1,1,0) 3:(0,1,0), 4 .. 7 the same at z + 1).
__device__ __forceinline__ uint32_t slice_case(uint32_t l, uint32_t r)
{
    return (l & 1u) | ((r & 1u) << 1) | ((r & 2u) << 1) | ((l & 2u) << 2) |
           ((l & 4u) << 2) | ((r & 4u) << 3) | ((r & 8u) << 3) | ((l & 8u) << 4);
}

// The vertex on the edge between corners a and b of cell (x, y, z): position
// after (v + min_coord) * scale, colour in w.
template <typename T>
__device__ __forceinline__ float4 slice_vertex(const SliceJob& j, const float* unit, const T* vol, uint32_t x,
                                               uint32_t y, uint32_t z, unsigned a, unsigned b)
{
    const uint32_t ax = x + (a & 1u), ay = y + ((a >> 1) & 1u), az = z + (a >> 2);
    const uint32_t bx = x + (b & 1u), by = y + ((b >> 1) & 1u), bz = z + (b >> 2);
    const T va = vol[(uint64_t)az * j.vol.slice + (uint64_t)ay * j.vol.pitch + ax];
    const T vb = vol[(uint64_t)bz * j.vol.slice + (uint64_t)by * j.vol.pitch + bx];
    const float v0x = __uint2float_rn(ax), v0y = __uint2float_rn(ay), v0z = __uint2float_rn(az);
    const float v1x = __uint2float_rn(bx), v1y = __uint2float_rn(by), v1z = __uint2float_rn(bz);
    const float p0 = plane_at(j, v0x, v0y, v0z), p1 = plane_at(j, v1x, v1y, v1z);
    const float ratio = fabsf(__fdiv_rn(p0, __fsub_rn(p1, p0)));
    const float s = __fsub_rn(1.0f, ratio);
    const float vx = __fadd_rn(__fmul_rn(s, v0x), __fmul_rn(ratio, v1x));
    const float vy = __fadd_rn(__fmul_rn(s, v0y), __fmul_rn(ratio, v1y));
    const float vz = __fadd_rn(__fmul_rn(s, v0z), __fmul_rn(ratio, v1z));
    const uchar3 rgb = color_at(j, unit, slice_value(va, vb, ratio));
    return make_float4(__fmul_rn(__fadd_rn(vx, j.min_coord[0]), j.scale[0]),
                       __fmul_rn(__fadd_rn(vy, j.min_coord[1]), j.scale[1]),
                       __fmul_rn(__fadd_rn(vz, j.min_coord[2]), j.scale[2]),
                       __uint_as_float((uint32_t)rgb.x | ((uint32_t)rgb.y << 8) | ((uint32_t)rgb.z << 16)));
}

// The cells of row (y, z) the plane can cut: an interval [x0, x1] of x (x0 >
// x1: none).  Over a cell the plane ranges over [a x + k1, a x + k2], k1 =
// min(0, a) + Bmin + Cmin + d, k2 = max(0, a) + Bmax + Cmax + d (B, C: b y',
// c z' over the cell's y', z').  A cell whose range lies on one side of zero
// for every node, evaluated in float as the cases are, has no triangle, so
// what matters is that k1 is not too high and k2 not too low.  With u = 2^-24
// and S = |a| cx + |b| (y + 1) + |c| (z + 1) + |d|, the float evaluation of a
// node is within 8 u S of the exact value, and k1 and k2, computed in float,
// within 8 u S of theirs (two roundings in a product, three sums, each below
// S); m = 64 u S + 1e-30 is more than both together and its own rounding.  The
// ends -k / a carry two roundings, below u (cx + 2) each where they lie in
// the row: 4 u (cx + 4) is added.  FP64 would need less margin, but its two
// divisions a row took most of the passes' time (512 x 480 x 500 nodes
// have 2.4e5 rows); the float margin costs 0.01 cells a row there.
__device__ __forceinline__ void row_interval(const SliceJob& j, uint32_t cx, uint32_t y, uint32_t z, uint32_t& x0,
                                             uint32_t& len)
{
    const float a = j.coef[0], b = j.coef[1], c = j.coef[2], d = j.coef[3];
    const float fcx = (float)cx;
    const float by0 = b * (float)y, by1 = b * (float)(y + 1), cz0 = c * (float)z, cz1 = c * (float)(z + 1);
    const float S = ((fabsf(a) * fcx + fmaxf(fabsf(by0), fabsf(by1))) + fmaxf(fabsf(cz0), fabsf(cz1))) + fabsf(d);
    x0 = 0;
    len = cx;
    if (!(S < 1e37f)) return;   // (NaN and overflow too) every cell is evaluated
    const float m = S * 3.814697265625e-06f + 1e-30f;
    const float k1 = ((fminf(0.0f, a) + fminf(by0, by1)) + fminf(cz0, cz1)) + d - m;   // low end: a x + k1 <= 0
    const float k2 = ((fmaxf(0.0f, a) + fmaxf(by0, by1)) + fmaxf(cz0, cz1)) + d + m;   // high end: a x + k2 > 0
    if (a == 0.0f) {
        if (!(k1 <= 0.0f && k2 > 0.0f)) len = 0;
        return;
    }
    const float e0 = -k2 / a, e1 = -k1 / a;
    const float eps = 2.384185791015625e-07f * (fcx + 4.0f);
    float lo = (a > 0.0f ? e0 : e1) - eps;   // x in [lo, hi]
    const float hi = (a > 0.0f ? e1 : e0) + eps;
    lo = fmaxf(lo, 0.0f);
    if (!(lo <= hi)) {
        len = 0;
        return;
    }
    x0 = (uint32_t)ceilf(lo);               // (these conversions saturate)
    uint32_t x1 = (uint32_t)floorf(hi);
    if (x1 > cx - 1) x1 = cx - 1;
    len = x1 >= x0 ? x1 - x0 + 1 : 0u;
}

// Count of groups of 32 rows, a row per lane: the case of each cell of the row's
// interval, the plane's signs at x carried from the cell before.  512 x 480 x 500
// nodes, an oblique plane: 37 us in FP64 and eight plane values a cell, 8.6 us.
__global__ void __launch_bounds__(kSliceThreads) k_slice_count(SliceJob j)
{
    __shared__ uint8_t s_counts[256];
    for (unsigned i = threadIdx.x; i < 256; i += kSliceThreads) s_counts[i] = d_slice_tables.counts[i];
    __syncthreads();
    const uint32_t cx = j.vol.nx - 1, cy = j.vol.ny - 1;
    const uint64_t row = (uint64_t)blockIdx.x * kSliceThreads + threadIdx.x;
    uint32_t sum = 0;
    if (row < j.nrows) {
        const uint32_t z = (uint32_t)(row / cy), y = (uint32_t)(row - (uint64_t)z * cy);
        uint32_t x0, len;
        row_interval(j, cx, y, z, x0, len);
        if (len) {
            uint32_t left = slice_signs(j, x0, y, z);
            for (uint32_t x = x0; x < x0 + len; ++x) {
                const uint32_t right = slice_signs(j, x + 1, y, z);
                sum += s_counts[slice_case(left, right)] & 15u;
                left = right;
            }
        }
    }
    sum = __reduce_add_sync(FULL, sum);
    if ((threadIdx.x & 31u) == 0 && row < j.nrows) j.group_counts[row / 32] = sum;
}

// A group's rows, one per lane, and its cells as one index space in row and x
// order: lane l's row holds the items [first, inc).
struct SliceRows {
    uint32_t y, z, x0;
    uint64_t first, inc, total;   // (a row has up to 2^32 cells: 64 bits)
};

__device__ __forceinline__ SliceRows slice_rows(const SliceJob& j, uint64_t group, unsigned lane)
{
    SliceRows r;
    const uint32_t cx = j.vol.nx - 1, cy = j.vol.ny - 1;
    const uint64_t row = (group << j.group_shift) + lane;
    uint32_t len = 0;
    r.y = r.z = r.x0 = 0;
    if (lane < (1u << j.group_shift) && row < j.nrows) {
        r.z = (uint32_t)(row / cy);
        r.y = (uint32_t)(row - (uint64_t)r.z * cy);
        row_interval(j, cx, r.y, r.z, r.x0, len);
    }
    r.inc = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t t = __shfl_up_sync(FULL, r.inc, o);
        if (lane >= (unsigned)o) r.inc += t;
    }
    r.first = r.inc - len;
    r.total = __shfl_sync(FULL, r.inc, 31);
    return r;
}

// The case of item i and its place; lanes past the last item get case 0.
__device__ __forceinline__ uint32_t slice_item(const SliceJob& j, const SliceRows& r, uint64_t i, uint32_t& own,
                                               uint32_t& x)
{
    own = 0;   // the item's row: the first lane whose inclusive count exceeds i
#pragma unroll
    for (int s = 4; s >= 0; --s) {
        const uint32_t mid = own + (1u << s) - 1u;
        if (__shfl_sync(FULL, r.inc, mid) <= i) own = mid + 1;
    }
    own &= 31u;   // (lanes past the last cell)
    x = __shfl_sync(FULL, r.x0, own) + (uint32_t)(i - __shfl_sync(FULL, r.first, own));
    const uint32_t y = __shfl_sync(FULL, r.y, own), z = __shfl_sync(FULL, r.z, own);
    return i < r.total ? slice_case(slice_signs(j, x, y, z), slice_signs(j, x + 1, y, z)) : 0u;
}

// Count of groups of fewer rows, whose intervals are long: a warp per group, a
// cell per lane.
__global__ void __launch_bounds__(kSliceThreads) k_slice_count_long(SliceJob j)
{
    const unsigned lane = threadIdx.x & 31u;
    const uint64_t group = (uint64_t)blockIdx.x * kSliceWarps + (threadIdx.x >> 5);
    if ((group << j.group_shift) >= j.nrows) return;
    const SliceRows r = slice_rows(j, group, lane);
    uint32_t sum = 0;
    for (uint64_t b0 = 0; b0 < r.total; b0 += 32) {
        uint32_t own, x;
        sum += d_slice_tables.counts[slice_item(j, r, b0 + lane, own, x)] & 15u;
    }
    sum = __reduce_add_sync(FULL, sum);
    if (lane == 0) j.group_counts[group] = sum;
}

struct alignas(16) SliceWarp {
    float4 pv[kSliceVerts];   // the round's vertices: x, y, z, colour
    uint32_t cells[64];       // gathered cut cells: x, and
    uint16_t tags[64];        // case | lane of the row << 8
};

// Emit: the group's cells are evaluated 32 at a time (whatever row they are
// in) and those with triangles gathered, so that the rounds below, which read
// the volume, are full: a round's vertices one per lane (each used edge of a
// cell once), its triangles one per lane, in row, x and table order.  Bound by
// the latency of the volume's reads.  512 x 480 x 500
// nodes, an oblique plane: 89 us three vertices a triangle from half-empty
// rounds, 45 us; a plane z = const, one row a warp: 2500 -> 170 us a call.
template <typename T>
__global__ void __launch_bounds__(kSliceThreads) k_slice_emit(SliceJob j)
{
    __shared__ SliceTables TB;
    __shared__ SliceWarp sw[kSliceWarps];
    __shared__ float unit[256];
    // launched before the host knows the total: nothing is written unless all fits
    if (*j.d_total > j.cap_tris) return;
    const unsigned lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    const uint64_t group = (uint64_t)blockIdx.x * kSliceWarps + (threadIdx.x >> 5);
    const bool any = (group << j.group_shift) < j.nrows && j.group_counts[group] != 0;
    if (!__syncthreads_or(any)) return;   // (most groups of an axis-aligned plane)
    static_assert(sizeof(SliceTables) % 16 == 0, "copied as 16-byte words");
    for (unsigned i = threadIdx.x; i < sizeof(SliceTables) / 16; i += kSliceThreads)
        reinterpret_cast<uint4*>(&TB)[i] = reinterpret_cast<const uint4*>(&d_slice_tables)[i];
    fill_unit(unit);
    __syncthreads();
    if (!any) return;
    SliceWarp& W = sw[threadIdx.x >> 5];
    const T* vol = static_cast<const T*>(j.vol.data);
    uint64_t run = j.group_offsets[group];   // the next output triangle
    const SliceRows rows = slice_rows(j, group, lane);
    uint32_t held = 0;   // gathered cells
    for (uint64_t b0 = 0; b0 < rows.total || held;) {
        // ---- gather cut cells until a round is full or none are left
        while (held < 32 && b0 < rows.total) {
            uint32_t own, x;
            const uint32_t code = slice_item(j, rows, b0 + lane, own, x);
            const bool cut = (TB.counts[code] & 15u) != 0;
            const uint32_t cuts = __ballot_sync(FULL, cut);
            if (cut) {
                const uint32_t at = held + (uint32_t)__popc(cuts & lt);
                W.cells[at] = x;
                W.tags[at] = (uint16_t)(code | (own << 8));
            }
            held += (uint32_t)__popc(cuts);
            b0 += 32;
            __syncwarp();
        }
        // ---- one cell per lane, as many as the vertex pool holds
        bool has = lane < held;
        const uint32_t x = W.cells[lane], tag = W.tags[lane];
        const uint32_t code = has ? tag & 255u : 0u;
        const uint32_t own = has ? tag >> 8 : 0u;
        const uint32_t y = __shfl_sync(FULL, rows.y, own), z = __shfl_sync(FULL, rows.z, own);
        const uint32_t cnt = has ? TB.counts[code] : 0u, ne = cnt >> 4;
        uint32_t vpre = 0;
#pragma unroll
        for (int bit = 0; bit < 4; ++bit) vpre += (uint32_t)__popc(__ballot_sync(FULL, (ne >> bit) & 1u) & lt) << bit;
        has = has && vpre + ne <= kSliceVerts;   // a suffix of lanes waits
        const uint32_t taken = (uint32_t)__popc(__ballot_sync(FULL, has));
        if (taken == 0) break;   // (nothing was cut)
        const uint32_t nv = __shfl_sync(FULL, vpre + ne, taken - 1);
        const uint32_t nt = has ? cnt & 15u : 0u;
        uint32_t tpre = 0, ntr = 0;
#pragma unroll
        for (int bit = 0; bit < 3; ++bit) {
            const uint32_t bm = __ballot_sync(FULL, (nt >> bit) & 1u);
            tpre += (uint32_t)__popc(bm & lt) << bit;
            ntr += (uint32_t)__popc(bm) << bit;
        }
        const uint32_t pe = code | (vpre << 8) | (tpre << 20);
        uint32_t seen = 0;
        for (uint32_t j0 = 0; j0 < nv; j0 += 32) {
            const uint32_t i = j0 + lane;
            // the cells' first items as bits: an item's cell is the number of first items up to it
            const uint32_t starts = __reduce_or_sync(FULL, has && vpre - j0 < 32u ? 1u << (vpre - j0) : 0u);
            const uint32_t q = seen + (uint32_t)__popc(starts & (lt | (1u << lane))) - 1u;
            seen += (uint32_t)__popc(starts);
            const uint32_t qe = __shfl_sync(FULL, pe, q), qx = __shfl_sync(FULL, x, q);
            const uint32_t qy = __shfl_sync(FULL, y, q), qz = __shfl_sync(FULL, z, q);
            if (i < nv) {
                const uint32_t ed = TB.edges[qe & 255u][i - ((qe >> 8) & 0xfffu)];
                W.pv[i] = slice_vertex<T>(j, unit, vol, qx, qy, qz, ed & 15u, ed >> 4);
            }
        }
        __syncwarp();
        seen = 0;
        for (uint32_t j0 = 0; j0 < ntr; j0 += 32) {
            const uint32_t i = j0 + lane;
            const uint32_t starts = __reduce_or_sync(FULL, has && tpre - j0 < 32u ? 1u << (tpre - j0) : 0u);
            const uint32_t q = seen + (uint32_t)__popc(starts & (lt | (1u << lane))) - 1u;
            seen += (uint32_t)__popc(starts);
            const uint32_t qe = __shfl_sync(FULL, pe, q);
            const uint64_t t = run + i;
            if (i < ntr && t < j.cap_tris) {   // never past the outputs
                const uint32_t sl = (uint32_t)(TB.slots[qe & 255u] >> (12 * (i - (qe >> 20))));
                const float4* pv = W.pv + ((qe >> 8) & 0xfffu);
                const float4 corner[3] = {pv[sl & 15u], pv[(sl >> 4) & 15u], pv[(sl >> 8) & 15u]};
                const float3 A = make_float3(corner[0].x, corner[0].y, corner[0].z);
                const float3 B = make_float3(corner[1].x, corner[1].y, corner[1].z);
                const float3 C = make_float3(corner[2].x, corner[2].y, corner[2].z);
                store_triangle(j.coords + 9 * t, j.normals + 3 * t, A, B, C, slice_normal(A, B, C));
                uint8_t* o = j.colors + 9 * t;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const uint32_t w = __float_as_uint(corner[k].w);
                    o[3 * k] = (uint8_t)w;
                    o[3 * k + 1] = (uint8_t)(w >> 8);
                    o[3 * k + 2] = (uint8_t)(w >> 16);
                }
            }
        }
        run += ntr;
        // ---- the cells that wait move to the front
        __syncwarp();
        const uint32_t left = held - taken;   // (below 64)
        uint32_t kx[2] = {0, 0}, kt[2] = {0, 0};
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (lane + 32 * h < left) {
                kx[h] = W.cells[taken + lane + 32 * h];
                kt[h] = W.tags[taken + lane + 32 * h];
            }
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (lane + 32 * h < left) {
                W.cells[lane + 32 * h] = kx[h];
                W.tags[lane + 32 * h] = (uint16_t)kt[h];
            }
        held = left;
        __syncwarp();
    }
}

unsigned slice_grid(const SliceJob& j)
{
    const uint64_t groups = (j.nrows + (1ull << j.group_shift) - 1) >> j.group_shift;
    return (unsigned)((groups + kSliceWarps - 1) / kSliceWarps);
}

}  // namespace

cudaError_t launch_slice_count(const SliceJob& j, const Launch& L)
{
    if (j.nrows == 0) return cudaSuccess;
    prof_begin(L, "slice_count");
    if (j.group_shift == 5) k_slice_count<<<slice_grid(j), kSliceThreads, 0, L.stream>>>(j);
    else k_slice_count_long<<<slice_grid(j), kSliceThreads, 0, L.stream>>>(j);
    prof_end(L);
    *L.counter += 1;
    return cudaGetLastError();
}

cudaError_t launch_slice_emit(const SliceJob& j, const Launch& L)
{
    if (j.nrows == 0) return cudaSuccess;
    prof_begin(L, "slice_emit");
    switch (j.vol.dtype) {
    case 0: k_slice_emit<int8_t><<<slice_grid(j), kSliceThreads, 0, L.stream>>>(j); break;
    case 1: k_slice_emit<int16_t><<<slice_grid(j), kSliceThreads, 0, L.stream>>>(j); break;
    case 2: k_slice_emit<int32_t><<<slice_grid(j), kSliceThreads, 0, L.stream>>>(j); break;
    case 3: k_slice_emit<long long><<<slice_grid(j), kSliceThreads, 0, L.stream>>>(j); break;
    case 4: k_slice_emit<uint8_t><<<slice_grid(j), kSliceThreads, 0, L.stream>>>(j); break;
    case 5: k_slice_emit<uint16_t><<<slice_grid(j), kSliceThreads, 0, L.stream>>>(j); break;
    case 6: k_slice_emit<uint32_t><<<slice_grid(j), kSliceThreads, 0, L.stream>>>(j); break;
    case 7: k_slice_emit<unsigned long long><<<slice_grid(j), kSliceThreads, 0, L.stream>>>(j); break;
    case 8: k_slice_emit<float><<<slice_grid(j), kSliceThreads, 0, L.stream>>>(j); break;
    case 9: k_slice_emit<double><<<slice_grid(j), kSliceThreads, 0, L.stream>>>(j); break;
    default: prof_end(L); return cudaErrorInvalidValue;
    }
    prof_end(L);
    *L.counter += 1;
    return cudaGetLastError();
}

}  // namespace kvsmc

namespace {

using kvsmc_host::fail;

// Plan, count and scan one slice on a resident volume into the context's
// scratch (total in j.d_total; j.nrows is 0 when there are no cells).  The job
// stays valid until the scratch is next used.
kvsmc_status slice_count_enqueue(kvsmc_context* ctx, kvsmc_volume* v, const kvsmc_slice_params* p, kvsmc::SliceJob& j)
{
    using namespace kvsmc_host;
    std::memset(&j, 0, sizeof j);
    if (!p || !p->tf_table || p->tf_resolution < 1)
        return fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "slice: bad parameters (colour table)");
    volume_use(ctx, v);
    const kvsmc::VolumeView& vv = v->view;
    if (vv.nx < 2 || vv.ny < 2 || vv.nz < 2) return KVSMC_OK;   // no cells
    j.vol = vv;
    for (int k = 0; k < 4; ++k) j.coef[k] = p->coefficients[k];
    for (int k = 0; k < 3; ++k) { j.min_coord[k] = p->min_coord[k]; j.scale[k] = p->scale[k]; }
    j.tf_min = p->tf_min;
    j.tf_max = p->tf_max;
    j.tf_res = p->tf_resolution;
    const uint64_t nrows = (uint64_t)(vv.ny - 1) * (vv.nz - 1);
    // rows per warp: 32 where the plane cuts a few cells of a row, fewer where
    // it runs along the rows, so that a warp gets some 512 cells at most
    const double a = std::fabs((double)j.coef[0]), bc2 = std::fabs((double)j.coef[1]) + std::fabs((double)j.coef[2]);
    const double len = bc2 < a * (double)(vv.nx - 2) ? 1.0 + bc2 / a : (double)(vv.nx - 1);   // (NaN: the whole row)
    j.group_shift = 5;
    while (j.group_shift > 0 && len * (double)(1 << j.group_shift) > 512.0) --j.group_shift;
    const uint64_t ngroups = (nrows + (1ull << j.group_shift) - 1) >> j.group_shift;
    const size_t bt = align_up((size_t)3 * j.tf_res, 256), bc = align_up(ngroups * 4, 256),
                 bo = align_up(ngroups * 8, 256), bs = align_up(kvsmc::scan_scratch_bytes(ngroups), 256);
    kvsmc_status st = ensure_scratch(ctx, bt + bc + bo + bs + 256);
    if (st) return st;
    char* base = static_cast<char*>(ctx->scratch);
    uint8_t* d_table = reinterpret_cast<uint8_t*>(base);
    j.table = d_table;
    j.nrows = nrows;
    j.group_counts = reinterpret_cast<uint32_t*>(base + bt);
    j.group_offsets = reinterpret_cast<uint64_t*>(base + bt + bc);
    void* d_scan = base + bt + bc + bo;
    j.d_total = reinterpret_cast<uint64_t*>(base + bt + bc + bo + bs);
    if ((st = ensure_stage(ctx, (size_t)3 * j.tf_res))) return st;
    std::memcpy(ctx->h_stage, p->tf_table, (size_t)3 * j.tf_res);
    KVSMC_CUDA(ctx, cudaMemcpyAsync(d_table, ctx->h_stage, (size_t)3 * j.tf_res, cudaMemcpyHostToDevice, ctx->stream));
    const kvsmc::Launch L = launch_of(ctx);
    KVSMC_CUDA(ctx, kvsmc::launch_slice_count(j, L));
    KVSMC_CUDA(ctx, kvsmc::launch_scan(j.group_counts, j.group_offsets, ngroups, d_scan, j.d_total, L));
    return KVSMC_OK;
}

// Wait for everything enqueued and read the total.
kvsmc_status slice_total(kvsmc_context* ctx, const kvsmc::SliceJob& j, uint64_t* ntri)
{
    using namespace kvsmc_host;
    *ntri = 0;
    if (j.nrows == 0) return KVSMC_OK;
    KVSMC_CUDA(ctx, cudaMemcpyAsync(ctx->h_small, j.d_total, sizeof(uint64_t), cudaMemcpyDeviceToHost, ctx->stream));
    KVSMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    *ntri = ctx->h_small[0];
    return KVSMC_OK;
}

kvsmc_status slice_emit(kvsmc_context* ctx, kvsmc::SliceJob& j, float* d_coords, uint8_t* d_colors, float* d_normals,
                        uint64_t cap)
{
    using namespace kvsmc_host;
    if (j.nrows == 0) return KVSMC_OK;
    j.coords = d_coords;
    j.colors = d_colors;
    j.normals = d_normals;
    j.cap_tris = cap;
    KVSMC_CUDA(ctx, kvsmc::launch_slice_emit(j, launch_of(ctx)));
    return KVSMC_OK;
}

}  // namespace

extern "C" {

kvsmc_status kvsmc_slice_count(kvsmc_context* ctx, kvsmc_volume* vol, const kvsmc_slice_params* p,
                               uint64_t* ntriangles)
{
    if (!ctx || !vol || !ntriangles) return KVSMC_ERR_INVALID_ARGUMENT;
    KVSMC_CUDA(ctx, cudaSetDevice(ctx->device));
    *ntriangles = 0;
    kvsmc::SliceJob j;
    const kvsmc_status st = slice_count_enqueue(ctx, vol, p, j);
    return st ? st : slice_total(ctx, j, ntriangles);
}

kvsmc_status kvsmc_slice_extract_device(kvsmc_context* ctx, kvsmc_volume* vol, const kvsmc_slice_params* p,
                                        float* d_coords, uint64_t coords_capacity, uint8_t* d_colors,
                                        uint64_t colors_capacity, float* d_normals, uint64_t normals_capacity,
                                        uint64_t* ntriangles)
{
    if (!ctx || !vol || !ntriangles) return KVSMC_ERR_INVALID_ARGUMENT;
    KVSMC_CUDA(ctx, cudaSetDevice(ctx->device));
    *ntriangles = 0;
    kvsmc::SliceJob j;
    kvsmc_status st = slice_count_enqueue(ctx, vol, p, j);
    if (st) return st;
    // the emit goes behind the count when there are outputs (it writes nothing
    // unless the total fits them): one host round trip per call
    const bool outs = d_coords && d_colors && d_normals;
    const uint64_t cap = outs ? std::min(std::min(coords_capacity / 9, colors_capacity / 9), normals_capacity / 3) : 0;
    if (cap && (st = slice_emit(ctx, j, d_coords, d_colors, d_normals, cap))) return st;
    if ((st = slice_total(ctx, j, ntriangles))) return st;
    if (*ntriangles > cap)
        return fail(ctx, KVSMC_ERR_CAPACITY, "slice: %llu triangles do not fit the outputs",
                    (unsigned long long)*ntriangles);
    return KVSMC_OK;
}

kvsmc_status kvsmc_slice_plane(kvsmc_context* ctx, kvsmc_volume* vol, const kvsmc_slice_params* p,
                               kvsmc_host_alloc_fn alloc, void* user, uint64_t* ntriangles)
{
    using namespace kvsmc_host;
    if (!ctx || !vol || !alloc || !ntriangles) return KVSMC_ERR_INVALID_ARGUMENT;
    KVSMC_CUDA(ctx, cudaSetDevice(ctx->device));
    uint64_t n = 0;
    kvsmc::SliceJob j;
    *ntriangles = 0;
    kvsmc_status st = slice_count_enqueue(ctx, vol, p, j);
    if (!st) st = slice_total(ctx, j, &n);
    *ntriangles = n;
    if (st || n == 0) return st;
    const size_t bc = align_up(n * 36, 256), bn = align_up(n * 12, 256), bk = align_up(n * 9, 256);
    if (bc + bn + bk > ctx->out_bytes) {
        KVSMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        if (ctx->out_arena) cudaFree(ctx->out_arena);
        ctx->out_arena = nullptr;
        ctx->out_bytes = 0;
        const size_t want = align_up(bc + bn + bk, 1 << 20);
        KVSMC_CUDA(ctx, kvsmc_host::device_malloc(ctx, &ctx->out_arena, want));
        ctx->out_bytes = want;
    }
    char* base = static_cast<char*>(ctx->out_arena);
    float* dc = reinterpret_cast<float*>(base);
    float* dn = reinterpret_cast<float*>(base + bc);
    uint8_t* dk = reinterpret_cast<uint8_t*>(base + bc + bn);
    if ((st = slice_emit(ctx, j, dc, dk, dn, n))) return st;
    void* hc = alloc(user, 0, 9 * n);
    void* hn = hc ? alloc(user, 1, 3 * n) : nullptr;
    void* hk = hn ? alloc(user, 3, 9 * n) : nullptr;
    if (!hc || !hn || !hk) return fail(ctx, KVSMC_ERR_OUT_OF_MEMORY, "slice: host alloc");
    KVSMC_CUDA(ctx, cudaMemcpyAsync(hc, dc, n * 36, cudaMemcpyDeviceToHost, ctx->stream));
    KVSMC_CUDA(ctx, cudaMemcpyAsync(hn, dn, n * 12, cudaMemcpyDeviceToHost, ctx->stream));
    KVSMC_CUDA(ctx, cudaMemcpyAsync(hk, dk, n * 9, cudaMemcpyDeviceToHost, ctx->stream));
    KVSMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return KVSMC_OK;
}

}  // extern "C"
