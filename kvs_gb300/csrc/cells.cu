// cells.cu -- marching tetrahedra / hexahedra / pyramids / prisms on
// unstructured volumes, on the GPU.
//
// The reference mappers (Source/Core/Visualization/Mapper/MarchingTetrahedra.cpp,
// MarchingHexahedra.cpp, MarchingPyramid.cpp, MarchingPrism.cpp) share one
// structure, restated here once: cells in order; a cell's case has bit k set
// iff double(value of local node k) > isolevel (calculate_table_index), the
// local nodes being the cell's connections (hexahedra take connections 4-7
// then 0-3, MarchingHexahedra.cpp:105-112); pyramid cases 10, 11, 20, 21 are
// resolved by the sign of (iso - A) D + B C over the base's four values
// (calculate_special_table_index, MarchingPyramid.cpp:293-315); triangles
// come from the cell type's table in the mapper's vertex order (cell_tables.h);
// a vertex on the edge (n0, n1) is, in double, c0 + r (c1 - c0) per axis with
// r = |(iso - v0) / (v1 - v0)|, v clamped to the volume's [min, max], c1 - c0
// a float difference, then rounded to float (interpolate_vertex) -- here
// computed in FP32 double-float arithmetic with a rigorous error bound and
// taken only when no float rounding boundary lies within it (cell_axis),
// else by the FP64 sequence, so the bits are the reference's either way; one
// normal per triangle (v1 - v0) x (v2 - v0).  Duplicated vertices only (the
// reference's shared-vertex branch is not built, :164-206).
//
// Two passes, a warp per block of up to 32 groups of 32 cells: count (per group
// a word of which cells have triangles, per block their number), an exclusive
// scan over the blocks, emit.  An emitting warp takes the block's cut cells by
// the words' bits, 32 at a time whatever groups they are in, so its lanes stay
// busy where a surface passes a few cells of each group.  A connection index
// outside the nodes sets a flag and reads node 0 instead.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "cell_tables.h"
#include "context.h"
#include "batch.h"
#include "mc_device.cuh"
#include "mc_emit.cuh"
#include "mc_interp.cuh"
#include "mc_slots.cuh"
#include "slice_common.cuh"

namespace kvsmc {

namespace {

// A cell type's case tables, laid out at compile time: per case the triangle
// corners as ranks among the case's edges (4 bits each, table order), the edges
// (local nodes, 4 bits each) and triangles | edges << 4.
template <int CASES> struct alignas(16) CellTables {
    static constexpr int kCases = CASES;
    uint64_t slots[CASES];
    uint8_t edges[CASES][12];
    uint8_t counts[CASES];
};

template <int CASES>
constexpr CellTables<CASES> make_cell_tables(const uint8_t* ntri, const uint64_t* tri, const uint8_t* edge)
{
    CellTables<CASES> t{};
    for (int c = 0; c < CASES; ++c) {
        int n = 0;
        uint64_t of[12] = {};
        for (int k = 0; k < 3 * (int)ntri[c]; ++k) {
            const uint64_t e = (tri[c] >> (4 * k)) & 15u;
            int r = 0;
            while (r < n && of[r] != e) ++r;
            if (r == n) {
                of[n] = e;
                t.edges[c][n++] = edge[e];
            }
            t.slots[c] |= (uint64_t)r << (4 * k);
        }
        t.counts[c] = (uint8_t)(ntri[c] | (n << 4));
    }
    return t;
}

constexpr uint8_t h_tet_ntri[CELL_TETRA_CASES] = CELL_TETRA_NTRI_INIT;
constexpr uint64_t h_tet_tri[CELL_TETRA_CASES] = CELL_TETRA_TRI_INIT;
constexpr uint8_t h_tet_edge[CELL_TETRA_EDGES] = CELL_TETRA_EDGE_INIT;
constexpr uint8_t h_hex_ntri[CELL_HEXA_CASES] = CELL_HEXA_NTRI_INIT;
constexpr uint64_t h_hex_tri[CELL_HEXA_CASES] = CELL_HEXA_TRI_INIT;
constexpr uint8_t h_hex_edge[CELL_HEXA_EDGES] = CELL_HEXA_EDGE_INIT;
constexpr uint8_t h_pyr_ntri[CELL_PYRAMID_CASES] = CELL_PYRAMID_NTRI_INIT;
constexpr uint64_t h_pyr_tri[CELL_PYRAMID_CASES] = CELL_PYRAMID_TRI_INIT;
constexpr uint8_t h_pyr_edge[CELL_PYRAMID_EDGES] = CELL_PYRAMID_EDGE_INIT;
constexpr uint8_t h_pri_ntri[CELL_PRISM_CASES] = CELL_PRISM_NTRI_INIT;
constexpr uint64_t h_pri_tri[CELL_PRISM_CASES] = CELL_PRISM_TRI_INIT;
constexpr uint8_t h_pri_edge[CELL_PRISM_EDGES] = CELL_PRISM_EDGE_INIT;

__device__ const CellTables<CELL_TETRA_CASES> d_tet_tables =
    make_cell_tables<CELL_TETRA_CASES>(h_tet_ntri, h_tet_tri, h_tet_edge);
__device__ const CellTables<CELL_HEXA_CASES> d_hex_tables =
    make_cell_tables<CELL_HEXA_CASES>(h_hex_ntri, h_hex_tri, h_hex_edge);
__device__ const CellTables<CELL_PYRAMID_CASES> d_pyr_tables =
    make_cell_tables<CELL_PYRAMID_CASES>(h_pyr_ntri, h_pyr_tri, h_pyr_edge);
__device__ const CellTables<CELL_PRISM_CASES> d_pri_tables =
    make_cell_tables<CELL_PRISM_CASES>(h_pri_ntri, h_pri_tri, h_pri_edge);

constexpr int kCellThreads = 256;
// 32-cell groups per warp step of the count pass
template <int CT> constexpr int kCountGroups = CT == KVSMC_TETRAHEDRA ? 4 : 2;
constexpr unsigned FULL = 0xffffffffu;

template <int CT> struct CellTraits;
template <> struct CellTraits<KVSMC_TETRAHEDRA> {
    static constexpr int kNodes = 4;
    using Tables = CellTables<CELL_TETRA_CASES>;
    __device__ static int node(int k) { return k; }
    __device__ static const Tables& tables() { return d_tet_tables; }
};
template <> struct CellTraits<KVSMC_HEXAHEDRA> {
    static constexpr int kNodes = 8;
    using Tables = CellTables<CELL_HEXA_CASES>;
    __device__ static int node(int k) { return k < 4 ? k + 4 : k - 4; }   // MarchingHexahedra.cpp:105-112
    __device__ static const Tables& tables() { return d_hex_tables; }
};
template <> struct CellTraits<KVSMC_PYRAMID> {
    static constexpr int kNodes = 5;
    using Tables = CellTables<CELL_PYRAMID_CASES>;
    __device__ static int node(int k) { return k; }
    __device__ static const Tables& tables() { return d_pyr_tables; }
};
template <> struct CellTraits<KVSMC_PRISM> {
    static constexpr int kNodes = 6;
    using Tables = CellTables<CELL_PRISM_CASES>;
    __device__ static int node(int k) { return k; }
    __device__ static const Tables& tables() { return d_pri_tables; }
};

// Copy the cell type's tables into shared memory (whole CTA; the caller
// synchronizes).
template <typename TB> __device__ __forceinline__ void load_tables(TB& dst, const TB& src)
{
    static_assert(sizeof(TB) % 16 == 0, "copied as 16-byte words");
    for (unsigned i = threadIdx.x; i < sizeof(TB) / 16; i += kCellThreads)
        reinterpret_cast<uint4*>(&dst)[i] = reinterpret_cast<const uint4*>(&src)[i];
}

template <typename T> __device__ __forceinline__ double dval(const void* v, uint64_t i)
{
    return to_double(static_cast<const T*>(v)[i]);
}

// The cell's connections: one or two 16-byte loads when they allow it
// (tetrahedra, hexahedra on a 16-byte aligned array), else 32-bit loads.
template <int CT>
__device__ __forceinline__ void cell_conn(const CellJob& j, uint64_t cell, uint32_t* raw)
{
    using Tr = CellTraits<CT>;
    const uint32_t* conn = j.conn + (uint64_t)Tr::kNodes * cell;
    if ((CT == KVSMC_TETRAHEDRA || CT == KVSMC_HEXAHEDRA) && j.conn_vec16) {
#pragma unroll
        for (int q = 0; q < Tr::kNodes / 4; ++q) {
            const uint4 w = __ldg(reinterpret_cast<const uint4*>(conn) + q);
            raw[4 * q] = w.x; raw[4 * q + 1] = w.y; raw[4 * q + 2] = w.z; raw[4 * q + 3] = w.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < Tr::kNodes; ++k) raw[k] = __ldg(conn + k);
    }
}

// The local node indices of a cell's connections, checked against the node count.
template <int CT>
__device__ __forceinline__ void cell_nodes_of(const CellJob& j, const uint32_t* raw, uint32_t* nodes)
{
    using Tr = CellTraits<CT>;
#pragma unroll
    for (int k = 0; k < Tr::kNodes; ++k) {
        uint32_t n = raw[Tr::node(k)];
        if (n >= j.nnodes) {
            atomicExch(j.bad_index, 1);
            n = 0;
        }
        nodes[k] = n;
    }
}

template <int CT>
__device__ __forceinline__ void cell_nodes(const CellJob& j, uint64_t cell, uint32_t* nodes)
{
    uint32_t raw[CellTraits<CT>::kNodes];
    cell_conn<CT>(j, cell, raw);
    cell_nodes_of<CT>(j, raw, nodes);
}

// The case: bit k iff double(value of local node k) > isolevel, decided
// without FP64 for float and up-to-32-bit integer values (Classifier).
template <int CT, typename T>
__device__ __forceinline__ unsigned case_of(const Classifier& cls, double iso, const T* v)
{
    using Tr = CellTraits<CT>;
    unsigned c = 0;
#pragma unroll
    for (int k = 0; k < Tr::kNodes; ++k) c |= above(cls, v[k]) ? (1u << k) : 0u;
    if (CT == KVSMC_PYRAMID && (c == 10u || c == 11u || c == 20u || c == 21u)) {
        // x / 4 as x * 0.25: the same correctly rounded result
        const double v1 = to_double(v[1]), v2 = to_double(v[2]);
        const double v3 = to_double(v[3]), v4 = to_double(v[4]);
        const double A = __dmul_rn(__dadd_rn(__dadd_rn(__dadd_rn(v1, v2), v3), v4), 0.25);
        const double B = __dmul_rn(__dsub_rn(__dadd_rn(__dadd_rn(-v1, v2), v3), v4), 0.25);
        const double C = __dmul_rn(__dadd_rn(__dadd_rn(__dsub_rn(-v1, v2), v3), v4), 0.25);
        const double D = __dmul_rn(__dsub_rn(__dadd_rn(__dsub_rn(v1, v2), v3), v4), 0.25);
        const double E = __dadd_rn(__dmul_rn(__dsub_rn(iso, A), D), __dmul_rn(B, C));
        if (c == 10u && E < 0) c = 32u;
        else if (c == 11u && E >= 0) c = 33u;
        else if (c == 20u && E >= 0) c = 34u;
        else if (c == 21u && E < 0) c = 35u;
    }
    return c;
}

// The nodes' values.
template <int CT, typename T>
__device__ __forceinline__ void cell_values(const CellJob& j, const uint32_t* nodes, T* v)
{
    const T* vals = static_cast<const T*>(j.values);
#pragma unroll
    for (int k = 0; k < CellTraits<CT>::kNodes; ++k) v[k] = __ldg(vals + nodes[k]);
}

// The reference's FP64 sequence, out of line (it runs for the vertices the
// FP32 certificate cannot decide, and for 32/64-bit integer and double values).
template <typename T>
static __device__ __noinline__ float3 cell_vertex_exact(const CellJob& j, double iso, uint32_t n0, uint32_t n1)
{
    const double lo = j.vmin, hi = j.vmax;
    double v0 = dval<T>(j.values, n0), v1 = dval<T>(j.values, n1);
    v0 = v0 <= lo ? lo : (v0 <= hi ? v0 : hi);   // Math::Clamp
    v1 = v1 <= lo ? lo : (v1 <= hi ? v1 : hi);
    const double q = __ddiv_rn(__dsub_rn(iso, v0), __dsub_rn(v1, v0));
    const double r = q < 0.0 ? -q : q;
    const float* c0 = j.coords + 3 * (uint64_t)n0;
    const float* c1 = j.coords + 3 * (uint64_t)n1;
    float3 o;
    o.x = __double2float_rn(__dadd_rn((double)c0[0], __dmul_rn(r, (double)__fsub_rn(c1[0], c0[0]))));
    o.y = __double2float_rn(__dadd_rn((double)c0[1], __dmul_rn(r, (double)__fsub_rn(c1[1], c0[1]))));
    o.z = __double2float_rn(__dadd_rn((double)c0[2], __dmul_rn(r, (double)__fsub_rn(c1[2], c0[2]))));
    return o;
}

// Value types whose values are floats exactly (the FP32 certificate applies).
template <typename T> struct CellFast { static constexpr bool value = false; };
template <> struct CellFast<float> { static constexpr bool value = true; };
template <> struct CellFast<int8_t> { static constexpr bool value = true; };
template <> struct CellFast<int16_t> { static constexpr bool value = true; };
template <> struct CellFast<uint8_t> { static constexpr bool value = true; };
template <> struct CellFast<uint16_t> { static constexpr bool value = true; };

// interpolate_vertex: the FP32 certificate (cell_ratio / cell_axis), else FP64.
template <typename T>
__device__ __forceinline__ float3 cell_vertex(const CellJob& j, const FastIso& f, double iso, uint32_t n0, uint32_t n1)
{
    if constexpr (CellFast<T>::value) {
        const T* vals = static_cast<const T*>(j.values);
        const float v0 = clampf_ref((float)__ldg(vals + n0), f.vmin_f, f.vmax_f);
        const float v1 = clampf_ref((float)__ldg(vals + n1), f.vmin_f, f.vmax_f);
        const CellRatio c = cell_ratio(v0, v1, f);
        const float* c0 = j.coords + 3 * (uint64_t)n0;
        const float* c1 = j.coords + 3 * (uint64_t)n1;
        float3 o;
        const bool ox = cell_axis(c, __ldg(c0), __ldg(c1), o.x);
        const bool oy = cell_axis(c, __ldg(c0 + 1), __ldg(c1 + 1), o.y);
        const bool oz = cell_axis(c, __ldg(c0 + 2), __ldg(c1 + 2), o.z);
        if (ox && oy && oz) return o;
    }
    return cell_vertex_exact<T>(j, iso, n0, n1);
}

// ---- kvs::SlicePlane on unstructured volumes (SlicePlane.cpp:291-800):
// per cell type, a case from the plane's sign at the cell's node coordinates
// (calculate_*_table_index, :828-942; no pyramid re-mapping), the cell type's
// triangle table in table order [i], [i+1], [i+2] for all four types, each
// vertex (1 - r) v0 + r v1 with r = |p0 / (p1 - p0)| in float on the node
// coordinates (interpolate_vertex, :986-995, no coordinate transform), its
// colour ColorMap::at of the value interpolated with the same r in the value
// type's arithmetic (interpolate_value, :1043-1056), one normal
// -((v2 - v0) x (v1 - v0)).

template <int CT>
__device__ __forceinline__ float3 node_xyz(const CellJob& j, uint32_t n)
{
    const float* c = j.coords + 3 * (uint64_t)n;
    return make_float3(__ldg(c), __ldg(c + 1), __ldg(c + 2));
}

template <int CT>
__device__ __forceinline__ unsigned slice_cell_case(const CellJob& j, const uint32_t* nodes)
{
    unsigned c = 0;
#pragma unroll
    for (int k = 0; k < CellTraits<CT>::kNodes; ++k) {
        const float3 p = node_xyz<CT>(j, nodes[k]);
        c |= plane_at(j, p.x, p.y, p.z) > 0.0f ? (1u << k) : 0u;
    }
    return c;
}

// A cell's case: of an isolevel, or of the plane.
template <int CT, typename T, bool SLICE>
__device__ __forceinline__ unsigned cell_case(const CellJob& j, const Classifier& cls, double iso, const uint32_t* nodes)
{
    if constexpr (SLICE) {
        return slice_cell_case<CT>(j, nodes);
    } else {
        T v[CellTraits<CT>::kNodes];
        cell_values<CT, T>(j, nodes, v);
        return case_of<CT, T>(cls, iso, v);
    }
}

template <typename T>
__device__ __forceinline__ void slice_cell_vertex(const CellJob& j, const float* unit, uint32_t n0, uint32_t n1,
                                                  float3& v, uchar3& rgb)
{
    const float3 a = node_xyz<0>(j, n0), b = node_xyz<0>(j, n1);
    const float p0 = plane_at(j, a.x, a.y, a.z), p1 = plane_at(j, b.x, b.y, b.z);
    const float r = fabsf(__fdiv_rn(p0, __fsub_rn(p1, p0)));
    const float s = __fsub_rn(1.0f, r);
    v.x = __fadd_rn(__fmul_rn(s, a.x), __fmul_rn(r, b.x));
    v.y = __fadd_rn(__fmul_rn(s, a.y), __fmul_rn(r, b.y));
    v.z = __fadd_rn(__fmul_rn(s, a.z), __fmul_rn(r, b.z));
    const T* vals = static_cast<const T*>(j.values);
    rgb = color_at(j, unit, slice_value(vals[n0], vals[n1], r));
}

// ---- the two passes.  A warp's work is a block of 2^block_shift consecutive
// groups of 32 cells (at most 32 groups; fewer on small meshes, so that every
// warp the GPU holds gets one, see cells_block_shift).
//
// Count: per group the word of its cells with triangles, per block the number
// of its triangles; kCountGroups groups' loads are in flight together.
// Bound by the latency of two dependent reads (connections, then values): 9.1e6
// tetrahedra (146 MB of connections) take 40 us, 57% of the copy rate; more
// groups in flight (8), or reading the next step's connections ahead (60 us:
// twice the registers), do not help.
template <int CT, typename T, bool SLICE>
__global__ void __launch_bounds__(kCellThreads) k_cells_count(CellJob j)
{
    using Tr = CellTraits<CT>;
    __shared__ typename Tr::Tables TB;
    load_tables(TB, Tr::tables());
    __syncthreads();
    const unsigned lane = threadIdx.x & 31u;
    const uint64_t groups = (j.ncells + 31) / 32;
    const uint64_t blk = (uint64_t)blockIdx.x * (kCellThreads / 32) + (threadIdx.x >> 5);
    const uint64_t g0 = blk << j.block_shift;
    if (g0 >= groups) return;
    const uint32_t ng = (uint32_t)(groups - g0 < (1ull << j.block_shift) ? groups - g0 : 1ull << j.block_shift);
    constexpr int G = kCountGroups<CT>;
    uint32_t sum = 0, mine = 0;   // this lane's triangles; the word of group g0 + lane
    for (uint32_t g = 0; g < ng; g += G) {
        uint32_t n[G];
#pragma unroll
        for (int q = 0; q < G; ++q) {
            const uint64_t c = (g0 + g + q) * 32 + lane;
            n[q] = 0;
            if (g + q < ng && c < j.ncells) {
                uint32_t nodes[Tr::kNodes];
                cell_nodes<CT>(j, c, nodes);
                n[q] = TB.counts[cell_case<CT, T, SLICE>(j, j.cls, j.iso, nodes)] & 15u;
            }
        }
#pragma unroll
        for (int q = 0; q < G; ++q) {
            const uint32_t word = __ballot_sync(FULL, n[q] != 0);
            if (lane == g + q) mine = word;
            sum += n[q];
        }
    }
    sum = __reduce_add_sync(FULL, sum);
    if (lane < ng) j.cut_words[g0 + lane] = mine;
    if (lane == 0) j.block_counts[blk] = sum;
}

// A warp's shared memory in the emit pass: the nodes of a round's cells (an
// odd stride: a column meets 32 banks) and the round's vertices.
template <int CT> struct alignas(16) CellWarp {
    static constexpr uint32_t kVerts = CT == KVSMC_TETRAHEDRA ? 128 : 192;
    float4 pv[kVerts];   // x, y, z, colour (slices)
    uint32_t nodes[32][CellTraits<CT>::kNodes | 1];
};

// Emit one block: lane u holds the cut cells' word of group u; their bits are
// one index space, taken 32 cells at a time, one per lane.  A round's vertices
// are then computed one per lane (each edge a cell uses once, whatever number
// of its triangles share it), and its triangles written one per lane, in cell
// and table order from `run` on.
template <int CT, typename T, bool SLICE>
__device__ __forceinline__ void emit_block(const CellJob& j, const Classifier& cls, double iso, const FastIso& f,
                                           float* out_coords, float* out_normals, uint64_t cap,
                                           const typename CellTraits<CT>::Tables& TB, CellWarp<CT>& W,
                                           const float* unit, uint32_t word, uint64_t g0, uint64_t run, unsigned lane)
{
    using Tr = CellTraits<CT>;
    // hexahedra and pyramids are packed in the mappers' [i], [i+2], [i+1]
    // order; the slicer takes [i], [i+1], [i+2]
    constexpr bool kSwapped = SLICE && (CT == KVSMC_HEXAHEDRA || CT == KVSMC_PYRAMID);
    const unsigned lt = (1u << lane) - 1u;
    const uint32_t cut = (uint32_t)__popc(word);
    uint32_t inc = cut;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(FULL, inc, o);
        if (lane >= (unsigned)o) inc += t;
    }
    const uint32_t ncut = __shfl_sync(FULL, inc, 31);
    uint32_t taken = 0;
    for (uint32_t r0 = 0; r0 < ncut; r0 += taken) {
        const uint32_t p = r0 + lane;
        bool has = p < ncut;
        uint32_t own = 0;   // its group: the first lane whose inclusive count exceeds p
#pragma unroll
        for (int s = 4; s >= 0; --s) {
            const uint32_t mid = own + (1u << s) - 1u;
            if (__shfl_sync(FULL, inc, mid) <= p) own = mid + 1;
        }
        own &= 31u;   // (lanes past the last cell)
        const uint32_t first = __shfl_sync(FULL, inc - cut, own), bits = __shfl_sync(FULL, word, own);
        unsigned code = 0;
        if (has) {
            const uint64_t cell = (g0 + own) * 32 + nth_set_bit(bits, p - first);
            uint32_t nodes[Tr::kNodes];
            cell_nodes<CT>(j, cell, nodes);
            code = cell_case<CT, T, SLICE>(j, cls, iso, nodes);
#pragma unroll
            for (int k = 0; k < Tr::kNodes; ++k) W.nodes[lane][k] = nodes[k];
        }
        const uint32_t cnt = has ? TB.counts[code] : 0u, ne = cnt >> 4;
        uint32_t vpre = 0;
#pragma unroll
        for (int bit = 0; bit < 4; ++bit) vpre += (uint32_t)__popc(__ballot_sync(FULL, (ne >> bit) & 1u) & lt) << bit;
        has = has && vpre + ne <= CellWarp<CT>::kVerts;   // a suffix of lanes waits
        taken = (uint32_t)__popc(__ballot_sync(FULL, has));
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
        __syncwarp();   // the nodes are there
        uint32_t seen = 0;
        for (uint32_t j0 = 0; j0 < nv; j0 += 32) {
            const uint32_t i = j0 + lane;
            // the cells' first items as bits: an item's cell is the number of first items up to it
            const uint32_t starts = __reduce_or_sync(FULL, has && vpre - j0 < 32u ? 1u << (vpre - j0) : 0u);
            const uint32_t q = seen + (uint32_t)__popc(starts & (lt | (1u << lane))) - 1u;
            seen += (uint32_t)__popc(starts);
            const uint32_t qe = __shfl_sync(FULL, pe, q);
            if (i < nv) {
                const uint32_t r = i - ((qe >> 8) & 0xfffu);
                const uint32_t ed = TB.edges[qe & 255u][r < 11u ? r : 11u];
                const uint32_t n0 = W.nodes[q][ed & 15u], n1 = W.nodes[q][ed >> 4];
                if constexpr (SLICE) {
                    float3 v;
                    uchar3 rgb;
                    slice_cell_vertex<T>(j, unit, n0, n1, v, rgb);
                    W.pv[i] = make_float4(v.x, v.y, v.z, __uint_as_float((uint32_t)rgb.x | ((uint32_t)rgb.y << 8) |
                                                                         ((uint32_t)rgb.z << 16)));
                } else {
                    const float3 v = cell_vertex<T>(j, f, iso, n0, n1);
                    W.pv[i] = make_float4(v.x, v.y, v.z, 0.0f);
                }
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
            if (i < ntr && t < cap) {   // never past the outputs
                const uint32_t sl = (uint32_t)(TB.slots[qe & 255u] >> (12 * (i - (qe >> 20))));
                const float4* pv = W.pv + ((qe >> 8) & 0xfffu);
                const float4 fa = pv[sl & 15u], fb = pv[(sl >> (kSwapped ? 8 : 4)) & 15u];
                const float4 fc = pv[(sl >> (kSwapped ? 4 : 8)) & 15u];
                const float3 A = make_float3(fa.x, fa.y, fa.z), B = make_float3(fb.x, fb.y, fb.z);
                const float3 C = make_float3(fc.x, fc.y, fc.z);
                store_triangle(out_coords + 9 * t, out_normals + 3 * t, A, B, C,
                               SLICE ? slice_normal(A, B, C) : tri_normal(A, B, C));
                if constexpr (SLICE) {
                    uint8_t* o = j.out_colors + 9 * t;
                    const float4 corner[3] = {fa, fb, fc};
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const uint32_t w = __float_as_uint(corner[k].w);
                        o[3 * k] = (uint8_t)w;
                        o[3 * k + 1] = (uint8_t)(w >> 8);
                        o[3 * k + 2] = (uint8_t)(w >> 16);
                    }
                }
            }
        }
        run += ntr;
        __syncwarp();
    }
}

// Emit, one isolevel or a slice: a warp per block.  9.1e6 tetrahedra, 6% of
// them cut: 88 us with a warp to each group of 32 cells and three vertices a
// triangle, 47 us.  Bound by latency: two or three rounds a warp, each a chain
// of dependent reads (connections, values, coordinates).
template <int CT, typename T, bool SLICE>
__global__ void __launch_bounds__(kCellThreads) k_cells_emit(CellJob j)
{
    using Tr = CellTraits<CT>;
    __shared__ typename Tr::Tables TB;
    __shared__ CellWarp<CT> sw[kCellThreads / 32];
    __shared__ float s_unit[SLICE ? 256 : 1];
    // launched before the host knows the total: nothing is written unless all fits
    if (j.d_total && *j.d_total > j.cap_tris) return;
    load_tables(TB, Tr::tables());
    if (SLICE) fill_unit(s_unit);
    __syncthreads();
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint64_t groups = (j.ncells + 31) / 32;
    const uint64_t blk = (uint64_t)blockIdx.x * (kCellThreads / 32) + warp;
    const uint64_t g0 = blk << j.block_shift;
    if (g0 >= groups) return;
    const uint32_t ng = (uint32_t)(groups - g0 < (1ull << j.block_shift) ? groups - g0 : 1ull << j.block_shift);
    emit_block<CT, T, SLICE>(j, j.cls, j.iso, j.f, j.out_coords, j.out_normals, j.cap_tris, TB, sw[warp], s_unit,
                             lane < ng ? j.cut_words[g0 + lane] : 0u, g0, j.block_offsets[blk], lane);
}

// ---- min/max over the cells' nodes (GetMinMaxValues with connections,
// UnstructuredVolumeObject.cpp:123-143): the scan starts at values[0] and
// then visits values[conn[p]] for every connection p in order; Min/Max keep
// the earlier value on ties and never take a NaN (a NaN values[0] stays).
template <typename T> struct CellMinMax {
    T lo, hi;
    unsigned long long ilo, ihi;   // scan positions (values[0] is position 0)
    int any;
};

template <typename T> __device__ __forceinline__ void cmm_combine(CellMinMax<T>& a, const CellMinMax<T>& b)
{
    if (!b.any) return;
    if (!a.any) { a = b; return; }
    if (b.lo < a.lo || (b.lo == a.lo && b.ilo < a.ilo)) { a.lo = b.lo; a.ilo = b.ilo; }
    if (b.hi > a.hi || (b.hi == a.hi && b.ihi < a.ihi)) { a.hi = b.hi; a.ihi = b.ihi; }
}

template <typename T> __device__ void cmm_block(CellMinMax<T>& m, CellMinMax<T>* sm)
{
    sm[threadIdx.x] = m;
    __syncthreads();
    for (unsigned s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            CellMinMax<T> a = sm[threadIdx.x];
            cmm_combine(a, sm[threadIdx.x + s]);
            sm[threadIdx.x] = a;
        }
        __syncthreads();
    }
    m = sm[0];
}

template <typename T>
__global__ void __launch_bounds__(kCellThreads) k_cells_minmax_partial(CellJob j, uint64_t nconn, CellMinMax<T>* partial)
{
    __shared__ CellMinMax<T> sm[kCellThreads];
    const T* vals = static_cast<const T*>(j.values);
    CellMinMax<T> m;
    m.any = 0; m.lo = T(0); m.hi = T(0); m.ilo = m.ihi = 0;
    const uint64_t per = (nconn + gridDim.x - 1) / gridDim.x;
    const uint64_t p0 = (uint64_t)blockIdx.x * per, p1 = p0 + per < nconn ? p0 + per : nconn;
    for (uint64_t p = p0 + threadIdx.x; p < p1; p += blockDim.x) {
        const uint32_t n = j.conn[p];
        if (n >= j.nnodes) { atomicExch(j.bad_index, 1); continue; }
        const T v = vals[n];
        if (v != v) continue;
        const unsigned long long pos = p + 1;
        if (!m.any) { m.lo = m.hi = v; m.ilo = m.ihi = pos; m.any = 1; continue; }
        if (v < m.lo) { m.lo = v; m.ilo = pos; }
        if (v > m.hi) { m.hi = v; m.ihi = pos; }
    }
    cmm_block(m, sm);
    if (threadIdx.x == 0) partial[blockIdx.x] = m;
}

template <typename T>
__global__ void __launch_bounds__(kCellThreads) k_cells_minmax_final(CellJob j, const CellMinMax<T>* partial, int n, double* out)
{
    __shared__ CellMinMax<T> sm[kCellThreads];
    CellMinMax<T> m;
    m.any = 0; m.lo = T(0); m.hi = T(0); m.ilo = m.ihi = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) cmm_combine(m, partial[i]);
    cmm_block(m, sm);
    if (threadIdx.x == 0) {
        const T first = static_cast<const T*>(j.values)[0];
        if (first != first) {
            out[0] = out[1] = to_double(first);
            return;
        }
        CellMinMax<T> f;
        f.lo = f.hi = first; f.ilo = f.ihi = 0; f.any = 1;
        cmm_combine(f, m);
        out[0] = to_double(f.lo);
        out[1] = to_double(f.hi);
    }
}

// ---- bounding box (UnstructuredVolumeObject::updateMinMaxCoords,
// UnstructuredVolumeObject.cpp:396-466): per axis the fold
// Min(cur, x) = cur < x ? cur : x (Max alike) over the sequence
// [conn[0], conn[0], conn[1], ...] of node coordinates (the nodes in order
// when there are no connections), from its first element.  A NaN x is
// taken and the next element replaces it, ties keep the later element.  So
// the result is NaN when the last element is NaN, else the min (max) over
// the elements after the last NaN, the latest on ties (the sign of a zero).

__device__ __forceinline__ uint64_t bounds_node(const CellJob& j, uint64_t p, bool has_conn)
{
    return has_conn ? (p == 0 ? j.conn[0] : j.conn[p - 1]) : p;
}

__global__ void __launch_bounds__(kCellThreads) k_bounds_last_nan(CellJob j, uint64_t npos, int has_conn,
                                                                  unsigned long long* last_nan)
{
    for (uint64_t p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; p < npos;
         p += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t n = bounds_node(j, p, has_conn != 0);
        if (n >= j.nnodes) { atomicExch(j.bad_index, 1); continue; }
        const float* c = j.coords + 3 * n;
#pragma unroll
        for (int ax = 0; ax < 3; ++ax)
            if (isnan(c[ax])) atomicMax(&last_nan[ax], (unsigned long long)(p + 1));
    }
}

struct BoundPart {
    float mn[3], mx[3];
    unsigned long long pmn[3], pmx[3];   // position + 1 (0: none)
};

__device__ __forceinline__ void bound_take(float& v, unsigned long long& pv, float w, unsigned long long pw, bool less)
{
    if (pw == 0) return;
    if (pv == 0 || (less ? w < v : w > v) || (w == v && pw > pv)) { v = w; pv = pw; }
}

__global__ void __launch_bounds__(kCellThreads) k_bounds_partial(CellJob j, uint64_t npos, int has_conn,
                                                                 const unsigned long long* last_nan, BoundPart* parts)
{
    __shared__ BoundPart sm[kCellThreads];
    BoundPart b;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) { b.mn[ax] = b.mx[ax] = 0.0f; b.pmn[ax] = b.pmx[ax] = 0; }
    const uint64_t per = (npos + gridDim.x - 1) / gridDim.x;
    const uint64_t p0 = (uint64_t)blockIdx.x * per, p1 = p0 + per < npos ? p0 + per : npos;
    for (uint64_t p = p0 + threadIdx.x; p < p1; p += blockDim.x) {
        const uint64_t n = bounds_node(j, p, has_conn != 0);
        if (n >= j.nnodes) continue;
        const float* c = j.coords + 3 * n;
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            if (p + 1 <= last_nan[ax]) continue;   // at or before the last NaN
            bound_take(b.mn[ax], b.pmn[ax], c[ax], p + 1, true);
            bound_take(b.mx[ax], b.pmx[ax], c[ax], p + 1, false);
        }
    }
    sm[threadIdx.x] = b;
    __syncthreads();
    for (unsigned st = blockDim.x / 2; st > 0; st >>= 1) {
        if (threadIdx.x < st) {
            BoundPart a = sm[threadIdx.x];
            const BoundPart& o = sm[threadIdx.x + st];
#pragma unroll
            for (int ax = 0; ax < 3; ++ax) {
                bound_take(a.mn[ax], a.pmn[ax], o.mn[ax], o.pmn[ax], true);
                bound_take(a.mx[ax], a.pmx[ax], o.mx[ax], o.pmx[ax], false);
            }
            sm[threadIdx.x] = a;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) parts[blockIdx.x] = sm[0];
}

__global__ void __launch_bounds__(kCellThreads) k_bounds_final(CellJob j, uint64_t npos, int has_conn,
                                                               const unsigned long long* last_nan,
                                                               const BoundPart* parts, int nparts, float* out)
{
    __shared__ BoundPart sm[kCellThreads];
    BoundPart b;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) { b.mn[ax] = b.mx[ax] = 0.0f; b.pmn[ax] = b.pmx[ax] = 0; }
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            bound_take(b.mn[ax], b.pmn[ax], parts[i].mn[ax], parts[i].pmn[ax], true);
            bound_take(b.mx[ax], b.pmx[ax], parts[i].mx[ax], parts[i].pmx[ax], false);
        }
    }
    sm[threadIdx.x] = b;
    __syncthreads();
    for (unsigned st = blockDim.x / 2; st > 0; st >>= 1) {
        if (threadIdx.x < st) {
            BoundPart a = sm[threadIdx.x];
            const BoundPart& o = sm[threadIdx.x + st];
#pragma unroll
            for (int ax = 0; ax < 3; ++ax) {
                bound_take(a.mn[ax], a.pmn[ax], o.mn[ax], o.pmn[ax], true);
                bound_take(a.mx[ax], a.pmx[ax], o.mx[ax], o.pmx[ax], false);
            }
            sm[threadIdx.x] = a;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const uint64_t last = bounds_node(j, npos - 1, has_conn != 0);
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            if (last_nan[ax] == npos && last < j.nnodes) {
                // the last element is a NaN: the fold ends on it
                out[ax] = out[3 + ax] = j.coords[3 * last + ax];
            } else {
                out[ax] = sm[0].mn[ax];
                out[3 + ax] = sm[0].mx[ax];
            }
        }
    }
}

// ---- isolevel sweep: one count pass classifies every cell for all the
// isolevels (its connections and node values read once), one scan over the
// isolevels' group counts, one emit pass over (isolevel, 32 groups) items.

template <int CT, typename T>
__global__ void __launch_bounds__(kCellThreads) k_cells_sweep_count(CellJob j)
{
    using Tr = CellTraits<CT>;
    __shared__ typename Tr::Tables TB;
    __shared__ CellIso s_iso[kCellSweepMax];
    load_tables(TB, Tr::tables());
    for (int i = threadIdx.x; i < j.niso; i += blockDim.x) s_iso[i] = j.isos[i];
    __syncthreads();
    const unsigned lane = threadIdx.x & 31u;
    const uint64_t groups = (j.ncells + 31) / 32, blocks = (groups + (1ull << j.block_shift) - 1) >> j.block_shift;
    const uint64_t blk = (uint64_t)blockIdx.x * (kCellThreads / 32) + (threadIdx.x >> 5);
    const uint64_t g0 = blk << j.block_shift;
    if (g0 >= groups) return;
    const uint32_t ng = (uint32_t)(groups - g0 < (1ull << j.block_shift) ? groups - g0 : 1ull << j.block_shift);
    uint32_t sum[2] = {0, 0};   // lane l: the block's triangles of isolevels l and l + 32
    for (uint32_t g = 0; g < ng; ++g) {
        const uint64_t cell = (g0 + g) * 32 + lane;
        const bool ok = cell < j.ncells;
        uint32_t nodes[Tr::kNodes];
        T v[Tr::kNodes];
        if (ok) {
            cell_nodes<CT>(j, cell, nodes);
            cell_values<CT, T>(j, nodes, v);
        }
        uint32_t words[2] = {0, 0};
        for (int k = 0; k < j.niso; ++k) {
            const uint32_t n = ok ? TB.counts[case_of<CT, T>(s_iso[k].cls, s_iso[k].iso, v)] & 15u : 0u;
            const uint32_t w = __ballot_sync(FULL, n != 0), t = __reduce_add_sync(FULL, n);
            if (lane == (unsigned)(k & 31)) {
                if (k < 32) { words[0] = w; sum[0] += t; }
                else { words[1] = w; sum[1] += t; }
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if ((int)lane + 32 * h < j.niso) j.cut_words[(lane + 32 * h) * groups + g0 + g] = words[h];
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
        if ((int)lane + 32 * h < j.niso) j.block_counts[(lane + 32 * h) * blocks + blk] = sum[h];
}

// A warp takes 2^emit_shift groups of one isolevel: a sweep has isolevels times
// blocks of work, so its blocks can be larger than the count's (whose triangles
// are consecutive).  2e5 tetrahedra, 64 isolevels, most groups cut by none: with
// the count's blocks of one group 205 us a call (emit 31), with blocks of 16 110
// (16).  Twice the count's blocks an SM: a warp's rounds over crowded blocks (every
// cell cut) would leave the last wave half empty.
template <int CT, typename T>
__global__ void __launch_bounds__(kCellThreads) k_cells_sweep_emit(CellJob j)
{
    using Tr = CellTraits<CT>;
    __shared__ typename Tr::Tables TB;
    __shared__ CellWarp<CT> sw[kCellThreads / 32];
    load_tables(TB, Tr::tables());
    __syncthreads();
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint64_t groups = (j.ncells + 31) / 32, blocks = (groups + (1ull << j.block_shift) - 1) >> j.block_shift;
    const uint64_t eblocks = (groups + (1ull << j.emit_shift) - 1) >> j.emit_shift;
    const uint64_t it = (uint64_t)blockIdx.x * (kCellThreads / 32) + warp;   // (isolevel, emit block)
    const uint64_t k = it / eblocks, eb = it - k * eblocks;
    if (k >= (uint64_t)j.niso) return;
    const uint64_t g0 = eb << j.emit_shift;
    const uint32_t ng = (uint32_t)(groups - g0 < (1ull << j.emit_shift) ? groups - g0 : 1ull << j.emit_shift);
    const CellIso& I = j.isos[k];
    emit_block<CT, T, false>(j, I.cls, I.iso, I.f, I.out_coords, I.out_normals, I.cap_tris, TB, sw[warp], nullptr,
                             lane < ng ? j.cut_words[k * groups + g0 + lane] : 0u, g0,
                             j.block_offsets[k * blocks + (g0 >> j.block_shift)] - I.base, lane);
}

// base[k] = the first scanned offset of isolevel k, base[niso] = the total.
__global__ void k_sweep_bases(const uint64_t* offsets, uint64_t blocks, int niso, const uint64_t* total, uint64_t* out)
{
    for (int k = threadIdx.x; k <= niso; k += blockDim.x) out[k] = k < niso ? offsets[(uint64_t)k * blocks] : *total;
}

// CTAs for `items` warps (at most (2^32 / 32 groups) x 64 isolevels: 2^30).
unsigned cell_grid(uint64_t items) { return (unsigned)((items + kCellThreads / 32 - 1) / (kCellThreads / 32)); }

#define KVSMC_CELL_SWITCH(CTV, DT, ...)                                                     \
    switch (CTV) {                                                                          \
    case KVSMC_TETRAHEDRA: { constexpr int CT = KVSMC_TETRAHEDRA; KVSMC_VALUE_SWITCH(DT, __VA_ARGS__); } break; \
    case KVSMC_HEXAHEDRA: { constexpr int CT = KVSMC_HEXAHEDRA; KVSMC_VALUE_SWITCH(DT, __VA_ARGS__); } break;   \
    case KVSMC_PYRAMID: { constexpr int CT = KVSMC_PYRAMID; KVSMC_VALUE_SWITCH(DT, __VA_ARGS__); } break;       \
    case KVSMC_PRISM: { constexpr int CT = KVSMC_PRISM; KVSMC_VALUE_SWITCH(DT, __VA_ARGS__); } break;           \
    default: return cudaErrorInvalidValue;                                                  \
    }

#define KVSMC_VALUE_SWITCH(DT, ...)                                 \
    switch (DT) {                                                   \
    case 0: { using T = int8_t; __VA_ARGS__; } break;               \
    case 1: { using T = int16_t; __VA_ARGS__; } break;              \
    case 2: { using T = int32_t; __VA_ARGS__; } break;              \
    case 3: { using T = long long; __VA_ARGS__; } break;            \
    case 4: { using T = uint8_t; __VA_ARGS__; } break;              \
    case 5: { using T = uint16_t; __VA_ARGS__; } break;             \
    case 6: { using T = uint32_t; __VA_ARGS__; } break;             \
    case 7: { using T = unsigned long long; __VA_ARGS__; } break;   \
    case 8: { using T = float; __VA_ARGS__; } break;                \
    case 9: { using T = double; __VA_ARGS__; } break;               \
    default: return cudaErrorInvalidValue;                          \
    }

}  // namespace

cudaError_t launch_cells_count(const CellJob& j, const Launch& L)
{
    if (j.ncells == 0) return cudaSuccess;
    prof_begin(L, "cells_count");
    KVSMC_CELL_SWITCH(j.cell_type, j.dtype, {
        k_cells_count<CT, T, false><<<cell_grid(cells_blocks(j.ncells, j.block_shift)), kCellThreads, 0, L.stream>>>(j);
    });
    prof_end(L);
    *L.counter += 1;
    return cudaGetLastError();
}

cudaError_t launch_cells_emit(const CellJob& j, const Launch& L)
{
    if (j.ncells == 0) return cudaSuccess;
    prof_begin(L, "cells_emit");
    KVSMC_CELL_SWITCH(j.cell_type, j.dtype, {
        k_cells_emit<CT, T, false><<<cell_grid(cells_blocks(j.ncells, j.block_shift)), kCellThreads, 0, L.stream>>>(j);
    });
    prof_end(L);
    *L.counter += 1;
    return cudaGetLastError();
}

cudaError_t launch_cells_slice_count(const CellJob& j, const Launch& L)
{
    if (j.ncells == 0) return cudaSuccess;
    prof_begin(L, "cells_slice_count");
    KVSMC_CELL_SWITCH(j.cell_type, j.dtype, {
        k_cells_count<CT, T, true><<<cell_grid(cells_blocks(j.ncells, j.block_shift)), kCellThreads, 0, L.stream>>>(j);
    });
    prof_end(L);
    *L.counter += 1;
    return cudaGetLastError();
}

cudaError_t launch_cells_slice_emit(const CellJob& j, const Launch& L)
{
    if (j.ncells == 0) return cudaSuccess;
    prof_begin(L, "cells_slice_emit");
    KVSMC_CELL_SWITCH(j.cell_type, j.dtype, {
        k_cells_emit<CT, T, true><<<cell_grid(cells_blocks(j.ncells, j.block_shift)), kCellThreads, 0, L.stream>>>(j);
    });
    prof_end(L);
    *L.counter += 1;
    return cudaGetLastError();
}

cudaError_t launch_cells_sweep_count(const CellJob& j, const Launch& L)
{
    if (j.ncells == 0 || j.niso <= 0) return cudaSuccess;
    prof_begin(L, "cells_sweep_count");
    KVSMC_CELL_SWITCH(j.cell_type, j.dtype, {
        k_cells_sweep_count<CT, T><<<cell_grid(cells_blocks(j.ncells, j.block_shift)), kCellThreads, 0, L.stream>>>(j);
    });
    prof_end(L);
    *L.counter += 1;
    return cudaGetLastError();
}

cudaError_t launch_cells_sweep_emit(const CellJob& j, const Launch& L)
{
    if (j.ncells == 0 || j.niso <= 0) return cudaSuccess;
    prof_begin(L, "cells_sweep_emit");
    KVSMC_CELL_SWITCH(j.cell_type, j.dtype, {
        k_cells_sweep_emit<CT, T><<<cell_grid(cells_blocks(j.ncells, j.emit_shift) * (uint64_t)j.niso), kCellThreads, 0, L.stream>>>(j);
    });
    prof_end(L);
    *L.counter += 1;
    return cudaGetLastError();
}

cudaError_t launch_sweep_bases(const uint64_t* offsets, uint64_t blocks, int niso, const uint64_t* total,
                               uint64_t* out, const Launch& L)
{
    k_sweep_bases<<<1, 96, 0, L.stream>>>(offsets, blocks, niso, total, out);
    *L.counter += 1;
    return cudaGetLastError();
}

size_t cells_bounds_scratch_bytes(int num_sms) { return 64 + (size_t)num_sms * 4 * sizeof(BoundPart); }

cudaError_t launch_cells_bounds(const CellJob& j, bool has_conn, void* scratch, float* d_out, const Launch& L)
{
    const uint64_t npos = has_conn ? j.ncells * (uint64_t)(j.cell_type == KVSMC_TETRAHEDRA ? 4 : j.cell_type ==
                                                           KVSMC_HEXAHEDRA ? 8 : j.cell_type == KVSMC_PYRAMID ? 5 : 6) + 1
                                   : j.nnodes;
    if (npos == 0) return cudaSuccess;
    unsigned long long* last_nan = static_cast<unsigned long long*>(scratch);
    BoundPart* parts = reinterpret_cast<BoundPart*>(static_cast<char*>(scratch) + 64);
    const int nb = L.num_sms * 4;
    cudaError_t e = cudaMemsetAsync(last_nan, 0, 3 * sizeof(unsigned long long), L.stream);
    if (e != cudaSuccess) return e;
    prof_begin(L, "cells_bounds");
    k_bounds_last_nan<<<nb, kCellThreads, 0, L.stream>>>(j, npos, has_conn ? 1 : 0, last_nan);
    k_bounds_partial<<<nb, kCellThreads, 0, L.stream>>>(j, npos, has_conn ? 1 : 0, last_nan, parts);
    k_bounds_final<<<1, kCellThreads, 0, L.stream>>>(j, npos, has_conn ? 1 : 0, last_nan, parts, nb, d_out);
    prof_end(L);
    *L.counter += 3;
    return cudaGetLastError();
}

size_t cells_minmax_scratch_bytes(int num_sms) { return (size_t)num_sms * 4 * 64; }

cudaError_t launch_cells_minmax(const CellJob& j, void* scratch, double* d_out, const Launch& L)
{
    const uint64_t nconn = j.ncells * (uint64_t)(j.cell_type == KVSMC_TETRAHEDRA ? 4 : j.cell_type == KVSMC_HEXAHEDRA ? 8
                                                 : j.cell_type == KVSMC_PYRAMID ? 5 : 6);
    const int nb = L.num_sms * 4;
    prof_begin(L, "cells_minmax");
    KVSMC_VALUE_SWITCH(j.dtype, {
        static_assert(sizeof(CellMinMax<T>) <= 64, "partial slot");
        CellMinMax<T>* part = static_cast<CellMinMax<T>*>(scratch);
        k_cells_minmax_partial<T><<<nb, kCellThreads, 0, L.stream>>>(j, nconn, part);
        k_cells_minmax_final<T><<<1, kCellThreads, 0, L.stream>>>(j, part, nb, d_out);
    });
    prof_end(L);
    *L.counter += 2;
    return cudaGetLastError();
}

uint64_t cells_groups(uint64_t ncells) { return (ncells + 31) / 32; }

uint64_t cells_blocks(uint64_t ncells, int block_shift)
{
    return (cells_groups(ncells) + (1ull << block_shift) - 1) >> block_shift;
}

// Groups per block (a power of two, at most 32, a lane each): as many as leave
// every SM 64 blocks, a block or two for each warp that an SM holds.  Larger
// blocks fill the emit's rounds and shorten the scan; fewer of them would leave
// warps idle: a mesh of 1e4 cells in blocks of one group takes 37 us a call,
// where one warp to 32 groups in turn took 90.
int cells_block_shift(uint64_t groups, int num_sms)
{
    int s = 0;
    while (s < 5 && (groups >> (s + 1)) >= (uint64_t)num_sms * 64) ++s;
    return s;
}

}  // namespace kvsmc

namespace {

using kvsmc_host::fail;

int nodes_per_cell(int ct)
{
    return ct == KVSMC_TETRAHEDRA ? 4 : ct == KVSMC_HEXAHEDRA ? 8 : ct == KVSMC_PYRAMID ? 5 : ct == KVSMC_PRISM ? 6 : 0;
}

// kvs::Math::Equal (Utility/Math.h:135-138)
bool equal_abs(double a, double b)
{
    const double d = a - b;
    return (d < 0 ? -d : d) < 1.e-6;
}

kvsmc_status check_args(kvsmc_context* ctx, int cell_type, int dtype, uint64_t nnodes, const void* values,
                        const float* coords, const uint32_t* connections, uint64_t ncells)
{
    if (nodes_per_cell(cell_type) == 0)
        return fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "cells: unknown cell type %d", cell_type);
    if (kvsmc::dtype_size(dtype) == 0) return fail(ctx, KVSMC_ERR_UNSUPPORTED_DTYPE, "cells: data type %d", dtype);
    if (nnodes == 0 || !values || !coords || (ncells && !connections))
        return fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "cells: empty or null volume arrays");
    // the mappers hold node ids in int and loop cells with a UInt32 counter
    if (nnodes > 0x7fffffffull || ncells > 0xffffffffull)
        return fail(ctx, KVSMC_ERR_TOO_LARGE, "cells: %llu nodes / %llu cells beyond the 32-bit ids",
                    (unsigned long long)nnodes, (unsigned long long)ncells);
    return KVSMC_OK;
}

// The count pass's scratch (group words, block counts, offsets, scan scratch, a tail for
// the total or the min/max) in the context's arena, and the bad-index flag.
struct CellsScratch {
    void* d_scan;
    uint64_t* d_tail;
    uint64_t blocks;     // of one isolevel
    uint64_t nscan;      // scanned entries: blocks x isolevels
    void* d_extra;       // sweep: isolevel records (kCellSweepMax) and bases (kCellSweepMax + 1)
};

kvsmc_status cells_prepare(kvsmc_context* ctx, kvsmc::CellJob& j, CellsScratch* sc, int niso = 1)
{
    using namespace kvsmc_host;
    if (!ctx->d_flag) KVSMC_CUDA(ctx, kvsmc_host::device_malloc(ctx, &ctx->d_flag, sizeof(int)));
    j.bad_index = ctx->d_flag;
    KVSMC_CUDA(ctx, cudaMemsetAsync(ctx->d_flag, 0, sizeof(int), ctx->stream));
    j.block_shift = kvsmc::cells_block_shift(kvsmc::cells_groups(j.ncells), ctx->num_sms);
    // (whole blocks of the count: half of one isolevel's groups asks for less)
    j.emit_shift = std::max(j.block_shift, kvsmc::cells_block_shift(kvsmc::cells_groups(j.ncells) * (uint64_t)niso / 2,
                                                                    ctx->num_sms));
    sc->blocks = kvsmc::cells_blocks(j.ncells, j.block_shift);
    sc->nscan = sc->blocks * (uint64_t)niso;
    const size_t bw = align_up(kvsmc::cells_groups(j.ncells) * (uint64_t)niso * 4, 256),
                 bc = align_up(sc->nscan * 4, 256), bo = align_up(sc->nscan * 8, 256),
                 bs = align_up(std::max(std::max(kvsmc::scan_scratch_bytes(sc->nscan),
                                                 kvsmc::cells_minmax_scratch_bytes(ctx->num_sms)),
                                        kvsmc::minmax_scratch_bytes(ctx->num_sms)), 256),
                 be = align_up(kvsmc::kCellSweepMax * sizeof(kvsmc::CellIso) + (kvsmc::kCellSweepMax + 1) * 8, 256);
    kvsmc_status st = ensure_scratch(ctx, bw + bc + bo + bs + 256 + be);
    if (st) return st;
    char* base = static_cast<char*>(ctx->scratch);
    j.cut_words = reinterpret_cast<uint32_t*>(base);
    base += bw;
    j.block_counts = reinterpret_cast<uint32_t*>(base);
    j.block_offsets = reinterpret_cast<uint64_t*>(base + bc);
    sc->d_scan = base + bc + bo;
    sc->d_tail = reinterpret_cast<uint64_t*>(base + bc + bo + bs);
    sc->d_extra = base + bc + bo + bs + 256;
    return KVSMC_OK;
}

int read_bad(kvsmc_context* ctx)
{
    int bad = 0;
    std::memcpy(&bad, ctx->h_small + 2, sizeof(int));
    return bad;
}

// Min/max (when not given) and the Math::Equal early exit.  *go is false
// when no cell is to be visited; sizes holds the range.
kvsmc_status cells_range(kvsmc_context* ctx, kvsmc::CellJob& j, const CellsScratch& sc, int32_t has_minmax,
                         double min_value, double max_value, kvsmc_sizes* sizes, bool* go)
{
    using namespace kvsmc_host;
    *go = false;
    const kvsmc::Launch L = launch_of(ctx);
    // MapperBase::setRange: the volume's min/max, computed when not set
    double vmin = min_value, vmax = max_value;
    if (!has_minmax) {
        if (j.ncells) {
            KVSMC_CUDA(ctx, kvsmc::launch_cells_minmax(j, sc.d_scan, reinterpret_cast<double*>(sc.d_tail), L));
        } else {
            // no connections: the scan runs over the nodes (UnstructuredVolumeObject.cpp:88-102)
            kvsmc::VolumeView v1;
            std::memset(&v1, 0, sizeof v1);
            v1.data = j.values;
            v1.dtype = j.dtype;
            v1.nx = (uint32_t)j.nnodes;
            v1.ny = v1.nz = 1;
            v1.pitch = v1.slice = j.nnodes;
            KVSMC_CUDA(ctx, kvsmc::launch_minmax(v1, sc.d_scan, reinterpret_cast<double*>(sc.d_tail), L));
        }
        KVSMC_CUDA(ctx, cudaMemcpyAsync(ctx->h_small, sc.d_tail, 2 * sizeof(double), cudaMemcpyDeviceToHost,
                                        ctx->stream));
        KVSMC_CUDA(ctx, cudaMemcpyAsync(ctx->h_small + 2, ctx->d_flag, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
        KVSMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        std::memcpy(&vmin, ctx->h_small, sizeof(double));
        std::memcpy(&vmax, ctx->h_small + 1, sizeof(double));
        if (read_bad(ctx)) return fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "cells: a connection index is >= nnodes");
    }
    sizes->min_value = vmin;
    sizes->max_value = vmax;
    if (equal_abs(vmin, vmax)) return KVSMC_OK;   // MarchingTetrahedra.cpp:118-119
    sizes->extracted = 1;
    if (j.ncells == 0) return KVSMC_OK;
    j.vmin = vmin;
    j.vmax = vmax;
    j.f = make_fast(j.iso, vmin, vmax, j.dtype);
    *go = true;
    return KVSMC_OK;
}

// Count and scan (total in sc.d_tail), and, when `emit` is set, the emit pass
// right behind them with the caller's capacity, guarded on the device by the
// total; then one read-back of the total and the flag.
kvsmc_status cells_passes(kvsmc_context* ctx, kvsmc::CellJob& j, const CellsScratch& sc, bool emit,
                          kvsmc_sizes* sizes)
{
    using namespace kvsmc_host;
    const kvsmc::Launch L = launch_of(ctx);
    KVSMC_CUDA(ctx, kvsmc::launch_cells_count(j, L));
    KVSMC_CUDA(ctx, kvsmc::launch_scan(j.block_counts, j.block_offsets, sc.nscan, sc.d_scan, sc.d_tail, L));
    if (emit) {
        j.d_total = sc.d_tail;
        KVSMC_CUDA(ctx, kvsmc::launch_cells_emit(j, L));
    }
    KVSMC_CUDA(ctx, cudaMemcpyAsync(ctx->h_small, sc.d_tail, sizeof(uint64_t), cudaMemcpyDeviceToHost, ctx->stream));
    KVSMC_CUDA(ctx, cudaMemcpyAsync(ctx->h_small + 2, ctx->d_flag, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    KVSMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (read_bad(ctx)) return fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "cells: a connection index is >= nnodes");
    const uint64_t t = ctx->h_small[0];
    sizes->ntriangles = t;
    sizes->nvertices = 3 * t;
    sizes->ncoords = 9 * t;
    sizes->nnormals = 3 * t;
    return KVSMC_OK;
}

kvsmc::CellJob make_job(int cell_type, int dtype, const void* values, uint64_t nnodes, const float* coords,
                        const uint32_t* conn, uint64_t ncells, double isolevel)
{
    kvsmc::CellJob j;
    std::memset(&j, 0, sizeof j);
    j.cell_type = cell_type;
    j.dtype = dtype;
    j.values = values;
    j.nnodes = nnodes;
    j.coords = coords;
    j.conn = conn;
    j.ncells = ncells;
    j.iso = isolevel;
    j.cls = kvsmc_host::make_classifier(isolevel);
    j.conn_vec16 = (reinterpret_cast<uintptr_t>(conn) & 15u) == 0;
    return j;
}

}  // namespace

extern "C" {

kvsmc_status kvsmc_marching_cells_device(kvsmc_context* ctx, kvsmc_cell_type cell_type, const void* values,
                                         kvsmc_dtype dtype, uint64_t nnodes, const float* coords,
                                         const uint32_t* connections, uint64_t ncells, double isolevel,
                                         int32_t has_minmax, double min_value, double max_value, float* out_coords,
                                         uint64_t coords_capacity, float* out_normals, uint64_t normals_capacity,
                                         kvsmc_sizes* sizes)
{
    using namespace kvsmc_host;
    if (!ctx || !sizes) return KVSMC_ERR_INVALID_ARGUMENT;
    std::memset(sizes, 0, sizeof *sizes);
    kvsmc_status st = check_args(ctx, cell_type, dtype, nnodes, values, coords, connections, ncells);
    if (st) return st;
    KVSMC_CUDA(ctx, cudaSetDevice(ctx->device));
    kvsmc::CellJob j = make_job(cell_type, dtype, values, nnodes, coords, connections, ncells, isolevel);
    CellsScratch sc;
    bool go = false;
    if ((st = cells_prepare(ctx, j, &sc)) || (st = cells_range(ctx, j, sc, has_minmax, min_value, max_value, sizes,
                                                                &go)) || !go)
        return st;
    // emit behind the count when outputs are given (the kernel writes nothing
    // unless the total fits them): one host round trip per call
    const bool outs = out_coords && out_normals;
    j.out_coords = out_coords;
    j.out_normals = out_normals;
    j.cap_tris = outs ? std::min(coords_capacity / 9, normals_capacity / 3) : 0;
    if ((st = cells_passes(ctx, j, sc, outs, sizes))) return st;
    const uint64_t t = sizes->ntriangles;
    if (t > j.cap_tris && t > 0)
        return fail(ctx, KVSMC_ERR_CAPACITY, "cells: %llu triangles do not fit the outputs", (unsigned long long)t);
    return KVSMC_OK;
}

kvsmc_status kvsmc_marching_cells_host(kvsmc_context* ctx, kvsmc_cell_type cell_type, const void* values,
                                       kvsmc_dtype dtype, uint64_t nnodes, const float* coords,
                                       const uint32_t* connections, uint64_t ncells, double isolevel,
                                       int32_t has_minmax, double min_value, double max_value,
                                       kvsmc_host_alloc_fn alloc, void* user, kvsmc_sizes* sizes)
{
    using namespace kvsmc_host;
    if (!ctx || !alloc || !sizes) return KVSMC_ERR_INVALID_ARGUMENT;
    std::memset(sizes, 0, sizeof *sizes);
    kvsmc_status st = check_args(ctx, cell_type, dtype, nnodes, values, coords, connections, ncells);
    if (st) return st;
    KVSMC_CUDA(ctx, cudaSetDevice(ctx->device));
    const int npc = nodes_per_cell(cell_type);
    const size_t es = kvsmc::dtype_size(dtype);
    // inputs and outputs in one device allocation: values | coords | connections | outputs
    const size_t bv = align_up(nnodes * es, 256), bx = align_up(nnodes * 12, 256),
                 bk = align_up(std::max<uint64_t>(1, ncells * npc) * 4, 256);
    char* d_in = nullptr;
    float* d_out = nullptr;
    auto done = [&](kvsmc_status s) {
        cudaStreamSynchronize(ctx->stream);
        cudaFree(d_in);
        cudaFree(d_out);
        return s;
    };
    cudaError_t e = kvsmc_host::device_malloc(ctx, &d_in, bv + bx + bk);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_in, values, nnodes * es, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_in + bv, coords, nnodes * 12, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess && ncells)
        e = cudaMemcpyAsync(d_in + bv + bx, connections, ncells * npc * 4, cudaMemcpyHostToDevice, ctx->stream);
    if (e != cudaSuccess)
        return done(fail(ctx, e == cudaErrorMemoryAllocation ? KVSMC_ERR_OUT_OF_MEMORY : KVSMC_ERR_CUDA,
                         "cells: %s", cudaGetErrorString(e)));
    kvsmc::CellJob j = make_job(cell_type, dtype, d_in, nnodes, reinterpret_cast<const float*>(d_in + bv),
                                reinterpret_cast<const uint32_t*>(d_in + bv + bx), ncells, isolevel);
    CellsScratch sc;
    bool go = false;
    if ((st = cells_prepare(ctx, j, &sc)) || (st = cells_range(ctx, j, sc, has_minmax, min_value, max_value, sizes,
                                                                &go)) || !go ||
        (st = cells_passes(ctx, j, sc, false, sizes)) || sizes->ntriangles == 0)
        return done(st);
    const uint64_t t = sizes->ntriangles;
    if ((e = kvsmc_host::device_malloc(ctx, &d_out, t * 12 * sizeof(float))) != cudaSuccess)
        return done(fail(ctx, KVSMC_ERR_OUT_OF_MEMORY, "cells: %s", cudaGetErrorString(e)));
    j.out_coords = d_out;
    j.out_normals = d_out + 9 * t;
    j.cap_tris = t;
    if ((e = kvsmc::launch_cells_emit(j, launch_of(ctx))) != cudaSuccess)
        return done(fail(ctx, KVSMC_ERR_CUDA, "cells: %s", cudaGetErrorString(e)));
    void* hc = alloc(user, 0, 9 * t);
    void* hn = hc ? alloc(user, 1, 3 * t) : nullptr;
    if (!hc || !hn) return done(fail(ctx, KVSMC_ERR_OUT_OF_MEMORY, "cells: host alloc"));
    e = cudaMemcpyAsync(hc, d_out, t * 9 * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(hn, d_out + 9 * t, t * 3 * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return done(fail(ctx, KVSMC_ERR_CUDA, "cells: %s", cudaGetErrorString(e)));
    return done(KVSMC_OK);
}

kvsmc_status kvsmc_slice_cells_host(kvsmc_context* ctx, kvsmc_cell_type cell_type, const void* values,
                                    kvsmc_dtype dtype, uint64_t nnodes, const float* coords,
                                    const uint32_t* connections, uint64_t ncells, const kvsmc_slice_params* p,
                                    kvsmc_host_alloc_fn alloc, void* user, uint64_t* ntriangles)
{
    using namespace kvsmc_host;
    if (!ctx || !alloc || !ntriangles) return KVSMC_ERR_INVALID_ARGUMENT;
    *ntriangles = 0;
    if (!p || !p->tf_table || p->tf_resolution < 1)
        return fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "slice: bad parameters (colour table)");
    kvsmc_status st = check_args(ctx, cell_type, dtype, nnodes, values, coords, connections, ncells);
    if (st) return st;
    KVSMC_CUDA(ctx, cudaSetDevice(ctx->device));
    if (ncells == 0) return KVSMC_OK;
    const int npc = nodes_per_cell(cell_type);
    const size_t es = kvsmc::dtype_size(dtype);
    // values | coords | connections | colour table in one device allocation
    const size_t bv = align_up(nnodes * es, 256), bx = align_up(nnodes * 12, 256), bk = align_up(ncells * npc * 4, 256),
                 bt = align_up((size_t)3 * p->tf_resolution, 256);
    char* d_in = nullptr;
    char* d_out = nullptr;
    auto done = [&](kvsmc_status s) {
        cudaStreamSynchronize(ctx->stream);
        cudaFree(d_in);
        cudaFree(d_out);
        return s;
    };
    cudaError_t e = kvsmc_host::device_malloc(ctx, &d_in, bv + bx + bk + bt);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_in, values, nnodes * es, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_in + bv, coords, nnodes * 12, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(d_in + bv + bx, connections, ncells * npc * 4, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(d_in + bv + bx + bk, p->tf_table, (size_t)3 * p->tf_resolution, cudaMemcpyHostToDevice,
                            ctx->stream);
    if (e != cudaSuccess)
        return done(fail(ctx, e == cudaErrorMemoryAllocation ? KVSMC_ERR_OUT_OF_MEMORY : KVSMC_ERR_CUDA,
                         "slice cells: %s", cudaGetErrorString(e)));
    kvsmc::CellJob j = make_job(cell_type, dtype, d_in, nnodes, reinterpret_cast<const float*>(d_in + bv),
                                reinterpret_cast<const uint32_t*>(d_in + bv + bx), ncells, 0.0);
    for (int k = 0; k < 4; ++k) j.coef[k] = p->coefficients[k];
    j.tf_min = p->tf_min;
    j.tf_max = p->tf_max;
    j.tf_res = p->tf_resolution;
    j.table = reinterpret_cast<const uint8_t*>(d_in + bv + bx + bk);
    CellsScratch sc;
    if ((st = cells_prepare(ctx, j, &sc))) return done(st);
    const kvsmc::Launch L = launch_of(ctx);
    e = kvsmc::launch_cells_slice_count(j, L);
    if (e == cudaSuccess) e = kvsmc::launch_scan(j.block_counts, j.block_offsets, sc.nscan, sc.d_scan, sc.d_tail, L);
    if (e == cudaSuccess) e = cudaMemcpyAsync(ctx->h_small, sc.d_tail, sizeof(uint64_t), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(ctx->h_small + 2, ctx->d_flag, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return done(fail(ctx, KVSMC_ERR_CUDA, "slice cells: %s", cudaGetErrorString(e)));
    if (read_bad(ctx)) return done(fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "cells: a connection index is >= nnodes"));
    const uint64_t t = ctx->h_small[0];
    *ntriangles = t;
    if (t == 0) return done(KVSMC_OK);
    const size_t oc = align_up(t * 36, 256), on = align_up(t * 12, 256);
    if ((e = kvsmc_host::device_malloc(ctx, &d_out, oc + on + t * 9)) != cudaSuccess)
        return done(fail(ctx, KVSMC_ERR_OUT_OF_MEMORY, "slice cells: %s", cudaGetErrorString(e)));
    j.out_coords = reinterpret_cast<float*>(d_out);
    j.out_normals = reinterpret_cast<float*>(d_out + oc);
    j.out_colors = reinterpret_cast<uint8_t*>(d_out + oc + on);
    j.cap_tris = t;
    if ((e = kvsmc::launch_cells_slice_emit(j, L)) != cudaSuccess)
        return done(fail(ctx, KVSMC_ERR_CUDA, "slice cells: %s", cudaGetErrorString(e)));
    void* hc = alloc(user, 0, 9 * t);
    void* hn = hc ? alloc(user, 1, 3 * t) : nullptr;
    void* hk = hn ? alloc(user, 3, 9 * t) : nullptr;
    if (!hc || !hn || !hk) return done(fail(ctx, KVSMC_ERR_OUT_OF_MEMORY, "slice cells: host alloc"));
    e = cudaMemcpyAsync(hc, j.out_coords, t * 36, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(hn, j.out_normals, t * 12, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(hk, j.out_colors, t * 9, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return done(fail(ctx, KVSMC_ERR_CUDA, "slice cells: %s", cudaGetErrorString(e)));
    return done(KVSMC_OK);
}

kvsmc_status kvsmc_cells_bounds(kvsmc_context* ctx, kvsmc_cell_type cell_type, const float* coords, uint64_t nnodes,
                                const uint32_t* connections, uint64_t ncells, float* min_coord, float* max_coord)
{
    using namespace kvsmc_host;
    if (!ctx || !min_coord || !max_coord) return KVSMC_ERR_INVALID_ARGUMENT;
    const int npc = nodes_per_cell(cell_type);
    if (npc == 0) return fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "cells: unknown cell type %d", (int)cell_type);
    if (nnodes == 0 || !coords || (ncells && !connections))
        return fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "cells: empty or null volume arrays");
    KVSMC_CUDA(ctx, cudaSetDevice(ctx->device));
    const size_t bx = align_up(nnodes * 12, 256), bk = align_up(std::max<uint64_t>(1, ncells * npc) * 4, 256);
    char* d_in = nullptr;
    auto done = [&](kvsmc_status st) {
        cudaStreamSynchronize(ctx->stream);
        cudaFree(d_in);
        return st;
    };
    cudaError_t e = kvsmc_host::device_malloc(ctx, &d_in, bx + bk);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_in, coords, nnodes * 12, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess && ncells)
        e = cudaMemcpyAsync(d_in + bx, connections, ncells * npc * 4, cudaMemcpyHostToDevice, ctx->stream);
    if (e != cudaSuccess)
        return done(fail(ctx, e == cudaErrorMemoryAllocation ? KVSMC_ERR_OUT_OF_MEMORY : KVSMC_ERR_CUDA,
                         "cells bounds: %s", cudaGetErrorString(e)));
    kvsmc::CellJob j = make_job(cell_type, KVSMC_F32, nullptr, nnodes, reinterpret_cast<const float*>(d_in),
                                reinterpret_cast<const uint32_t*>(d_in + bx), ncells, 0.0);
    const size_t bs = align_up(kvsmc::cells_bounds_scratch_bytes(ctx->num_sms), 256);
    kvsmc_status st = ensure_scratch(ctx, bs + 256);
    if (st) return done(st);
    if (!ctx->d_flag) {
        if ((e = kvsmc_host::device_malloc(ctx, &ctx->d_flag, sizeof(int))) != cudaSuccess)
            return done(fail(ctx, KVSMC_ERR_OUT_OF_MEMORY, "cells bounds: %s", cudaGetErrorString(e)));
    }
    j.bad_index = ctx->d_flag;
    char* base = static_cast<char*>(ctx->scratch);
    float* d_out = reinterpret_cast<float*>(base + bs);
    e = cudaMemsetAsync(ctx->d_flag, 0, sizeof(int), ctx->stream);
    if (e == cudaSuccess) e = kvsmc::launch_cells_bounds(j, ncells > 0, base, d_out, launch_of(ctx));
    if (e == cudaSuccess) e = cudaMemcpyAsync(ctx->h_small, d_out, 6 * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream);
    // the six floats fill h_small[0..2]; the flag goes behind them
    if (e == cudaSuccess) e = cudaMemcpyAsync(ctx->h_small + 4, ctx->d_flag, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return done(fail(ctx, KVSMC_ERR_CUDA, "cells bounds: %s", cudaGetErrorString(e)));
    int bad = 0;
    std::memcpy(&bad, ctx->h_small + 4, sizeof(int));
    if (bad) return done(fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "cells: a connection index is >= nnodes"));
    float out[6];
    std::memcpy(out, ctx->h_small, sizeof out);
    for (int k = 0; k < 3; ++k) {
        min_coord[k] = out[k];
        max_coord[k] = out[3 + k];
    }
    return done(KVSMC_OK);
}

kvsmc_status kvsmc_marching_cells_sweep_device(kvsmc_context* ctx, kvsmc_cell_type cell_type, const void* values,
                                               kvsmc_dtype dtype, uint64_t nnodes, const float* coords,
                                               const uint32_t* connections, uint64_t ncells,
                                               const double* isolevels, int32_t niso, int32_t has_minmax,
                                               double min_value, double max_value, float* const* out_coords,
                                               const uint64_t* coords_capacity, float* const* out_normals,
                                               const uint64_t* normals_capacity, kvsmc_sizes* sizes)
{
    using namespace kvsmc_host;
    if (!ctx || !isolevels || !sizes || niso < 1) return KVSMC_ERR_INVALID_ARGUMENT;
    if (niso > kvsmc::kCellSweepMax)
        return fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "cells sweep: %d isolevels (at most %d)", (int)niso,
                    kvsmc::kCellSweepMax);
    std::memset(sizes, 0, sizeof(kvsmc_sizes) * (size_t)niso);
    kvsmc_status st = check_args(ctx, cell_type, dtype, nnodes, values, coords, connections, ncells);
    if (st) return st;
    KVSMC_CUDA(ctx, cudaSetDevice(ctx->device));
    kvsmc::CellJob j = make_job(cell_type, dtype, values, nnodes, coords, connections, ncells, isolevels[0]);
    CellsScratch sc;
    bool go = false;
    if ((st = cells_prepare(ctx, j, &sc, niso)) ||
        (st = cells_range(ctx, j, sc, has_minmax, min_value, max_value, &sizes[0], &go)))
        return st;
    for (int k = 1; k < niso; ++k) {
        sizes[k].min_value = sizes[0].min_value;
        sizes[k].max_value = sizes[0].max_value;
        sizes[k].extracted = sizes[0].extracted;
    }
    if (!go) return KVSMC_OK;
    std::vector<kvsmc::CellIso> isos((size_t)niso);
    for (int k = 0; k < niso; ++k) {
        kvsmc::CellIso& I = isos[k];
        std::memset(&I, 0, sizeof I);
        I.iso = isolevels[k];
        I.cls = make_classifier(isolevels[k]);
        I.f = make_fast(isolevels[k], j.vmin, j.vmax, j.dtype);
    }
    kvsmc::CellIso* d_isos = static_cast<kvsmc::CellIso*>(sc.d_extra);
    uint64_t* d_bases = reinterpret_cast<uint64_t*>(static_cast<char*>(sc.d_extra) +
                                                    kvsmc::kCellSweepMax * sizeof(kvsmc::CellIso));
    j.isos = d_isos;
    j.niso = niso;
    const kvsmc::Launch L = launch_of(ctx);
    KVSMC_CUDA(ctx, cudaMemcpyAsync(d_isos, isos.data(), sizeof(kvsmc::CellIso) * niso, cudaMemcpyHostToDevice,
                                    ctx->stream));
    KVSMC_CUDA(ctx, kvsmc::launch_cells_sweep_count(j, L));
    KVSMC_CUDA(ctx, kvsmc::launch_scan(j.block_counts, j.block_offsets, sc.nscan, sc.d_scan, sc.d_tail, L));
    KVSMC_CUDA(ctx, kvsmc::launch_sweep_bases(j.block_offsets, sc.blocks, niso, sc.d_tail, d_bases, L));
    std::vector<uint64_t> bases((size_t)niso + 1);
    int bad = 0;
    KVSMC_CUDA(ctx, cudaMemcpyAsync(bases.data(), d_bases, 8 * ((size_t)niso + 1), cudaMemcpyDeviceToHost, ctx->stream));
    KVSMC_CUDA(ctx, cudaMemcpyAsync(&bad, ctx->d_flag, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    KVSMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (bad) return fail(ctx, KVSMC_ERR_INVALID_ARGUMENT, "cells: a connection index is >= nnodes");
    bool fits = out_coords && out_normals && coords_capacity && normals_capacity;
    for (int k = 0; k < niso; ++k) {
        const uint64_t t = bases[k + 1] - bases[k];
        sizes[k].ntriangles = t;
        sizes[k].nvertices = 3 * t;
        sizes[k].ncoords = 9 * t;
        sizes[k].nnormals = 3 * t;
        if (t && (!fits || !out_coords[k] || !out_normals[k] || coords_capacity[k] < 9 * t ||
                  normals_capacity[k] < 3 * t))
            fits = false;
        isos[k].base = bases[k];
        isos[k].out_coords = fits ? out_coords[k] : nullptr;
        isos[k].out_normals = fits ? out_normals[k] : nullptr;
        isos[k].cap_tris = t;
    }
    if (!fits) return fail(ctx, KVSMC_ERR_CAPACITY, "cells sweep: the triangles do not fit the outputs");
    if (bases[niso] == 0) return KVSMC_OK;
    KVSMC_CUDA(ctx, cudaMemcpyAsync(d_isos, isos.data(), sizeof(kvsmc::CellIso) * niso, cudaMemcpyHostToDevice,
                                    ctx->stream));
    KVSMC_CUDA(ctx, kvsmc::launch_cells_sweep_emit(j, L));
    // the records' host copy must outlive the copies above
    KVSMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return KVSMC_OK;
}

}  // extern "C"
