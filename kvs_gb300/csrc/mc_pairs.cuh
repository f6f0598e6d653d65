// mc_pairs.cuh -- what the kernels over listed pairs share: the case tables by
// corner code, and the walk over a block of units' pairs, one per lane.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "mc_internal.h"
#include "mc_interp.cuh"
#include "mc_tables.h"

namespace kvsmc {

constexpr int kPairThreads = 256;
constexpr int kPairWarps = kPairThreads / 32;
constexpr int kPairVerts = 192;          // vertex items of one round

namespace {

constexpr unsigned FULL = 0xffffffffu;

// Case tables indexed by the corner code (bit r: row r's node i above, rows
// (y, z) (y+1, z) (y, z+1) (y+1, z+1); bit 4 + r: its node i + 1), laid out
// at compile time and copied into shared memory by one bulk copy per CTA.
struct alignas(16) PairTables {
    uint64_t tri_slots[256];   // per triangle corner: its edge's rank among the used edges, 4 bits each
    uint8_t edges[256][12];    // the used edges in increasing order: corner A | corner B << 3 | axis << 6
                               // (corner: dx + 2 dy + 4 dz)
    uint8_t counts[256];       // triangles | used edges << 3
    uint8_t users[256][12];    // per used edge, in their order: the triangles that use it, as bits
};
static_assert(sizeof(PairTables) % 16 == 0, "copied by a bulk copy");

constexpr uint64_t h_tri[256] = MC_TRI_PACKED_INIT;
constexpr uint8_t h_ntri[256] = MC_NTRI_INIT;
constexpr uint16_t h_mask[256] = MC_EDGE_MASK_INIT;
constexpr uint8_t h_edge[12] = MC_EDGE_PACKED_INIT;

constexpr uint32_t h_case(uint32_t c)
{
    return (c & 1u) | (((c >> 4) & 1u) << 1) | (((c >> 5) & 1u) << 2) | (((c >> 1) & 1u) << 3) |
           (((c >> 2) & 1u) << 4) | (((c >> 6) & 1u) << 5) | (((c >> 7) & 1u) << 6) | (((c >> 3) & 1u) << 7);
}

constexpr PairTables make_pair_tables()
{
    PairTables t{};
    for (uint32_t code = 0; code < 256; ++code) {
        const uint32_t cs = h_case(code), em = h_mask[cs];
        int n = 0;
        for (uint32_t e = 0; e < 12; ++e)
            if ((em >> e) & 1u) {
                const uint32_t c0 = h_edge[e] & 7u, c1 = h_edge[e] >> 3, d = c0 ^ c1;
                t.edges[code][n++] = (uint8_t)(c0 | (c1 << 3) | ((d == 1u ? 0u : (d == 2u ? 1u : 2u)) << 6));
            }
        t.counts[code] = (uint8_t)(h_ntri[cs] | (n << 3));
        for (int c = 0; c < 3 * (int)h_ntri[cs]; ++c) {
            const uint32_t e = (uint32_t)(h_tri[cs] >> (4 * c)) & 15u;
            uint64_t rank = 0;
            for (uint32_t b = 0; b < e; ++b) rank += (em >> b) & 1u;
            t.tri_slots[code] |= rank << (4 * c);
            t.users[code][rank] |= (uint8_t)(1u << (c / 3));
        }
    }
    return t;
}


// Value types that are floats exactly take the FP32 certificate; the others
// keep their corner values as doubles and take the FP64 sequence.
template <typename T> constexpr bool kPairFast = sizeof(T) < 4;
template <> constexpr bool kPairFast<float> = true;
template <typename T> struct PairValue { using type = double; };
template <> struct PairValue<float> { using type = float; };
template <> struct PairValue<int8_t> { using type = float; };
template <> struct PairValue<uint8_t> { using type = float; };
template <> struct PairValue<int16_t> { using type = float; };
template <> struct PairValue<uint16_t> { using type = float; };

// A task's pairs as one index space: lane u holds unit u's (a warp scan of
// their numbers), and its row and first cell.
struct PairBlock {
    uint32_t inc, first;  // pairs up to and with this lane's unit; entry of pair p of it: list[first + p]
    uint32_t npairs;
    uint32_t uy, ux;
};

// Units u0 .. u0 + units - 1 (at most 32; those there are) of cell plane z.
__device__ __forceinline__ PairBlock pair_block(const StreamGroup& G, const PairList& pl, uint32_t z, uint32_t u0,
                                                uint32_t units, unsigned lane)
{
    PairBlock b;
    const uint32_t wpr = G.wpr, plane_units = (G.vol.ny - 1) * wpr;
    uint32_t np = 0;
    b.first = 0;
    const uint32_t un = u0 + lane;
    if (lane < units && un < plane_units) {
        const uint64_t pu = G.pair_base + (uint64_t)z * plane_units + un;
        np = pl.unit_pairs[pu];
        if (np) b.first = pl.unit_list[pu];
    }
    b.inc = np;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(FULL, b.inc, o);
        if (lane >= (unsigned)o) b.inc += t;
    }
    b.npairs = __shfl_sync(FULL, b.inc, 31);
    b.first -= b.inc - np;
    b.uy = un / wpr;
    b.ux = (un - b.uy * wpr) * G.seg_cells;
    return b;
}

// Pair p's list entry, row and its unit's first cell (lanes past the last
// pair: of some unit).
__device__ __forceinline__ uint32_t pair_entry(const PairBlock& b, uint32_t p, uint32_t& x, uint32_t& y)
{
    uint32_t own = 0;   // its unit: the first lane whose inclusive count exceeds p
#pragma unroll
    for (int s = 4; s >= 0; --s) {
        const uint32_t mid = own + (1u << s) - 1u;
        if (__shfl_sync(FULL, b.inc, mid) <= p) own = mid + 1;
    }
    own &= 31u;
    y = __shfl_sync(FULL, b.uy, own);
    x = __shfl_sync(FULL, b.ux, own);
    return __shfl_sync(FULL, b.first, own) + p;
}

// The 8 corner values of the cell at c, left in cv (corner: dx + 2 dy + 4 dz);
// its corner code, up(v) deciding a value.
template <typename T, typename V, typename Up>
__device__ __forceinline__ uint32_t pair_corners(const T* c, uint64_t pitch, uint64_t slice, V* cv, Up up)
{
    const T v0 = __ldg(c), v1 = __ldg(c + 1), v2 = __ldg(c + pitch), v3 = __ldg(c + pitch + 1);
    const T v4 = __ldg(c + slice), v5 = __ldg(c + slice + 1);
    const T v6 = __ldg(c + slice + pitch), v7 = __ldg(c + slice + pitch + 1);
    auto val = [&](T v) -> V {
        if constexpr (kPairFast<T>) return (float)v;
        else return to_double(v);
    };
    cv[0] = val(v0); cv[1] = val(v1); cv[2] = val(v2); cv[3] = val(v3);
    cv[4] = val(v4); cv[5] = val(v5); cv[6] = val(v6); cv[7] = val(v7);
    return (up(v0) ? 1u : 0u) | (up(v2) ? 2u : 0u) | (up(v4) ? 4u : 0u) | (up(v6) ? 8u : 0u) |
           (up(v1) ? 16u : 0u) | (up(v3) ? 32u : 0u) | (up(v5) ? 64u : 0u) | (up(v7) ? 128u : 0u);
}

}  // namespace

}  // namespace kvsmc
