// mc_thermo.cuh -- threshold ("thermometer") masks of node values for up to
// kStreamMaxIso isolevels of one volume at once, and the cells' corner codes
// built from them.
//
// With the isolevels' thresholds sorted (t_0 <= t_1 <= ...), a value's mask
// has bit k set when v > t_k, so its set bits are 0 .. q-1.  A bucket index
// floor(kStreamBuckets * sat(v * bs + bo)) is monotone in v; a table of bytes
// holds the number of thresholds in lower buckets, and one compare with the
// next threshold finishes q: when that threshold lies in a higher bucket the
// compare is false by itself.  Only when some bucket holds two or more
// thresholds does a loop go on comparing.  NaN saturates to bucket 0 and is
// above no threshold, as in the reference's double compare.
// Byte and threshold lookups spread over few words (33 and 17), so 32 lanes'
// random ones meet in no more than two rows of a shared-memory bank; one table
// of 8-byte (mask, threshold) entries cost 4 to 5 wavefronts a lookup.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "mc_internal.h"

namespace kvsmc {

constexpr int kLut = kStreamBuckets + 1;   // bucket indices 0 .. kStreamBuckets
// Monotone (non-decreasing) bucket of a value in [0, kStreamBuckets]:
// floor(kStreamBuckets * sat(v * bs + bo)).  Thresholds and node values go
// through exactly this function, so a threshold in a lower bucket than v is
// below v, one in a higher bucket is not, and only a shared bucket needs an
// exact compare.  NaN saturates to 0 (the fma's .sat flushes NaN to +0).
__device__ __forceinline__ uint32_t bucket_index(float v, float bs, float bo)
{
    float u;
    asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(u) : "f"(v), "f"(bs), "f"(bo));
    // u * NB + 2^23 rounded down: 2^23 + floor(u * NB) exactly
    const float t = __fmaf_rd(u, (float)kStreamBuckets, 8388608.0f);
    return (uint32_t)__float_as_int(t) - 0x4B000000u;
}

// 8-bit values index the table by themselves (signed ones with the top bit
// flipped), and there is nothing to compare: three instructions a value for
// ten, 5% of a sweep's time on u8 data.  (16-bit values made comparable as
// 2^23 + value by one byte permute, without a conversion, took as long as
// converted ones.)
template <typename T> constexpr uint32_t kThermoFlip = 0;
template <> constexpr uint32_t kThermoFlip<int8_t> = 0x80808080u;
template <typename T> constexpr float kThermoBias = 0.0f;
template <> constexpr float kThermoBias<int8_t> = 128.0f;

// A group's threshold tables (shared memory).
template <typename T> struct ThermoTables {
    float thr[kStreamMaxIso + 1];   // sorted; +inf after the last one (no value is above it)
    uint32_t several;               // some bucket holds two or more thresholds
    // bucket -> number of thresholds in lower buckets; 8-bit: value -> number of thresholds below it
    uint8_t lut[sizeof(T) == 1 ? 256 : (kLut + 3) / 4 * 4];
};

// Fill W from the sorted thresholds, lane k holding t_k for k < niso: called by
// all 32 lanes of one warp (the caller synchronizes before W is read by others).
template <typename T>
__device__ __forceinline__ void thermo_build(ThermoTables<T>& W, float t, int niso, float bs, float bo, unsigned lane)
{
    if (lane <= (unsigned)niso) W.thr[lane] = lane < (unsigned)niso ? t : __int_as_float(0x7f800000);
    if constexpr (sizeof(T) == 1) {
        if (lane == 0) W.several = 0;
        for (unsigned v0 = 0; v0 < 256; v0 += 32) {
            uint32_t below = 0;
            for (int k = 0; k < niso; ++k)
                below += (float)(v0 + lane) - kThermoBias<T> > __shfl_sync(0xffffffffu, t, k) ? 1u : 0u;
            W.lut[v0 + lane] = (uint8_t)below;
        }
    } else {
        const uint32_t bucket = bucket_index(t, bs, bo);
        const uint32_t before = __shfl_up_sync(0xffffffffu, bucket, 1);
        const bool several = __any_sync(0xffffffffu, lane > 0 && lane < (unsigned)niso && before == bucket);
        if (lane == 0) W.several = several ? 1u : 0u;
        for (unsigned b0 = 0; b0 < (unsigned)kLut; b0 += 32) {
            uint32_t below = 0;
            for (int k = 0; k < niso; ++k) below += __shfl_sync(0xffffffffu, bucket, k) < b0 + lane ? 1u : 0u;
            if (b0 + lane < (unsigned)kLut) W.lut[b0 + lane] = (uint8_t)below;
        }
    }
    __syncwarp();
}

// The number of thresholds below v, a value of T's as a float.
template <typename T>
__device__ __forceinline__ uint32_t thermo_rank(const ThermoTables<T>& W, float bs, float bo, float v)
{
    if constexpr (sizeof(T) == 1) {
        return W.lut[(uint32_t)(v + kThermoBias<T>) & 255u];
    } else {
        uint32_t q = W.lut[bucket_index(v, bs, bo)];
        if (W.several) {
            while (v > W.thr[q]) ++q;   // (ends at the +inf after the last one)
        } else {
            q += v > W.thr[q] ? 1u : 0u;
        }
        return q;
    }
}

// The mask of one value: bit k set when v > t_k.
template <typename T>
__device__ __forceinline__ uint32_t thermo_mask(const ThermoTables<T>& W, float bs, float bo, float v)
{
    return (1u << thermo_rank(W, bs, bo, v)) - 1u;
}

// 8 consecutive values of a shared-memory row as floats (x0 multiple of 8).
__device__ __forceinline__ void load8(const float* row, uint32_t x0, float* o)
{
    const float4 a = *reinterpret_cast<const float4*>(row + x0);
    const float4 b = *reinterpret_cast<const float4*>(row + x0 + 4);
    o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
}
__device__ __forceinline__ void load8(const uint16_t* row, uint32_t x0, float* o)
{
    const uint4 a = *reinterpret_cast<const uint4*>(row + x0);
    const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { o[2 * i] = (float)(w[i] & 0xffffu); o[2 * i + 1] = (float)(w[i] >> 16); }
}
__device__ __forceinline__ void load8(const int16_t* row, uint32_t x0, float* o)
{
    const uint4 a = *reinterpret_cast<const uint4*>(row + x0);
    const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        o[2 * i] = (float)(int16_t)(w[i] & 0xffffu);
        o[2 * i + 1] = (float)(int16_t)(w[i] >> 16);
    }
}

// Thermometer masks of the N (8 or 9) nodes from x0 on of a staged row (x0 a
// multiple of 8): bit k set when the value is above isolevel k's threshold (v > t_k;
// thresholds sorted, so the set bits are 0 .. q-1), packed two nodes per word
// (node 2m in the low half of word m, node 2m+1 in the high half; word 4 holds
// node 8).
template <typename T, int N = 9>
__device__ __forceinline__ void row_masks(const T* row, uint32_t x0, const ThermoTables<T>& W, float bs, float bo,
                                          uint32_t* P)
{
    uint32_t q[9];
    if constexpr (sizeof(T) == 1) {
        uint2 w = *reinterpret_cast<const uint2*>(row + x0);
        w.x ^= kThermoFlip<T>;
        w.y ^= kThermoFlip<T>;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            q[i] = W.lut[(w.x >> (8 * i)) & 255u];
            q[4 + i] = W.lut[(w.y >> (8 * i)) & 255u];
        }
        if (N == 9) q[8] = W.lut[(uint8_t)row[x0 + 8] ^ (kThermoFlip<T> & 0xffu)];
    } else {
        float v[9];
        load8(row, x0, v);
        if (N == 9) v[8] = (float)row[x0 + 8];
#pragma unroll
        for (int i = 0; i < N; ++i) q[i] = W.lut[bucket_index(v[i], bs, bo)];
#pragma unroll
        for (int i = 0; i < N; ++i) q[i] += v[i] > W.thr[q[i]] ? 1u : 0u;
        if (W.several) {
#pragma unroll
            for (int i = 0; i < N; ++i)
                while (v[i] > W.thr[q[i]]) ++q[i];   // (ends at the +inf after the last one)
        }
    }
    // (1 << a) - 1 in the low and (1 << b) - 1 in the high half (a, b <= 16: the
    // sum is right modulo 2^32)
#pragma unroll
    for (int m = 0; m < 4; ++m)
        P[m] = (1u << q[2 * m]) + ((1u << q[2 * m + 1]) << 16) - 0x10001u;
    if (N == 9) P[4] = (1u << q[8]) - 1u;
}

// The row word of cell i (0..7): node i in the low half, node i+1 in the high half.
__device__ __forceinline__ uint32_t cell_word(const uint32_t* P, int i)
{
    return (i & 1) ? __funnelshift_r(P[i >> 1], P[(i >> 1) + 1], 16) : P[i >> 1];
}

// Corner code of a cell for isolevel k from its four row words (plane z rows
// y, y+1 = a0, a1; plane z+1 = b0, b1): bit r = row r's node i above, bit
// 4 + r = row r's node i+1 above.
__device__ __forceinline__ uint32_t case_code(uint32_t a0, uint32_t a1, uint32_t b0, uint32_t b1, uint32_t k)
{
    const uint32_t m0 = (a0 >> k) & 0x10001u, m1 = (a1 >> k) & 0x10001u;
    const uint32_t m2 = (b0 >> k) & 0x10001u, m3 = (b1 >> k) & 0x10001u;
    const uint32_t x = m0 | (m1 << 1) | (m2 << 2) | (m3 << 3);
    return (x & 0xfu) | ((x >> 12) & 0xf0u);
}

// The reference's case number of a corner code: bit c = corner c above, with
// corners (x,y,z) 0:(0,0,0) 1:(1,0,0) 2:(1,1,0) 3:(0,1,0) 4:(0,0,1) 5:(1,0,1)
// 6:(1,1,1) 7:(0,1,1) (MarchingCubes.cpp:187-194).
__device__ __forceinline__ uint32_t code_to_case(uint32_t c)
{
    return (c & 1u) | (((c >> 4) & 1u) << 1) | (((c >> 5) & 1u) << 2) | (((c >> 1) & 1u) << 3) |
           (((c >> 2) & 1u) << 4) | (((c >> 6) & 1u) << 5) | (((c >> 7) & 1u) << 6) | (((c >> 3) & 1u) << 7);
}

}  // namespace kvsmc
