// mc_slots.cuh -- small device helpers: the n-th set bit of a word, and the
// vertex slots that start from zero (mc_connect.cu, mc_snode.cu, cells.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace kvsmc {

// The position of m's bit number n (from 0).
__device__ __forceinline__ uint32_t nth_set_bit(uint32_t m, uint32_t n)
{
    uint32_t pos = 0;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        const uint32_t c = (uint32_t)__popc(m & ((1u << s) - 1u));
        if (n >= c) {
            n -= c;
            m >>= s;
            pos += s;
        }
    }
    return pos;
}

// A vertex of a node on the volume's faces may lack cells around its edge: its
// slots start from zero (the connection pass writes the ones there are).
__device__ __forceinline__ void clear_face_slots(uint2* slots, uint64_t id, uint32_t x, uint32_t y, uint32_t z,
                                                 uint32_t nx, uint32_t ny, uint32_t nz)
{
    if (x != 0 && y != 0 && z != 0 && x + 1 != nx && y + 1 != ny && z + 1 != nz) return;
    uint4* s = reinterpret_cast<uint4*>(slots + 4 * id);
    s[0] = make_uint4(0, 0, 0, 0);
    s[1] = make_uint4(0, 0, 0, 0);
}

}  // namespace kvsmc
