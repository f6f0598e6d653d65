// mc_emit.cuh -- what the duplicated mode's emit kernels share: an
// isolevel's constants in shared memory, and one triangle's stores.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "mc_internal.h"

namespace kvsmc {

// An isolevel's constants as the emit loops read them (copied from the
// group's StreamIso entries when a warp starts on a group).
struct __align__(16) IsoConst {
    FastIso f;
    float mc[3], sc[3];   // min_coord, scale
    float* coords;
    float* normals;
    uint64_t cap_tris;
};

// An isolevel's interpolation constants in registers, read from its IsoConst
// with four 16-byte loads.
struct IsoRegs {
    FastIso f;
    float mc[3], sc[3];
};

static_assert(offsetof(IsoConst, f) == 0 && sizeof(FastIso) == 32 && offsetof(IsoConst, mc) == 32 &&
                  offsetof(IsoConst, sc) == 44 && sizeof(IsoConst) % 16 == 0,
              "load_iso reads IsoConst as four float4");

__device__ __forceinline__ IsoRegs load_iso(const IsoConst& c)
{
    const float4* p = reinterpret_cast<const float4*>(&c);
    const float4 a = p[0], b = p[1], m = p[2], n = p[3];
    IsoRegs r;
    r.f.ih = a.x;
    r.f.il = a.y;
    r.f.iso_err = a.z;
    r.f.f_thr = a.w;
    r.f.vmin_f = b.x;
    r.f.vmax_f = b.y;
    r.f.fast_ok = __float_as_int(b.z);
    r.f.lean_ok = __float_as_int(b.w);
    r.mc[0] = m.x;
    r.mc[1] = m.y;
    r.mc[2] = m.z;
    r.sc[0] = m.w;
    r.sc[1] = n.x;
    r.sc[2] = n.y;
    return r;
}

// Fill an isolevel's constants from its record; a request that does not fit
// its outputs is not written at all (totals null: up to its capacity).
__device__ __forceinline__ void fill_iso(IsoConst& c, const StreamIso& I, const uint64_t* totals, int index)
{
    c.f = I.f;
    for (int a = 0; a < 3; ++a) { c.mc[a] = I.ip.min_coord[a]; c.sc[a] = I.ip.scale[a]; }
    c.coords = totals && totals[index] > I.cap_tris ? nullptr : I.coords;
    c.normals = I.normals;
    c.cap_tris = I.cap_tris;
}

// One triangle's 9 coordinates and 3 normal components, as the 8-byte
// stores the addresses allow: a word whose address is 8-byte aligned pairs
// with the next one, the odd word out is stored alone (the first word when
// the array starts off an 8-byte boundary, else the last).  Seven stores
// instead of twelve; the values are chosen by selects, so lanes with either
// alignment run the same instructions.
__device__ __forceinline__ void store_triangle(float* oc, float* on, float3 A, float3 B, float3 C, float3 n)
{
    const bool ho = (reinterpret_cast<uintptr_t>(oc) & 4u) != 0;
    *(ho ? oc : oc + 8) = ho ? A.x : C.z;
    float2* p2 = reinterpret_cast<float2*>(ho ? oc + 1 : oc);
    p2[0] = make_float2(ho ? A.y : A.x, ho ? A.z : A.y);
    p2[1] = make_float2(ho ? B.x : A.z, ho ? B.y : B.x);
    p2[2] = make_float2(ho ? B.z : B.y, ho ? C.x : B.z);
    p2[3] = make_float2(ho ? C.y : C.x, ho ? C.z : C.y);
    const bool hn = (reinterpret_cast<uintptr_t>(on) & 4u) != 0;
    *(hn ? on : on + 2) = hn ? n.x : n.z;
    *reinterpret_cast<float2*>(hn ? on + 1 : on) = make_float2(hn ? n.y : n.x, hn ? n.z : n.y);
}

}  // namespace kvsmc
