// gwn_device.cuh — device helpers shared by the winding-number kernels (k_gwn.cu: sums
// over every triangle; k_fwn.cu: clusters).
#pragma once
#include "gbsdf_device.cuh"
#include "gbsdf_internal.h"

namespace gbsdf {

__device__ __forceinline__ void voxel_coords(const Lattice& L, long long v, int& x, int& y, int& z) {
    long long dx = L.dims[0], dy = L.dims[1];
    x = (int)(v % dx);
    long long r = v / dx;
    y = (int)(r % dy);
    z = (int)(r / dy);
}

__device__ __forceinline__ size_t word_of(const Lattice& L, int x, int y, int z) {
    return ((size_t)z * L.dims[1] + y) * L.wx + (x >> 5);
}

__device__ __forceinline__ void consume(const Lattice& L, long long v, bool inside, int consumer,
                                        uint32_t* sbits, DevState* ds) {
    int x, y, z;
    voxel_coords(L, v, x, y, z);
    size_t w = word_of(L, x, y, z);
    uint32_t bit = 1u << (x & 31);
    if (consumer == kGwnFixup) {
        if (inside) atomicOr(&sbits[w], bit);
    } else {
        bool s = (sbits[w] & bit) != 0u;
        if (s != inside) {
            int m = atomicAdd(&ds->probe_m, 1);
            if (m < kVerifySamples) ds->sites[m] = v;
        }
    }
}

// Kahan step
__device__ __forceinline__ void kahan_add(float& s, float& c, float x) {
    float y = x - c;
    float t = s + y;
    c = (t - s) - y;
    s = t;
}

}  // namespace gbsdf
