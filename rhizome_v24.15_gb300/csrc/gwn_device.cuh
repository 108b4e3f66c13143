// gwn_device.cuh — device helpers shared by the winding-number kernels (k_gwn.cu: sums
// over every triangle; k_fwn.cu: clusters) and of the band splat (k_splat.cu).
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

// ---- the clusters (internal header, Fwn) as kernels take them ----
struct FwnView {
    const float4* cells[3];
    const float4* box[3];
    const float4* leaf;
    int n[3];
    long long T;
};

inline FwnView view_of(const Fwn& f, long long T) {
    FwnView v{};
    for (int l = 0; l < 3; ++l) {
        v.cells[l] = reinterpret_cast<const float4*>(f.cells[l]);
        v.box[l] = f.box[l];
        v.n[l] = (int)f.n[l];
    }
    v.leaf = f.leaf;
    v.T = T;
    return v;
}

// Squared distance of a point to a box (2 float4: least and greatest corner); a NaN gives 0.
__device__ __forceinline__ float box_dist_sq(const float4* __restrict__ box, const f3& p) {
    const float4 lo = __ldg(box), hi = __ldg(box + 1);
    const float dx = max3f(lo.x - p.x, p.x - hi.x, 0.0f), dy = max3f(lo.y - p.y, p.y - hi.y, 0.0f),
                dz = max3f(lo.z - p.z, p.z - hi.z, 0.0f);
    return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx));
}

__device__ __forceinline__ float leaf_dist_sq(const float4* __restrict__ leaf, const f3& p) {
    const float4 a = __ldg(leaf + 2), b = __ldg(leaf + 3);
    return ptd_sq(p, mk(a.x, a.y, a.z), mk(a.w, b.x, b.y), mk(b.z, b.w, __ldg(&leaf[4].x)));
}

// The k of the least d (non-negative, or +inf) over the warp, the least k of equal ones.
__device__ __forceinline__ int warp_argmin(float d, int k) {
    unsigned long long key = ((unsigned long long)__float_as_uint(d) << 32) | (unsigned)k;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) key = min(key, __shfl_xor_sync(0xffffffffu, key, o));
    return (int)(unsigned)key;
}

// Voxel of a brick by its place in Morton order (32 consecutive ones are a 4 x 4 x 2 box, so a
// warp's voxels agree on what is near): x | y << 3 | z << 6.
__device__ __forceinline__ int morton_voxel(int o) {
    const int x = (o & 1) | ((o >> 2) & 2) | ((o >> 4) & 4), y = ((o >> 1) & 1) | ((o >> 3) & 2) | ((o >> 5) & 4),
              z = ((o >> 2) & 1) | ((o >> 4) & 2) | ((o >> 6) & 4);
    return x | (y << 3) | (z << 6);
}

__device__ __forceinline__ float lattice_mid(int mn, int first, float half, float h) {
    return ((float)(mn + first) + half) * h;
}

}  // namespace gbsdf
