// k_fwn.cu — the triangle clusters: build, exact winding decisions and nearest distances.
//
// The clusters are consecutive runs of the triangles in Hilbert order of their centroids
// (internal header), so they follow the mesh's own density: on a grid of cubes a cluster of
// the 512^3 vessel tree held about 25 triangles within 7 voxels, and a voxel near the surface
// summed some thousand triangles one by one. Three levels (8, 128 and 2048 triangles) and the
// triangles themselves as the last one (a far triangle by its dipole, about a quarter of the
// solid angle's work) leave the few triangles next to a voxel to the exact formula.
//
// A voxel-by-voxel query walks the levels for each voxel. Where many voxels are asked for (the
// legacy path's every voxel, patch boxes, proposed bricks; signs.h has the line) one CTA
// takes a block of BB^3 bricks instead and looks at the clusters in steps:
//   * a cluster far from the block enters a polynomial about the block's centre;
//   * the others are looked at again for each brick with marked voxels: far ones enter a
//     polynomial about the brick's centre;
//   * what is left, the clusters near the brick, is taken voxel by voxel.
// Every step keeps the bound of what it leaves out, and a voxel is decided only when |w|
// clears 0.5 by more than all of it (and the rounding slack); the others are walked one by one
// with wider near ranges and at last summed triangle by triangle, so the decisions are those of
// the per-triangle sum.
//
// Measured (voxels decided, before -> after, with k_caps.cu's pass in front): legacy path,
// 181 x 141 x 171 mug, 4.4M voxels: 102 -> 0.4 ms; 512^3 vessel tree, 5,161 proposed bricks and
// 0.52M fixup voxels: 160 -> 12 ms; 640^3 blob with holes, 3.96M fixup voxels: 307 -> 19 ms.
#include <algorithm>

#include "gwn_device.cuh"

namespace gbsdf {

namespace {

// A cluster is far when d > beta r: in a voxel's own sum, in a block's second pass (and
// a walk's), in a walk's third, and (d less the radius of what is queried) for a block's and a brick's polynomial.
constexpr float kFwnBeta = 4.0f, kFwnBetaFine = 8.0f, kFwnBetaRefine = 32.0f, kFwnBetaBlock = 6.0f,
                kFwnBetaBrick = 5.0f;
constexpr float kCapBound = 0.05f;  // a cap cluster of at most this solid angle enters by its bound alone
constexpr float kFwnSlackRel = 1e-5f;   // rounding slack per unit of summed |terms|
constexpr float kFwnSlackAbs = 1e-5f;   // rounding slack in w
constexpr int kQueryThreads = 256;

// ---- Hilbert order --------------------------------------------------------------------
constexpr int kKeyBits = 9;             // per axis: 512 cells over the lattice's longest side
constexpr int kDigitBits = 9, kDigits = 1 << kDigitBits, kPasses = 3 * kKeyBits / kDigitBits;
constexpr int kSortThreads = 256, kSortItems = 8, kSortTile = kSortThreads * kSortItems;

// Hilbert index of a cell (J. Skilling, "Programming the Hilbert curve", AIP Conf. Proc. 707,
// 2004: axes to transpose, then the bits interleaved).
__device__ __forceinline__ unsigned hilbert_key(unsigned x, unsigned y, unsigned z) {
    unsigned X[3] = {x, y, z};
    for (unsigned q = 1u << (kKeyBits - 1); q > 1u; q >>= 1) {
        const unsigned p = q - 1u;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            if (X[i] & q) {
                X[0] ^= p;
            } else {
                const unsigned t = (X[0] ^ X[i]) & p;
                X[0] ^= t;
                X[i] ^= t;
            }
        }
    }
    X[1] ^= X[0];
    X[2] ^= X[1];
    unsigned t = 0u;
    for (unsigned q = 1u << (kKeyBits - 1); q > 1u; q >>= 1)
        if (X[2] & q) t ^= q - 1u;
    unsigned key = 0u;
#pragma unroll
    for (int b = kKeyBits - 1; b >= 0; --b)
#pragma unroll
        for (int i = 0; i < 3; ++i) key = (key << 1) | (((X[i] ^ t) >> b) & 1u);
    return key;
}

__global__ void fwn_key_kernel(const float* __restrict__ t9, long long T, Lattice L, float scale,
                               unsigned* __restrict__ key, unsigned* __restrict__ idx) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T) return;
    const float* v = t9 + 9 * t;
    const float inv = 1.0f / L.h;
    unsigned c[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float g = ((v[k] + v[3 + k] + v[6 + k]) * (1.0f / 3.0f) * inv - (float)L.mn[k]) * scale;
        c[k] = (unsigned)fminf(fmaxf(g, 0.0f), (float)((1 << kKeyBits) - 1));  // a NaN goes to 0
    }
    key[t] = hilbert_key(c[0], c[1], c[2]);
    idx[t] = (unsigned)t;
}

// One pass of a stable least-significant-digit radix sort: tile histograms (digit-major), their
// scan, and the scatter (ranks within a warp by digit matching, warps and tiles in order).
__global__ void __launch_bounds__(kSortThreads) sort_hist_kernel(const unsigned* __restrict__ key, long long T,
                                                                 int shift, unsigned* __restrict__ hist,
                                                                 unsigned tiles) {
    __shared__ unsigned s[kDigits];
    for (int k = threadIdx.x; k < kDigits; k += kSortThreads) s[k] = 0u;
    __syncthreads();
    const long long base = (long long)blockIdx.x * kSortTile;
#pragma unroll
    for (int i = 0; i < kSortItems; ++i) {
        const long long k = base + i * kSortThreads + threadIdx.x;
        if (k < T) atomicAdd(&s[(key[k] >> shift) & (kDigits - 1)], 1u);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < kDigits; k += kSortThreads) hist[(size_t)k * tiles + blockIdx.x] = s[k];
}

// Exclusive scan of n counters by one CTA (n = 512 per 2048 triangles: 45,000 for 180,000
// triangles, six steps).
__global__ void __launch_bounds__(1024) sort_scan_kernel(const unsigned* __restrict__ in, unsigned* __restrict__ out,
                                                         long long n) {
    __shared__ unsigned wsum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned carry = 0u;
    for (long long base = 0; base < n; base += 8192) {
        const long long k0 = base + 8 * threadIdx.x;
        unsigned v[8], run = 0u;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const unsigned x = (k0 + i < n) ? in[k0 + i] : 0u;
            v[i] = run;
            run += x;
        }
        unsigned inc = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) wsum[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            unsigned x = wsum[lane], y = x;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned t = __shfl_up_sync(0xffffffffu, y, o);
                if (lane >= o) y += t;
            }
            wsum[lane] = y;
        }
        __syncthreads();
        const unsigned before = carry + (warp ? wsum[warp - 1] : 0u) + inc - run;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (k0 + i < n) out[k0 + i] = before + v[i];
        carry += wsum[31];
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kSortThreads) sort_scatter_kernel(const unsigned* __restrict__ key,
                                                                    const unsigned* __restrict__ idx, long long T,
                                                                    int shift, const unsigned* __restrict__ offs,
                                                                    unsigned tiles, unsigned* __restrict__ key_out,
                                                                    unsigned* __restrict__ idx_out) {
    constexpr int kWarps = kSortThreads / 32;
    __shared__ unsigned short cnt[kWarps][kDigits];  // a warp's 256 items at most
    for (int k = threadIdx.x; k < kWarps * kDigits; k += kSortThreads) (&cnt[0][0])[k] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long base = (long long)blockIdx.x * kSortTile + warp * (kSortTile / kWarps);
    unsigned kk[kSortItems], rank[kSortItems];
#pragma unroll
    for (int i = 0; i < kSortItems; ++i) {
        const long long k = base + i * 32 + lane;
        const bool on = k < T;
        kk[i] = on ? key[k] : 0u;
        const unsigned d = on ? (kk[i] >> shift) & (kDigits - 1) : (unsigned)kDigits;
        const unsigned same = __match_any_sync(0xffffffffu, d);
        const unsigned before = on ? cnt[warp][d] : 0u;
        rank[i] = before + __popc(same & ((1u << lane) - 1u));
        __syncwarp();
        if (on && lane == 31 - __clz(same)) cnt[warp][d] = (unsigned short)(before + __popc(same));
        __syncwarp();
    }
    __syncthreads();
    for (int d = threadIdx.x; d < kDigits; d += kSortThreads) {  // exclusive over the warps
        unsigned run = 0u;
        for (int w = 0; w < kWarps; ++w) {
            const unsigned c = cnt[w][d];
            cnt[w][d] = (unsigned short)run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kSortItems; ++i) {
        const long long k = base + i * 32 + lane;
        if (k >= T) continue;
        const unsigned d = (kk[i] >> shift) & (kDigits - 1);
        const unsigned pos = offs[(size_t)d * tiles + blockIdx.x] + cnt[warp][d] + rank[i];
        key_out[pos] = kk[i];
        idx_out[pos] = idx[k];
    }
}

// ---- clusters -------------------------------------------------------------------------
__device__ __forceinline__ double group_sum(double x, int width) {
    for (int o = width >> 1; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

__device__ __forceinline__ void group_box(float (&lo)[3], float (&hi)[3], int width) {
    for (int o = width >> 1; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
        }
}

// One lane per triangle in Hilbert order, eight lanes per cluster: the triangle's record (in
// line, so that a query reads it without an index) and the cluster's FP64 statistics. Bound by
// the FP64 pipes (about 400 instructions a warp at 16 cycles each); in CTAs of 64 so that small
// meshes spread over all SMs: 24,000 triangles, 33 us in CTAs of 256, 27 now.
constexpr int kStatThreads = 64;
__global__ void __launch_bounds__(kStatThreads) fwn_leaf_kernel(const float* __restrict__ t9, long long T,
                                                       const unsigned* __restrict__ idx, float4* __restrict__ leaf,
                                                       FwnCell* __restrict__ cells, float4* __restrict__ box) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool on = t < T;
    float v[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (on) {
        const float* p = t9 + 9ull * idx[t];
#pragma unroll
        for (int k = 0; k < 9; ++k) v[k] = p[k];
    }
    const double e1[3] = {(double)v[3] - v[0], (double)v[4] - v[1], (double)v[5] - v[2]};
    const double e2[3] = {(double)v[6] - v[0], (double)v[7] - v[1], (double)v[8] - v[2]};
    const double D[3] = {0.5 * (e1[1] * e2[2] - e1[2] * e2[1]), 0.5 * (e1[2] * e2[0] - e1[0] * e2[2]),
                         0.5 * (e1[0] * e2[1] - e1[1] * e2[0])};
    const double a = sqrt(D[0] * D[0] + D[1] * D[1] + D[2] * D[2]);
    double g[3], l2 = 0.0;
    float fg[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        g[k] = ((double)v[k] + v[3 + k] + v[6 + k]) / 3.0;
        fg[k] = (float)g[k];
        const double e3 = e2[k] - e1[k];
        l2 += e1[k] * e1[k] + e2[k] * e2[k] + e3 * e3;
    }
    double rt2 = 0.0, off2 = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) off2 += (g[k] - fg[k]) * (g[k] - fg[k]);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const double dx = (double)v[3 * q] - fg[0], dy = (double)v[3 * q + 1] - fg[1], dz = (double)v[3 * q + 2] - fg[2];
        rt2 = fmax(rt2, dx * dx + dy * dy + dz * dz);
    }
    // the record's centroid is rounded to FP32: the second moment is the one about it, the first
    // one enters the bound where the dipole is used (leaf_term)
    const double qt = a * (l2 / 36.0 + off2);
    if (on) {
        float4* o = leaf + 5 * t;
        o[0] = make_float4(fg[0], fg[1], fg[2], (float)(sqrt(rt2) * (1.0 + 1e-6)) + 1e-30f);
        o[1] = make_float4((float)D[0], (float)D[1], (float)D[2], (float)(qt * (1.0 + 1e-5)));
        o[2] = make_float4(v[0], v[1], v[2], v[3]);
        o[3] = make_float4(v[4], v[5], v[6], v[7]);
        o[4] = make_float4(v[8], (float)(a * a), 0.0f, 0.0f);
    }
    float lo[3], hi[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        lo[k] = on ? fminf(v[k], fminf(v[3 + k], v[6 + k])) : __int_as_float(0x7f800000);
        hi[k] = on ? fmaxf(v[k], fmaxf(v[3 + k], v[6 + k])) : __int_as_float(0xff800000);
    }
    group_box(lo, hi, kFwnLeaf);
    if (on && (t % kFwnLeaf) == 0) {
        box[2 * (t / kFwnLeaf)] = make_float4(lo[0], lo[1], lo[2], 0.0f);
        box[2 * (t / kFwnLeaf) + 1] = make_float4(hi[0], hi[1], hi[2], 0.0f);
    }
    const double w1 = on ? 1.0 : 0.0;
    const double n = group_sum(w1, kFwnLeaf), A = group_sum(on ? a : 0.0, kFwnLeaf);
    double S[3], fc[3];
    float c[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        S[k] = group_sum(on ? D[k] : 0.0, kFwnLeaf);
        const double G = group_sum(on ? a * g[k] : 0.0, kFwnLeaf), mean = group_sum(on ? g[k] : 0.0, kFwnLeaf);
        c[k] = (float)((A > 0.0) ? G / A : mean / fmax(n, 1.0));
        fc[k] = c[k];
    }
    double M[9], d2 = 0.0, r2 = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        d2 += (g[i] - fc[i]) * (g[i] - fc[i]);
#pragma unroll
        for (int j = 0; j < 3; ++j) M[3 * i + j] = group_sum(on ? D[i] * (g[j] - fc[j]) : 0.0, kFwnLeaf);
    }
    const double Q = group_sum(on ? a * (l2 / 36.0 + d2) : 0.0, kFwnLeaf);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const double dx = (double)v[3 * q] - fc[0], dy = (double)v[3 * q + 1] - fc[1], dz = (double)v[3 * q + 2] - fc[2];
        r2 = fmax(r2, on ? dx * dx + dy * dy + dz * dz : 0.0);
        if (on && !(dx * dx + dy * dy + dz * dz >= 0.0)) r2 = dx + dy + dz;  // a NaN stays one
    }
    for (int o = kFwnLeaf >> 1; o > 0; o >>= 1) {
        const double u = __shfl_xor_sync(0xffffffffu, r2, o);
        r2 = (r2 >= u || r2 != r2) ? r2 : u;
    }
    if (on && (t % kFwnLeaf) == 0) {
        FwnCell C;
        C.cx = c[0];
        C.cy = c[1];
        C.cz = c[2];
        C.r = (float)(sqrt(r2) * (1.0 + 1e-6)) + 1e-30f;
        C.ax = (float)S[0];
        C.ay = (float)S[1];
        C.az = (float)S[2];
        C.area = (float)(A * (1.0 + 1e-6));
        for (int k = 0; k < 9; ++k) C.m[k] = (float)M[k];
        C.q = (float)(Q * (1.0 + 1e-5));
        C.pad[0] = C.pad[1] = 0.0f;
        cells[t / kFwnLeaf] = C;
    }
}

// One lane per cluster of the level below, sixteen per cluster: aggregated moments in FP64 --
// A = sum A_c, D = sum D_c, C = sum A_c c_c / A, M = sum (M_c + D_c (c_c - C)^T) and Q = sum
// (Q_c + A_c |c_c - C|^2), the triangles' own moments about C, and r = max (|c_c - C| + r_c).
// One warp a CTA, for the same reason: both levels of 24,000 triangles 34 us, 21 now.
__global__ void __launch_bounds__(32) fwn_level_kernel(const FwnCell* __restrict__ below,
                                                        const float4* __restrict__ box_below, long long nb,
                                                        FwnCell* __restrict__ cells, float4* __restrict__ box) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool on = k < nb;
    const float inf = __int_as_float(0x7f800000);
    const float4 b0 = on ? box_below[2 * k] : make_float4(inf, inf, inf, 0.0f),
                 b1 = on ? box_below[2 * k + 1] : make_float4(-inf, -inf, -inf, 0.0f);
    float lo[3] = {b0.x, b0.y, b0.z}, hi[3] = {b1.x, b1.y, b1.z};
    group_box(lo, hi, kFwnFan);
    if (on && (k % kFwnFan) == 0) {
        box[2 * (k / kFwnFan)] = make_float4(lo[0], lo[1], lo[2], 0.0f);
        box[2 * (k / kFwnFan) + 1] = make_float4(hi[0], hi[1], hi[2], 0.0f);
    }
    FwnCell c{};
    if (on) c = below[k];
    const double a = c.area, cc[3] = {c.cx, c.cy, c.cz}, D[3] = {c.ax, c.ay, c.az};
    const double n = group_sum(on ? 1.0 : 0.0, kFwnFan), A = group_sum(a, kFwnFan);
    double S[3], s[3], d2 = 0.0;
    float fc[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        S[i] = group_sum(D[i], kFwnFan);
        const double G = group_sum(a * cc[i], kFwnFan), mean = group_sum(cc[i], kFwnFan);
        fc[i] = (float)((A > 0.0) ? G / A : mean / fmax(n, 1.0));
        s[i] = cc[i] - fc[i];
        d2 += s[i] * s[i];
    }
    double M[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) M[3 * i + j] = group_sum(on ? c.m[3 * i + j] + D[i] * s[j] : 0.0, kFwnFan);
    const double Q = group_sum(on ? c.q + a * d2 : 0.0, kFwnFan);
    double R = on ? sqrt(d2) + c.r : 0.0;
    for (int o = kFwnFan >> 1; o > 0; o >>= 1) {
        const double u = __shfl_xor_sync(0xffffffffu, R, o);
        R = (R >= u || R != R) ? R : u;  // a NaN stays one
    }
    if (on && (k % kFwnFan) == 0) {
        FwnCell C;
        C.cx = fc[0];
        C.cy = fc[1];
        C.cz = fc[2];
        C.r = (float)(R * (1.0 + 1e-6)) + 1e-30f;
        C.ax = (float)S[0];
        C.ay = (float)S[1];
        C.az = (float)S[2];
        C.area = (float)(A * (1.0 + 1e-6));
        for (int i = 0; i < 9; ++i) C.m[i] = (float)M[i];
        C.q = (float)(Q * (1.0 + 1e-5));
        C.pad[0] = C.pad[1] = 0.0f;
        cells[k / kFwnFan] = C;
    }
}

// ---- terms ----------------------------------------------------------------------------
struct Sum {
    float s = 0.0f, c = 0.0f, err = 0.0f, mag = 0.0f;
    bool near = false;
};

// A cluster's term by its moments, with its bound, when d > beta r; false when it is near.
__device__ __forceinline__ bool cell_far(const float4* __restrict__ cell, const f3& p, float beta, Sum& a) {
    const float4 c0 = __ldg(cell);
    const float dx = c0.x - p.x, dy = c0.y - p.y, dz = c0.z - p.z;
    const float d2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx));
    const float ir = rsqrtf(d2), d = d2 * ir;
    if (!(d > beta * c0.w)) return false;
    const float4 c1 = __ldg(cell + 1), c2 = __ldg(cell + 2), c3 = __ldg(cell + 3), c4 = __ldg(cell + 4);
    const float ir2 = ir * ir, ir3 = ir * ir2;
    const float dip = __fmaf_rn(c1.z, dz, __fmaf_rn(c1.y, dy, c1.x * dx)) * ir3;
    const float my0 = __fmaf_rn(c2.z, dz, __fmaf_rn(c2.y, dy, c2.x * dx));
    const float my1 = __fmaf_rn(c3.y, dz, __fmaf_rn(c3.x, dy, c2.w * dx));
    const float my2 = __fmaf_rn(c4.x, dz, __fmaf_rn(c3.w, dy, c3.z * dx));
    const float yMy = __fmaf_rn(dz, my2, __fmaf_rn(dy, my1, dx * my0));
    const float quad = __fmaf_rn(-3.0f * yMy, ir2, c2.x + c3.x + c4.x) * ir3;
    kahan_add(a.s, a.c, dip + quad);
    a.mag += fabsf(dip) + fabsf(quad);
    const float e = (d - c0.w) * 0.9999f, e2 = e * e;
    a.err += __fdividef(3.0f * c4.y, e2 * e2);
    return true;
}

// Solid angle of a triangle in FP32, or in FP64 where FP32 cannot be trusted. CAPS: a point on the triangle, to
// within FP64's rounding of its side, sets `near`.
template <bool CAPS>
__device__ __forceinline__ float tri_angle(const f3& p, const f3& v0, const f3& v1, const f3& v2, bool& near) {
    const float ax = v0.x - p.x, ay = v0.y - p.y, az = v0.z - p.z;
    const float bx = v1.x - p.x, by = v1.y - p.y, bz = v1.z - p.z;
    const float cx = v2.x - p.x, cy = v2.y - p.y, cz = v2.z - p.z;
    const float la = sqrtf(__fmaf_rn(az, az, __fmaf_rn(ay, ay, ax * ax)));
    const float lb = sqrtf(__fmaf_rn(bz, bz, __fmaf_rn(by, by, bx * bx)));
    const float lc = sqrtf(__fmaf_rn(cz, cz, __fmaf_rn(cy, cy, cx * cx)));
    const float det = __fmaf_rn(az, __fmaf_rn(bx, cy, -(by * cx)),
                                __fmaf_rn(-ay, __fmaf_rn(bx, cz, -(bz * cx)), ax * __fmaf_rn(by, cz, -(bz * cy))));
    const float ab = __fmaf_rn(az, bz, __fmaf_rn(ay, by, ax * bx));
    const float bc = __fmaf_rn(bz, cz, __fmaf_rn(by, cy, bx * cx));
    const float ca = __fmaf_rn(cz, az, __fmaf_rn(cy, ay, cx * ax));
    const float labc = la * lb * lc;
    const float denom = __fmaf_rn(ca, lb, __fmaf_rn(bc, la, __fmaf_rn(ab, lc, labc)));
    if (angle_uncertain(det, denom, labc) || la <= 1e-6f || lb <= 1e-6f || lc <= 1e-6f) {
        double det64, denom64, labc64;
        const float angle = (float)solid_angle_f64(p, v0, v1, v2, det64, denom64, labc64);
        if (CAPS) near |= fabs(det64) <= 1e-9 * labc64 && denom64 <= 1e-9 * labc64;
        return angle;
    }
    return 2.0f * atan2f(det, denom);
}

// A triangle's term: by its dipole when d > beta r, else the exact solid angle.
template <bool CAPS = false>
__device__ __forceinline__ void leaf_term(const float4* __restrict__ leaf, const f3& p, float beta, Sum& a) {
    const float4 c0 = __ldg(leaf);
    const float dx = c0.x - p.x, dy = c0.y - p.y, dz = c0.z - p.z;
    const float d2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx));
    const float ir = rsqrtf(d2), d = d2 * ir;
    float term;
    if (d > beta * c0.w) {
        const float4 c1 = __ldg(leaf + 1);
        const float ir3 = ir * ir * ir;
        term = __fmaf_rn(c1.z, dz, __fmaf_rn(c1.y, dy, c1.x * dx)) * ir3;
        const float e = (d - c0.w) * 0.9999f, e2 = e * e;
        // the record's centroid is off by up to 2^-24 of itself, and a first moment s from it adds at
        // most 2 |D| |s| / d^3
        const float g = fabsf(c0.x) + fabsf(c0.y) + fabsf(c0.z), D = fabsf(c1.x) + fabsf(c1.y) + fabsf(c1.z);
        a.err += __fmaf_rn(1.2e-7f * g, D * ir3, __fdividef(3.0f * c1.w, e2 * e2));
    } else {
        const float4 u = __ldg(leaf + 2), v = __ldg(leaf + 3);
        const float w = __ldg(&leaf[4].x);
        term = tri_angle<CAPS>(p, mk(u.x, u.y, u.z), mk(u.w, v.x, v.y), mk(v.z, v.w, w), a.near);
    }
    kahan_add(a.s, a.c, term);
    a.mag += fabsf(term);
}

// ---- queries of listed voxels ---------------------------------------------------------
// One warp per listed voxel down the levels: the lanes take 32 clusters, the near ones' (by
// ballot, in order) children next, two clusters' sixteen or four clusters' eight triangles at a
// time. What a walk leaves undecided is walked again with a wider near range (smaller truncation
// bounds, more exact terms): beta0, 8, 32; then the voxel is handed to the sum over every
// triangle. The blocks' leftovers start at 32: most come from 8 undecided (512^3 vessel tree, its
// two queries 3.6 + 3.1 ms from 8, 3.1 + 3.0 from 16, 2.9 + 2.7 so; 640^3 blob 5.1, 6.1, 4.2).
// Latency-bound: a walk is a chain of some tens of loads and ballots, and one of beta 32 some
// thousand triangles long (29% of the issue slots).
__global__ void __launch_bounds__(kQueryThreads) fwn_query_kernel(
    FwnView f, Lattice L, const long long* __restrict__ list, const unsigned long long* __restrict__ list_n,
    long long cap, int consumer, int only_if, uint32_t* __restrict__ sbits, const float* __restrict__ dist, int dist_sq,
    float surf_tol_vox, DevState* ds, long long* __restrict__ fb, long long fb_cap, float beta0) {
    if (only_if && !ds->patching) return;
    const float tau = surf_tol_vox * L.h;
    const long long n = min((long long)*list_n, cap);
    const int lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    unsigned long long certified = 0, handed = 0;
    for (long long j = warp; j < n; j += nwarps) {
        const long long v = list[j];
        if (v < 0) continue;
        int x, y, z;
        voxel_coords(L, v, x, y, z);
        const f3 p = lattice_point(L.mn[0], L.mn[1], L.mn[2], x, y, z, L.h);
        if (dist) {
            const float d = dist[v];
            if (dist_sq ? (d <= tau * tau) : (d <= tau)) {  // on the surface: inside
                if (lane == 0) consume(L, v, true, consumer, sbits, ds);
                continue;
            }
        }
        auto lowest = [](unsigned& m) {  // takes the lowest set bit's place, -1 when none is left
            const int b = __ffs(m) - 1;
            m &= m - 1u;
            return b;
        };
        bool done = false;
        for (float beta = beta0; !done && beta <= kFwnBetaRefine; beta = beta < kFwnBetaFine ? kFwnBetaFine : 4.0f * beta) {
            Sum a;
            for (int base = 0; base < f.n[2]; base += 32) {
                const int k2 = base + lane;
                unsigned m2 =
                    __ballot_sync(0xffffffffu, k2 < f.n[2] && !cell_far(f.cells[2] + 5 * (size_t)k2, p, beta, a));
                while (m2) {
                    const int a2 = lowest(m2), b2 = lowest(m2), s2 = (lane < 16) ? a2 : b2;
                    const int k1 = (base + s2) * kFwnFan + (lane & 15);
                    unsigned m1 = __ballot_sync(0xffffffffu, s2 >= 0 && k1 < f.n[1] &&
                                                                 !cell_far(f.cells[1] + 5 * (size_t)k1, p, beta, a));
                    while (m1) {
                        const int a1 = lowest(m1), b1 = lowest(m1), s1 = (lane < 16) ? a1 : b1;
                        const int p1 = __shfl_sync(0xffffffffu, k1, s1 & 31);
                        const int k0 = p1 * kFwnFan + (lane & 15);
                        unsigned m0 = __ballot_sync(0xffffffffu, s1 >= 0 && k0 < f.n[0] &&
                                                                     !cell_far(f.cells[0] + 5 * (size_t)k0, p, beta, a));
                        while (m0) {
                            const int a0 = lowest(m0), b0 = lowest(m0), c0 = lowest(m0), d0 = lowest(m0);
                            const int s0 = (lane < 8) ? a0 : (lane < 16) ? b0 : (lane < 24) ? c0 : d0;
                            const long long t =
                                (long long)__shfl_sync(0xffffffffu, k0, s0 & 31) * kFwnLeaf + (lane & 7);
                            if (s0 >= 0 && t < f.T) leaf_term(f.leaf + 5 * t, p, beta, a);
                            __syncwarp();
                        }
                    }
                }
            }
            float tot = a.s - a.c, err = a.err, mag = a.mag;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                tot += __shfl_xor_sync(0xffffffffu, tot, o);
                err += __shfl_xor_sync(0xffffffffu, err, o);
                mag += __shfl_xor_sync(0xffffffffu, mag, o);
            }
            const float w = fabsf(tot * kInv4Pi);
            const float e = (err * 1.0001f + kFwnSlackRel * mag) * kInv4Pi + kFwnSlackAbs;
            const bool in = w - e >= 0.5f;
            done = in || w + e < 0.5f;
            if (done && lane == 0) {
                consume(L, v, in, consumer, sbits, ds);
                ++certified;
            }
        }
        if (!done && lane == 0) {
            const unsigned long long k = atomicAdd(&ds->fwn_sum, 1ull);
            if ((long long)k < fb_cap) fb[k] = v;
            ++handed;
        }
    }
    if (lane == 0) {
        if (certified) atomicAdd(&ds->fwn_certified, certified);
        if (handed) atomicAdd(&ds->fwn_fallback_total, handed);
    }
}

// ---- queries of whole blocks ----------------------------------------------------------
constexpr int kBqThreads = 256;
constexpr int kBqWarps = kBqThreads / 32;
constexpr int kBqCap2 = 512;     // near top-level clusters of a block
constexpr int kBqCap1 = 1024;    // near middle clusters of a block (and of a brick)
constexpr int kBqCap0 = 2048;    // near clusters of a brick
constexpr float kBqRatio = 0.25f; // largest brick radius / distance of a far cluster

// A block's pending flags: BB = 2 (16^3 voxels) on large lattices, BB = 1 (8^3) where 16^3
// blocks would be too few to fill the chip, four an SM. Blocks of 16^3 / 8^3, every voxel, ms:
// watertight mug of 23k triangles, by its crossings, 120^3 (512 blocks) 0.39 / 0.29, 144^3 (729)
// 0.41 / 0.33, 160^3 (1,000) 0.34 / 0.36, 256^3 0.89 / 1.00; by the clusters alone 120^3 26 / 12,
// 144^3 31 / 19, 256^3 131 / 116.
__host__ __device__ inline long long block_count(const Lattice& L, int BB) {
    return (long long)((L.nb[0] + BB - 1) / BB) * ((L.nb[1] + BB - 1) / BB) * ((L.nb[2] + BB - 1) / BB);
}
inline int block_bricks(const Lattice& L) { return block_count(L, 2) >= 152 * 4 ? 2 : 1; }

// One warp per word column of a block row: the words (32 voxels along x) of a block's (8 BB)^2
// rows, or-ed; each 8 BB bits of the result are one block's flag.
template <int BB>
__global__ void __launch_bounds__(256) list_blocks_kernel(const uint32_t* __restrict__ U, Lattice L,
                                                          long long* __restrict__ list, long long cap, DevState* ds,
                                                          int only_if) {
    if (only_if && !ds->patching) return;
    constexpr int E = 8 * BB, PW = 32 / E;  // block edge, blocks per word
    const int gx = (L.nb[0] + BB - 1) / BB, gy = (L.nb[1] + BB - 1) / BB, gz = (L.nb[2] + BB - 1) / BB;
    const long long cols = (long long)L.wx * gy * gz;
    const int lane = threadIdx.x & 31;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long c = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < cols; c += nw) {
        const int xw = (int)(c % L.wx), by = (int)(c / L.wx % gy), bz = (int)(c / ((long long)L.wx * gy));
        uint32_t any = 0u;
        unsigned n = 0;
        const int left = L.dims[0] - xw * 32;  // the last word's pad bits are no voxels
        const uint32_t row = left >= 32 ? 0xffffffffu : ((1u << left) - 1u);
        for (int r = lane; r < E * E; r += 32) {
            const int y = by * E + r % E, z = bz * E + r / E;
            if (y < L.dims[1] && z < L.dims[2]) {
                const uint32_t u = __ldg(&U[((size_t)z * L.dims[1] + y) * L.wx + xw]) & row;
                any |= u;
                n += __popc(u);
            }
        }
        any = __reduce_or_sync(0xffffffffu, any);
        if (!any) continue;
        n = __reduce_add_sync(0xffffffffu, n);
        if (lane == 0) {
            atomicAdd(&ds->listed_voxels, (unsigned long long)n);
            for (int k = 0; k < PW; ++k) {
                const uint32_t mask = (E == 32 ? 0xffffffffu : ((1u << (E & 31)) - 1u)) << (k * E);
                const int bx = xw * PW + k;
                if (!(any & mask) || bx >= gx) continue;
                const unsigned long long pos = atomicAdd(&ds->listed, 1ull);
                if ((long long)pos < cap) list[pos] = ((long long)bz * gy + by) * gx + bx;
                else atomicAdd(&ds->list_overflow, 1ull);
            }
        }
    }
}

// Polynomial of far clusters about a centre: value, gradient, half the Hessian (xx, yy, zz,
// xy + yx, xz + zx, yz + zy), the bound of what it leaves out and the summed term magnitudes.
struct Local {
    float v[12];  // L0, L1[3], L2[6], err, mag
};

// Adds cluster c to the polynomial about a centre it is seen from at (dx, dy, dz) = c - centre,
// when it is far enough for every point within rho of the centre; false when it is near.
//
// With y = c - q, the cluster's solid angle from q is f(y) + g(y) within 3 Q / (|y| - r)^4
// (gbsdf_internal.h), f = D.y / |y|^3, g = (tr M - 3 y^T M y / |y|^2) / |y|^3. f and g are first
// and second derivatives of 1/|y| contracted with D and M, and the n-th derivative form of
// 1/|y| has norm n! / |y|^(n+1) (n! P_n(cos) / |y|^(n+1) along one direction). With d the
// centre's distance and t = rho / d, f's terms of degree k in the offset are thus at most
// |D| (k+1) t^k / d^2 and g's at most |M|_* (k+2)(k+1) t^k / d^3, |D| <= A and the nuclear norm
// |M|_* <= sum a_i |g_i - c| <= A r. f is kept to degree 2, g to degree 1; the rests sum to
//   A t^3 (4 - 3 t) / ((1 - t)^2 d^2)  and  A r t^2 (12 - 16 t + 6 t^2) / ((1 - t)^3 d^3).
__device__ __forceinline__ bool local_add(const float4* __restrict__ cell, float px, float py, float pz, float rho,
                                          float beta, Local& a) {
    const float4 c0 = __ldg(cell);  // centre, radius
    const float dx = c0.x - px, dy = c0.y - py, dz = c0.z - pz;
    const float d2 = dx * dx + dy * dy + dz * dz;
    const float ir = rsqrtf(d2), d = d2 * ir;
    const float t = rho * ir;
    if (!(t <= kBqRatio && d - rho > beta * c0.w)) return false;
    const float4 c1 = __ldg(cell + 1), c2 = __ldg(cell + 2), c3 = __ldg(cell + 3), c4 = __ldg(cell + 4);
    const float A = c1.w;
    const float m0 = c2.x, m1 = c2.y, m2 = c2.z, m3 = c2.w, m4 = c3.x, m5 = c3.y, m6 = c3.z, m7 = c3.w, m8 = c4.x;
    const float ir2 = ir * ir, ir3 = ir * ir2, ir5 = ir3 * ir2;
    const float Dy = __fmaf_rn(c1.z, dz, __fmaf_rn(c1.y, dy, c1.x * dx));
    const float tr = m0 + m4 + m8;
    // (M + M^T) y; y^T M y = half of its product with y
    const float sx = __fmaf_rn(m2 + m6, dz, __fmaf_rn(m1 + m3, dy, 2.0f * m0 * dx));
    const float sy = __fmaf_rn(m5 + m7, dz, __fmaf_rn(2.0f * m4, dy, (m1 + m3) * dx));
    const float sz = __fmaf_rn(2.0f * m8, dz, __fmaf_rn(m5 + m7, dy, (m2 + m6) * dx));
    const float yMy = 0.5f * __fmaf_rn(sz, dz, __fmaf_rn(sy, dy, sx * dx));
    const float q2 = yMy * ir2;
    a.v[0] += __fmaf_rn(__fmaf_rn(-3.0f, q2, tr), ir3, Dy * ir3);
    // gradient in the offset (y = y0 - offset): -grad f - grad g
    const float gy = 3.0f * ir5 * (Dy + tr - 5.0f * q2), gs = 3.0f * ir5;
    a.v[1] += __fmaf_rn(gy, dx, __fmaf_rn(gs, sx, -c1.x * ir3));
    a.v[2] += __fmaf_rn(gy, dy, __fmaf_rn(gs, sy, -c1.y * ir3));
    a.v[3] += __fmaf_rn(gy, dz, __fmaf_rn(gs, sz, -c1.z * ir3));
    // half the Hessian of f
    const float h7 = 7.5f * Dy * ir5 * ir2, h5 = -1.5f * ir5;
    const float hd = h5 * Dy;
    a.v[4] += __fmaf_rn(h7 * dx, dx, __fmaf_rn(2.0f * h5 * c1.x, dx, hd));
    a.v[5] += __fmaf_rn(h7 * dy, dy, __fmaf_rn(2.0f * h5 * c1.y, dy, hd));
    a.v[6] += __fmaf_rn(h7 * dz, dz, __fmaf_rn(2.0f * h5 * c1.z, dz, hd));
    a.v[7] += 2.0f * __fmaf_rn(h7 * dx, dy, h5 * __fmaf_rn(c1.x, dy, c1.y * dx));
    a.v[8] += 2.0f * __fmaf_rn(h7 * dx, dz, h5 * __fmaf_rn(c1.x, dz, c1.z * dx));
    a.v[9] += 2.0f * __fmaf_rn(h7 * dy, dz, h5 * __fmaf_rn(c1.y, dz, c1.z * dy));
    const float e = (d - rho - c0.w) * 0.99999f, ie2 = 1.0f / (e * e);
    const float u = 1.0f / (1.0f - t), u2 = u * u;
    const float ad = A * ir2;
    const float rest = t * t * u2 * ad *
                       (t * (4.0f - 3.0f * t) + c0.w * ir * u * (12.0f + t * (6.0f * t - 16.0f)));
    a.v[10] += 1.0001f * (3.0f * c4.y * ie2 * ie2 + rest);
    a.v[11] += ad * u2 * (1.0f + 2.0f * c0.w * ir * u);
    return true;
}

// CAPS: a cluster of little solid angle (at most A / (d - rho - r)^2 from anywhere within rho)
// enters by that bound alone; caps are small and few, so nearly all do.
__device__ __forceinline__ bool bound_add(const float4* __restrict__ cell, float px, float py, float pz, float rho,
                                          float& err) {
    const float4 c0 = __ldg(cell);
    const float dx = c0.x - px, dy = c0.y - py, dz = c0.z - pz;
    const float e = (sqrtf(__fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx))) - rho - c0.w) * 0.9999f;
    const float A = __ldg(&cell[1].w);
    if (!(e > 0.0f && A <= kCapBound * (e * e))) return false;
    err += __fdividef(1.0001f * A, e * e);
    return true;
}
template <bool CAPS>
__device__ __forceinline__ bool far_add(const float4* __restrict__ cell, float px, float py, float pz, float rho,
                                        float beta, Local& a) {
    if constexpr (CAPS) return bound_add(cell, px, py, pz, rho, a.v[10]);
    else return local_add(cell, px, py, pz, rho, beta, a);
}

__device__ __forceinline__ float local_at(const float* v, float x, float y, float z) {
    float s = __fmaf_rn(v[4] * x, x, __fmaf_rn(v[5] * y, y, v[6] * z * z));
    s = __fmaf_rn(v[7] * x, y, __fmaf_rn(v[8] * x, z, __fmaf_rn(v[9] * y, z, s)));
    return v[0] + __fmaf_rn(v[1], x, __fmaf_rn(v[2], y, __fmaf_rn(v[3], z, s)));
}

// Sum of the CTA's polynomials (fixed order) into out[0..11]; red: kBqWarps x 12 scratch.
__device__ __forceinline__ void local_sum(const Local& a, float (*red)[12], float* out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 12; ++k) {
        float x = a.v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) red[warp][k] = x;
    }
    __syncthreads();
    if (threadIdx.x < 12) {
        float x = 0.0f;
        for (int w = 0; w < kBqWarps; ++w) x += red[w][threadIdx.x];
        out[threadIdx.x] = x;
    }
    __syncthreads();
}

// Slot of each flagged thread in thread order, `base` on; returns the flagged count of the CTA.
// cnt: kBqWarps words; two barriers.
__device__ __forceinline__ int cta_slots(bool flag, int base, int& slot, unsigned* cnt) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned bal = __ballot_sync(0xffffffffu, flag);
    if (lane == 0) cnt[warp] = __popc(bal);
    __syncthreads();
    int before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kBqWarps; ++w) {
        const int n = (int)cnt[w];
        before += (w < warp) ? n : 0;
        all += n;
    }
    __syncthreads();
    slot = base + before + __popc(bal & ((1u << lane) - 1u));
    return all;
}

// Appends the flagged of `n` items to a list of capacity `cap` in item order; returns how many
// there are (which may exceed the capacity). item(i): i's entry, or -1 when it is not flagged.
template <class F>
__device__ __forceinline__ int cta_list(int n, unsigned* list, int cap, unsigned* cnt, F item) {
    int total = 0;
    for (int base = 0; base < n; base += kBqThreads) {
        const int i = base + (int)threadIdx.x;
        const int e = i < n ? item(i) : -1;
        int slot;
        const int add = cta_slots(e >= 0, total, slot, cnt);
        if (e >= 0 && slot < cap) list[slot] = (unsigned)e;
        total += add;
    }
    __syncthreads();
    return total;
}

// The marked voxels of the listed blocks. Persistent CTAs.
// CAPS: f holds the mesh's caps (k_caps.cu) and a voxel with |w(caps)| < 1/2 is inside iff its
// bit of X.k is set, when neither it nor its column is left out and it lies on no cap; the
// others keep their marks, and so do those next to the mesh, whose side the FP64 sum defines
// where they are on it.
// What bounds it: the FP32 work of the near clusters and triangles of dense bricks, and the
// cluster tests of a block for sparse ones; nothing but a few bits a voxel goes to memory.
template <int BB, bool CAPS>
__global__ void __launch_bounds__(kBqThreads) winding_blocks_kernel(
    FwnView f, Lattice L, Crossings X, uint32_t* __restrict__ U, uint32_t* __restrict__ S, uint32_t* __restrict__ E,
    const long long* __restrict__ list, long long cap, int only_if, const float* __restrict__ dist, int dist_sq,
    float surf_tol_vox, DevState* ds, long long* __restrict__ fb, long long fb_cap) {
    if (only_if && !ds->patching) return;
    __shared__ unsigned s_2[kBqCap2], s_1[kBqCap1], s_1b[BB == 2 ? kBqCap1 : 1], s_0[kBqCap0];
    __shared__ float s_red[kBqWarps][12], s_blk[12], s_brk[12];
    __shared__ unsigned s_cnt[kBqWarps];
    __shared__ unsigned short s_pend[512];
    __shared__ unsigned s_mark[16], s_in[16], s_keep[16], s_und[16];
    const int tid = threadIdx.x, lane = tid & 31;
    const float tau = surf_tol_vox * L.h;
    const int gx = (L.nb[0] + BB - 1) / BB, gy = (L.nb[1] + BB - 1) / BB;
    const long long nblk = min((long long)ds->listed, cap);
    unsigned certified = 0, taken = 0;
    for (long long it = blockIdx.x; it < nblk; it += gridDim.x) {
        const long long blk = list[it];
        const int Bx = (int)(blk % gx) * BB, By = (int)(blk / gx % gy) * BB, Bz = (int)(blk / ((long long)gx * gy)) * BB;
        // ---- the block: far clusters of the upper levels into its polynomial, the others listed
        const float bcx = lattice_mid(L.mn[0], Bx * 8, 4.0f * BB - 0.5f, L.h),
                    bcy = lattice_mid(L.mn[1], By * 8, 4.0f * BB - 0.5f, L.h),
                    bcz = lattice_mid(L.mn[2], Bz * 8, 4.0f * BB - 0.5f, L.h);
        const float slop = 1e-6f * (fabsf(bcx) + fabsf(bcy) + fabsf(bcz));
        // half the diagonal of the block's (brick's) points
        const float rho_b = (BB == 2 ? 12.9904f : 6.0622f) * L.h * 1.0002f + slop;
        const float rho = 6.0622f * L.h * 1.0002f + slop;
        const float next = 7e-4f * L.h + 2.0f * slop, next_sq = next * next;  // CAPS: "next to the mesh"
        int n2, n1 = 0;
        {
            Local a{};
            n2 = cta_list(f.n[2], s_2, kBqCap2, s_cnt, [&](int i) {
                return far_add<CAPS>(f.cells[2] + 5 * (size_t)i, bcx, bcy, bcz, rho_b, kFwnBetaBlock, a) ? -1 : i;
            });
            if (n2 <= kBqCap2)
                n1 = cta_list(n2 * kFwnFan, s_1, kBqCap1, s_cnt, [&](int i) {
                    const int k = (int)s_2[i / kFwnFan] * kFwnFan + i % kFwnFan;
                    return k >= f.n[1] || far_add<CAPS>(f.cells[1] + 5 * (size_t)k, bcx, bcy, bcz, rho_b, kFwnBetaBlock, a) ? -1 : k;
                });
            local_sum(a, s_red, s_blk);
        }
        const bool too_many = n2 > kBqCap2 || n1 > kBqCap1;
        for (int sub = 0; sub < BB * BB * BB; ++sub) {
            const int bx = Bx + (sub & (BB - 1)), by = By + (BB == 2 ? ((sub >> 1) & 1) : 0),
                      bz = Bz + (BB == 2 ? (sub >> 2) : 0);
            if (bx >= L.nb[0] || by >= L.nb[1] || bz >= L.nb[2]) continue;
            // ---- the brick's marked voxels (voxel v: x = v & 7, y = v >> 3 & 7, z = v >> 6)
            const int shift = (bx * 8) & 31;
            if (tid < 16) {
                unsigned m = 0u;
                const int left = L.dims[0] - bx * 8;
                const unsigned row = left >= 8 ? 0xffu : ((1u << left) - 1u);
                for (int r = 0; r < 4; ++r) {
                    const int y = by * 8 + ((tid * 4 + r) & 7), z = bz * 8 + ((tid * 4 + r) >> 3);
                    if (y >= L.dims[1] || z >= L.dims[2]) continue;
                    const unsigned b = U[((size_t)z * L.dims[1] + y) * L.wx + (bx >> 2)] >> shift;
                    m |= (b & row) << (8 * r);
                }
                s_mark[tid] = m;
                s_in[tid] = 0u;
                s_keep[tid] = 0u;
            }
            __syncthreads();
            unsigned any = 0u;
#pragma unroll
            for (int k = 0; k < 16; ++k) any |= s_mark[k];
            if (!any) {
                __syncthreads();
                continue;
            }
            // voxels on the surface are inside; the others are pending, listed in Morton order
            int np = 0;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int v = morton_voxel(half * 256 + tid);
                bool pend = (s_mark[v >> 5] >> (v & 31)) & 1u;
                const int x = bx * 8 + (v & 7), y = by * 8 + ((v >> 3) & 7), z = bz * 8 + (v >> 6);
                if (pend && dist) {
                    const float d = dist[((size_t)z * L.dims[1] + y) * L.dims[0] + x];
                    if (dist_sq ? (d <= tau * tau) : (d <= tau)) {
                        atomicOr(&s_in[v >> 5], 1u << (v & 31));
                        pend = false;
                    } else if (CAPS) {
                        const size_t col = (size_t)y * L.dims[0] + x;
                        if (!(dist_sq ? (d > next_sq) : (d > next)) || ((X.bad[col >> 5] >> (col & 31)) & 1u) ||
                            ((X.unsure[word_of(L, x, y, z)] >> (x & 31)) & 1u)) {
                            atomicOr(&s_keep[v >> 5], 1u << (v & 31));
                            pend = false;
                        }
                    }
                }
                int slot;
                const int n = cta_slots(pend, np, slot, s_cnt);
                if (pend) s_pend[slot] = (unsigned short)v;
                np += n;
            }
            __syncthreads();
            // ---- the brick: the block's near clusters again, then their children
            int n0 = 0;
            const float kx = lattice_mid(L.mn[0], bx * 8, 3.5f, L.h), ky = lattice_mid(L.mn[1], by * 8, 3.5f, L.h),
                        kz = lattice_mid(L.mn[2], bz * 8, 3.5f, L.h);
            if (np > 0 && !too_many) {
                Local a{};
                const unsigned* up = s_1;
                int nu = n1;
                if (BB == 2) {
                    nu = cta_list(n1, s_1b, kBqCap1, s_cnt, [&](int i) {
                        return far_add<CAPS>(f.cells[1] + 5 * (size_t)s_1[i], kx, ky, kz, rho, kFwnBetaBlock, a) ? -1 : (int)s_1[i];
                    });
                    up = s_1b;
                }
                n0 = cta_list(nu * kFwnFan, s_0, kBqCap0, s_cnt, [&](int i) {
                    const int k = (int)up[i / kFwnFan] * kFwnFan + i % kFwnFan;
                    return k >= f.n[0] || far_add<CAPS>(f.cells[0] + 5 * (size_t)k, kx, ky, kz, rho, kFwnBetaBrick, a) ? -1 : k;
                });
                local_sum(a, s_red, s_brk);
            }
            const bool skip = too_many || n0 > kBqCap0;  // left to the refining stage
            // ---- the voxels: TEAM lanes each, enough teams to keep the CTA's lanes busy. What the
            // first pass leaves undecided takes a second one with a wider near range.
            for (int pass = 0; pass < 2 && np > 0; ++pass) {
                const float beta = pass ? kFwnBetaFine : kFwnBeta;
                if (tid < 16) s_und[tid] = 0u;
                __syncthreads();
                int lt = 0;
                while (lt < 5 && (kBqThreads >> (lt + 1)) >= np) ++lt;
                const int team = 1 << lt, teams = kBqThreads >> lt, me = tid & (team - 1);
                for (int jb = 0; jb < np; jb += teams) {
                    const int j = jb + (tid >> lt);
                    const bool on = j < np;
                    const int v = on ? s_pend[j] : 0;
                    const int x = bx * 8 + (v & 7), y = by * 8 + ((v >> 3) & 7), z = bz * 8 + (v >> 6);
                    const f3 p = lattice_point(L.mn[0], L.mn[1], L.mn[2], x, y, z, L.h);
                    Sum a;
                    if (on && !skip) {
                        if (me == 0) {
                            a.s = local_at(s_blk, p.x - bcx, p.y - bcy, p.z - bcz);
                            kahan_add(a.s, a.c, local_at(s_brk, p.x - kx, p.y - ky, p.z - kz));
                            a.err = s_blk[10] + s_brk[10];
                            a.mag = s_blk[11] + s_brk[11];
                        }
                        for (int i = me; i < n0; i += team) {
                            const unsigned k = s_0[i];
                            if (CAPS && pass == 0) {
                                if (bound_add(f.cells[0] + 5 * (size_t)k, p.x, p.y, p.z, 0.0f, a.err)) continue;
                            } else if (cell_far(f.cells[0] + 5 * (size_t)k, p, beta, a)) {
                                continue;
                            }
                            const long long t0 = (long long)k * kFwnLeaf;
                            const int m = (int)min((long long)kFwnLeaf, f.T - t0);
                            for (int t = 0; t < m; ++t) leaf_term<CAPS>(f.leaf + 5 * (t0 + t), p, beta, a);
                        }
                    }
                    __syncwarp();
                    float tot = a.s - a.c, err = a.err, mag = a.mag;
                    int near = a.near ? 1 : 0;
                    for (int o = team >> 1; o > 0; o >>= 1) {
                        tot += __shfl_xor_sync(0xffffffffu, tot, o);
                        err += __shfl_xor_sync(0xffffffffu, err, o);
                        mag += __shfl_xor_sync(0xffffffffu, mag, o);
                        if (CAPS) near |= __shfl_xor_sync(0xffffffffu, near, o);
                    }
                    if (on && me == 0) {
                        const float w = fabsf(tot * kInv4Pi);
                        const float e = (err * 1.0001f + kFwnSlackRel * mag) * kInv4Pi + kFwnSlackAbs;
                        const bool out = !skip && !near && w + e < 0.5f, in = !skip && w - e >= 0.5f;
                        if (CAPS ? out : (in || out)) {
                            if (CAPS ? (X.k[word_of(L, x, y, z)] >> (x & 31)) & 1u : in)
                                atomicOr(&s_in[v >> 5], 1u << (v & 31));
                            ++certified;
                        } else if (CAPS && (pass == 1 || skip || near || in)) {
                            atomicOr(&s_keep[v >> 5], 1u << (v & 31));
                        } else if (pass == 0 && !skip) {
                            atomicOr(&s_und[v >> 5], 1u << (v & 31));
                        } else {
                            const unsigned long long k = atomicAdd(&ds->fwn_left, 1ull);
                            if ((long long)k < fb_cap) {
                                fb[k] = ((long long)z * L.dims[1] + y) * L.dims[0] + x;
                            } else {  // no room: it stays marked for the next pass
                                atomicOr(&s_keep[v >> 5], 1u << (v & 31));
                                atomicAdd(&ds->list_overflow, 1ull);
                            }
                        }
                    }
                }
                __syncthreads();
                if (pass == 0) {
                    np = 0;
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        const int v = morton_voxel(half * 256 + tid);
                        const bool und = (s_und[v >> 5] >> (v & 31)) & 1u;
                        int slot;
                        const int n = cta_slots(und, np, slot, s_cnt);
                        if (und) s_pend[slot] = (unsigned short)v;
                        np += n;
                    }
                    __syncthreads();
                }
            }
            __syncthreads();
            // ---- the bits of the brick's rows (four bricks share a word)
            if (tid < 64) {
                const unsigned keep = (s_keep[tid >> 2] >> (8 * (tid & 3))) & 0xffu;
                const unsigned done = ((s_mark[tid >> 2] >> (8 * (tid & 3))) & 0xffu) & ~keep;
                const unsigned in = (s_in[tid >> 2] >> (8 * (tid & 3))) & 0xffu;
                if (done) {
                    const size_t w = ((size_t)(bz * 8 + (tid >> 3)) * L.dims[1] + by * 8 + (tid & 7)) * L.wx + (bx >> 2);
                    atomicAnd(&U[w], ~(done << shift));
                    atomicAnd(&S[w], ~(done << shift));
                    if (in) atomicOr(&S[w], in << shift);
                    if (E) atomicOr(&E[w], done << shift);
                    taken += __popc(done);
                }
            }
            __syncthreads();
        }
    }
    const unsigned cw = __reduce_add_sync(0xffffffffu, certified), tw = __reduce_add_sync(0xffffffffu, taken);
    if (lane == 0) {
        if (cw) atomicAdd(&ds->fwn_certified, (unsigned long long)cw);
        if (tw) atomicAdd(only_if ? &ds->patched_voxels : &ds->fixup_voxels, (unsigned long long)tw);
    }
}

// ---- nearest distances ----------------------------------------------------------------
constexpr int kNdCap2 = 512, kNdCap1 = 1024, kNdCap0 = 2048, kNdCapW = 512;

__device__ __forceinline__ float cta_min(float x, float* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = fminf(x, __shfl_xor_sync(0xffffffffu, x, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
    __syncthreads();
    x = red[0];
#pragma unroll
    for (int w = 1; w < kBqWarps; ++w) x = fminf(x, red[w]);
    __syncthreads();
    return x;
}

// A warp's walk down to one cluster near p: of the n clusters item(i) the one of the least
// box distance, then its nearest child, to the lowest level; returns the least distance to that
// cluster's triangles (an upper bound of p's distance to the mesh; the same in all lanes) and the
// cluster.
template <class F>
__device__ __forceinline__ float walk_near(const FwnView& f, int level, int n, const f3& p, F item, int& k) {
    const int lane = threadIdx.x & 31;
    float best = __int_as_float(0x7f800000);
    int bk = -1;
    for (int i = lane; i < n; i += 32) {
        const int k = item(i);
        const float d = box_dist_sq(f.box[level] + 2 * (size_t)k, p);
        if (d < best || bk < 0) {
            best = d;
            bk = k;
        }
    }
    k = warp_argmin(bk < 0 ? __int_as_float(0x7f800000) : best, bk < 0 ? 0x7fffffff : bk);
    for (int l = level - 1; l >= 0; --l) {
        const int c = k * kFwnFan + (lane & 15);
        const bool on = c < f.n[l];
        k = warp_argmin(on ? box_dist_sq(f.box[l] + 2 * (size_t)c, p) : __int_as_float(0x7f800000), on ? c : 0x7fffffff);
    }
    const long long t = (long long)k * kFwnLeaf + (lane & 7);
    float d = t < f.T ? sqrtf(leaf_dist_sq(f.leaf + 5 * t, p)) : __int_as_float(0x7f800000);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) d = fminf(d, __shfl_xor_sync(0xffffffffu, d, o));
    return d;
}

// Squared distance of every voxel of a brick to its nearest triangle: the exact distance's
// minimum over every triangle that can hold it. With u the distance from a centre to any
// triangle, no voxel within rho of the centre is farther than u + rho from the mesh, and a
// cluster whose box is farther than u + 2 rho from the centre holds no voxel's nearest triangle.
// The brick keeps the clusters of each level that pass, each of its octants those that pass for
// it, nearest ones first, and a voxel skips a cluster whose box, or a triangle whose bounding
// sphere or plane, lies beyond its best so far. The lanes first test (cluster, 2^3 cube) and
// (triangle, 2^3 cube) pairs, 32 at a time, against the cubes' worst bests: of what an octant
// keeps, most is near none of its voxels. The tests are widened by the rounding of both sides, so the
// minimum is that over all triangles. (Boxes, not spheres: a run of a mug wall's long
// triangles is flat, and a voxel within its sphere's radius of the wall would keep it.)
// Bound by the FP32 work of the tests and exact distances (71% of the issue slots while active, 26
// lanes of 32; 80 registers, three CTAs an SM: with the 97 the compiler takes, two, 3.5 ms below).
// Replaces a walk of 128-triangle tiles in input order for each voxel: 181 x 141 x 171 mug,
// 24,000 triangles, 56.5 -> 3.1 ms (3.4 without the pairs and the order); 48 x 48 x 52, 2,712
// triangles, 0.72 -> 0.33 (0.46); where bricks are too crowded to list, 179,840 triangles, 215 x
// 215 x 220 558 -> 43 and 48 x 48 x 52 20.5 -> 10.1.
// One CTA a brick and no persistent loop: the bricks' work differs by more than ten times (on
// a mug's axis the whole wall is equally near), and the hardware's own order balances it.
__global__ void __launch_bounds__(kBqThreads, 3) nearest_bricks_kernel(FwnView f, Lattice L, float* __restrict__ d2out) {
    __shared__ unsigned s_2[kNdCap2], s_1[kNdCap1], s_0[kNdCap0], s_w[kBqWarps][kNdCapW];
    __shared__ unsigned s_cnt[kBqWarps];
    __shared__ float s_u;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (long long b = blockIdx.x; b < L.nbricks; b += gridDim.x) {
        const int bx = (int)(b % L.nb[0]), by = (int)(b / L.nb[0] % L.nb[1]), bz = (int)(b / ((long long)L.nb[0] * L.nb[1]));
        const f3 kc = mk(lattice_mid(L.mn[0], bx * 8, 3.5f, L.h), lattice_mid(L.mn[1], by * 8, 3.5f, L.h),
                         lattice_mid(L.mn[2], bz * 8, 3.5f, L.h));
        const float slop = 2e-6f * (fabsf(kc.x) + fabsf(kc.y) + fabsf(kc.z));
        const float rho = 6.0622f * L.h * 1.0002f + slop;  // half the diagonal of the brick's points
        // the squared reach of a box: what its distance from the centre may be at most
        auto reach_sq = [&](float u, float rr) {
            const float r = (u + 2.0f * rr) * 1.00002f + slop;
            return r * r;
        };
        if (tid < 32) {
            int kn;
            const float u = walk_near(f, 2, f.n[2], kc, [](int i) { return i; }, kn);
            if (tid == 0) s_u = u;
        }
        __syncthreads();
        const float lim_b = reach_sq(s_u, rho);
        auto children = [&](const unsigned* up, int level, int i) {
            const int k = (int)up[i / kFwnFan] * kFwnFan + i % kFwnFan;
            return k >= f.n[level] || box_dist_sq(f.box[level] + 2 * (size_t)k, kc) > lim_b ? -1 : k;
        };
        int n1 = 0, n0 = 0;
        const int n2 = cta_list(f.n[2], s_2, kNdCap2, s_cnt, [&](int i) {
            return box_dist_sq(f.box[2] + 2 * (size_t)i, kc) > lim_b ? -1 : i;
        });
        if (n2 <= kNdCap2) n1 = cta_list(n2 * kFwnFan, s_1, kNdCap1, s_cnt, [&](int i) { return children(s_2, 1, i); });
        if (n2 <= kNdCap2 && n1 <= kNdCap1)
            n0 = cta_list(n1 * kFwnFan, s_0, kNdCap0, s_cnt, [&](int i) { return children(s_1, 0, i); });
        // too many to list, or none (an FP32 distance to a sliver can fall short of its own box):
        // every cluster
        const bool all = n2 > kNdCap2 || n1 > kNdCap1 || n0 > kNdCap0 || n0 == 0;
        {
            // a warp takes the 4 x 4 x 4 voxels of one octant (Morton order), two a lane, and
            // keeps the clusters that pass for the octant
            const int ox = (warp & 1) * 4, oy = (warp & 2) * 2, oz = (warp & 4);
            const f3 oc = mk(lattice_mid(L.mn[0], bx * 8 + ox, 1.5f, L.h), lattice_mid(L.mn[1], by * 8 + oy, 1.5f, L.h),
                             lattice_mid(L.mn[2], bz * 8 + oz, 1.5f, L.h));
            const float rho_o = 2.5981f * L.h * 1.0002f + slop;
            int vx[2];
            float best[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) vx[k] = morton_voxel(warp * 64 + k * 32 + lane);
            // A limit comes from the FP32 distance of a centre to some triangle. A triangle without
            // area has none for some points, and a sliver's can be far off, so a limit may not
            // hold for a voxel: a voxel left above its limit shows it, and the octant then takes every
            // cluster without one.
            for (bool again = false;; again = true) {
                const bool every = all || again;
                int nc = every ? f.n[0] : n0, kn = -1, far0 = 0;
                const unsigned* near = nullptr;  // null: every cluster
                // distances start at 1e6 (squared 1e12)
                float start = again ? 1e6f : fminf(1e6f, s_u + rho);
                if (!every) {
                    near = s_0;
                    const float u = walk_near(f, 0, n0, oc, [&](int i) { return (int)s_0[i]; }, kn);
                    start = fminf(start, u + rho_o);
                    const float lim = reach_sq(u, rho_o), soon = u * u;  // (u + rho / 4 to u + rho: within 1%)
                    int n = 0, m = 0;  // kept from the front (near ones) and from the back of the list
                    for (int base = 0; base < n0; base += 32) {
                        const int i = base + lane;
                        // (u, and with it lim, is NaN when the nearest cluster has no area: all pass)
                        const bool on = i < n0 && (int)s_0[i] != kn;
                        const float d = on ? box_dist_sq(f.box[0] + 2 * (size_t)s_0[i], oc) : 0.0f;
                        const bool keep = on && !(d > lim), first = keep && !(d > soon);
                        const unsigned bal = __ballot_sync(0xffffffffu, keep), balf = __ballot_sync(0xffffffffu, first);
                        const unsigned below = (1u << lane) - 1u;
                        const int slot = first ? n + __popc(balf & below) : kNdCapW - 1 - (m + __popc(bal & ~balf & below));
                        n += __popc(balf);
                        m += __popc(bal & ~balf);
                        if (keep && n + m <= kNdCapW) s_w[warp][slot] = s_0[i];
                    }
                    __syncwarp();
                    if (n + m <= kNdCapW) {
                        near = s_w[warp];
                        nc = n + m;
                        far0 = n;
                    }
                }
                f3 p[2];
                float lim[2], lim_sq[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    best[k] = 1e12f;
                    p[k] = lattice_point(L.mn[0], L.mn[1], L.mn[2], bx * 8 + (vx[k] & 7), by * 8 + ((vx[k] >> 3) & 7),
                                         bz * 8 + (vx[k] >> 6), L.h);
                    lim[k] = start * 1.00002f + slop;
                    lim_sq[k] = lim[k] * lim[k];
                }
                // the octant's eight 2^3 cubes: lane group g = lane / 8 holds voxels of cubes g and 4 + g
                f3 cc[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const int cv = morton_voxel(warp * 64 + k * 32 + (lane & 24));
                    cc[k] = mk(lattice_mid(L.mn[0], bx * 8 + (cv & 7), 0.5f, L.h),
                               lattice_mid(L.mn[1], by * 8 + ((cv >> 3) & 7), 0.5f, L.h),
                               lattice_mid(L.mn[2], bz * 8 + (cv >> 6), 0.5f, L.h));
                }
                const float rho_c = 0.8661f * L.h * 1.0002f + slop;
                auto cube_reach = [&](int k) {  // a cube's points are within this of whatever changes a voxel of it
                    float l = lim[k];
#pragma unroll
                    for (int o = 1; o < 8; o <<= 1) l = fmaxf(l, __shfl_xor_sync(0xffffffffu, l, o));
                    return l * 1.00002f + rho_c;
                };
                // the triangles of cluster k0: each against the cubes, a lane a pair, then those that
                // come near voxel by voxel
                auto take = [&](long long k0, unsigned cubes) {
                    bool need[2];
#pragma unroll
                    for (int k = 0; k < 2; ++k)
                        need[k] = ((cubes >> (4 * k + (lane >> 3))) & 1u) &&
                                  !(box_dist_sq(f.box[0] + 2 * k0, p[k]) > lim_sq[k]);
                    if (!__any_sync(0xffffffffu, need[0] || need[1])) return;
                    const float r0 = cube_reach(0), r1 = cube_reach(1);
                    const long long tl = k0 * kFwnLeaf + (lane & 7);
                    unsigned pass[2];
                    {
                        const bool on = tl < f.T;
                        const float4* o = f.leaf + 5 * (on ? tl : 0);
                        const float4 g = __ldg(o), n = __ldg(o + 1);
                        const float nn = __ldg(&o[4].y) * 1.0001f;
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            const float dx = g.x - cc[k].x, dy = g.y - cc[k].y, dz = g.z - cc[k].z;
                            const float rr = k ? r1 : r0, r = rr + g.w;
                            const float h = __fmaf_rn(n.z, dz, __fmaf_rn(n.y, dy, n.x * dx));
                            pass[k] = __ballot_sync(0xffffffffu, on && !(__fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx)) > r * r ||
                                                                         h * h > nn * (rr * rr)));
                        }
                    }
                    unsigned some = pass[0] | pass[1];
                    some |= some >> 16;
                    some = (some | some >> 8) & 0xffu;
                    for (; some; some &= some - 1) {
                        const int t = __ffs(some) - 1;
                        const float4* o = f.leaf + 5 * (k0 * kFwnLeaf + t);
                        const float4 g = __ldg(o), n = __ldg(o + 1);
                        const float nn = __ldg(&o[4].y) * 1.0001f;
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            const float dx = g.x - p[k].x, dy = g.y - p[k].y, dz = g.z - p[k].z, r = lim[k] + g.w;
                            const float h = __fmaf_rn(n.z, dz, __fmaf_rn(n.y, dy, n.x * dx));
                            if (!need[k] || !((pass[k] >> ((lane & 24) + t)) & 1u) ||
                                __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx)) > r * r || h * h > nn * lim_sq[k])
                                continue;
                            const float d2 = leaf_dist_sq(o, p[k]);
                            if (d2 < best[k]) {
                                best[k] = d2;
                                lim[k] = fminf(lim[k], sqrtf(d2) * 1.00002f + slop);
                                lim_sq[k] = lim[k] * lim[k];
                            }
                        }
                    }
                };
                // the cluster found nearest to the centre first, then the near ones, then the others:
                // four clusters at a time against the cubes, a lane a pair
                if (kn >= 0) take(kn, 0xffu);
                const int cv = morton_voxel(warp * 64 + 8 * (lane & 7));
                const f3 cl = mk(lattice_mid(L.mn[0], bx * 8 + (cv & 7), 0.5f, L.h),
                                 lattice_mid(L.mn[1], by * 8 + ((cv >> 3) & 7), 0.5f, L.h),
                                 lattice_mid(L.mn[2], bz * 8 + (cv >> 6), 0.5f, L.h));
                for (int base = 0; base < nc; base += 4) {
                    const float r0 = __shfl_sync(0xffffffffu, cube_reach(0), 8 * (lane & 3)),
                                r1 = __shfl_sync(0xffffffffu, cube_reach(1), 8 * (lane & 3));
                    const float r = (lane & 4) ? r1 : r0;
                    const int i = base + (lane >> 3);
                    unsigned k = i;
                    if (near == s_w[warp]) k = near[min(i, nc - 1) < far0 ? i : kNdCapW - 1 - (min(i, nc - 1) - far0)];
                    else if (near) k = near[min(i, nc - 1)];
                    unsigned pass = __ballot_sync(0xffffffffu, i < nc && (int)k != kn &&
                                                                   !(box_dist_sq(f.box[0] + 2 * (size_t)k, cl) > r * r));
                    while (pass) {
                        const int q = (__ffs(pass) - 1) & ~7;
                        const unsigned cubes = (pass >> q) & 0xffu;
                        pass &= ~(0xffu << q);
                        take((long long)__shfl_sync(0xffffffffu, k, q), cubes);
                    }
                }
                const float held = start * 1.00002f + slop;
                if (again || !__any_sync(0xffffffffu, fmaxf(best[0], best[1]) > held * held)) break;
            }
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int x = bx * 8 + (vx[k] & 7), y = by * 8 + ((vx[k] >> 3) & 7), z = bz * 8 + (vx[k] >> 6);
                if (x < L.dims[0] && y < L.dims[1] && z < L.dims[2])
                    d2out[((size_t)z * L.dims[1] + y) * L.dims[0] + x] = best[k];
            }
        }
        __syncthreads();
    }
}

inline unsigned sort_tiles(long long T) { return (unsigned)((T + kSortTile - 1) / kSortTile); }

// The listed voxels (or, list null, those the blocks left in f.fb2) by a walk each, then the rest
// of them triangle by triangle.
void winding_query(const Fwn& f, const float* tri9, long long T, const Lattice& L, const long long* list,
                   long long list_cap, int consumer, int only_if, uint32_t* sbits, long long* recheck,
                   long long recheck_cap, const float* dist, int dist_sq, float surf_tol_vox, DevState* ds, int num_sms,
                   cudaStream_t st) {
    GBSDF_COUNT_LAUNCH();
    fwn_query_kernel<<<(unsigned)(num_sms * 4), kQueryThreads, 0, st>>>(
        view_of(f, T), L, list ? list : f.fb2, list ? &ds->listed : &ds->fwn_left, list ? list_cap : f.fb_cap, consumer,
        only_if, sbits, dist, dist_sq, surf_tol_vox, ds, f.fb, f.fb_cap, list ? kFwnBeta : kFwnBetaRefine);
    launch_gwn_team(tri9, T, L, f.fb, f.fb_cap, consumer, sbits, recheck, recheck_cap, dist, dist_sq, surf_tol_vox, ds,
                    num_sms, st, only_if);
}

// The arrays of Fwn in one allocation: a sizing pass (base null), then a placing pass.
size_t fwn_layout(Fwn& f, char* base, long long T, long long cap) {
    size_t off = 0;
    auto take = [&](size_t b) {
        char* p = base ? base + off : nullptr;
        off += (b + 255) & ~size_t(255);
        return static_cast<void*>(p);
    };
    f.n[0] = (T + kFwnLeaf - 1) / kFwnLeaf;
    f.n[1] = (f.n[0] + kFwnFan - 1) / kFwnFan;
    f.n[2] = (f.n[1] + kFwnFan - 1) / kFwnFan;
    for (int l = 0; l < 3; ++l) {
        f.cells[l] = static_cast<FwnCell*>(take((size_t)f.n[l] * sizeof(FwnCell)));
        f.box[l] = static_cast<float4*>(take((size_t)f.n[l] * 2 * sizeof(float4)));
    }
    f.leaf = static_cast<float4*>(take((size_t)T * 5 * sizeof(float4)));
    for (int k = 0; k < 2; ++k) {
        f.key[k] = static_cast<unsigned*>(take((size_t)T * 4));
        f.idx[k] = static_cast<unsigned*>(take((size_t)T * 4));
    }
    f.hist = static_cast<unsigned*>(take((size_t)kDigits * sort_tiles(T) * 4));
    f.offs = static_cast<unsigned*>(take((size_t)kDigits * sort_tiles(T) * 4));
    f.fb = static_cast<long long*>(take((size_t)cap * 8));
    f.fb2 = static_cast<long long*>(take((size_t)cap * 8));
    f.fb_cap = cap;
    return off;
}

}  // namespace

size_t fwn_bytes(long long T, long long cap) {
    Fwn f{};
    return fwn_layout(f, nullptr, T, cap);
}

Fwn fwn_carve(void* base, long long T, long long cap) {
    Fwn f{};
    fwn_layout(f, static_cast<char*>(base), T, cap);
    return f;
}

void launch_fwn_build(const float* tri9, long long T, const Lattice& L, const Fwn& f, cudaStream_t st) {
    if (T <= 0) return;
    const unsigned tb = (unsigned)((T + 255) / 256), tiles = sort_tiles(T);
    const int side = std::max(L.dims[0], std::max(L.dims[1], L.dims[2]));
    GBSDF_COUNT_LAUNCH();
    fwn_key_kernel<<<tb, 256, 0, st>>>(tri9, T, L, (float)(1 << kKeyBits) / (float)side, f.key[0], f.idx[0]);
    for (int p = 0; p < kPasses; ++p) {
        const int a = p & 1, shift = p * kDigitBits;
        GBSDF_COUNT_LAUNCH();
        sort_hist_kernel<<<tiles, kSortThreads, 0, st>>>(f.key[a], T, shift, f.hist, tiles);
        GBSDF_COUNT_LAUNCH();
        sort_scan_kernel<<<1, 1024, 0, st>>>(f.hist, f.offs, (long long)kDigits * tiles);
        GBSDF_COUNT_LAUNCH();
        sort_scatter_kernel<<<tiles, kSortThreads, 0, st>>>(f.key[a], f.idx[a], T, shift, f.offs, tiles, f.key[a ^ 1],
                                                            f.idx[a ^ 1]);
    }
    GBSDF_COUNT_LAUNCH();
    // small CTAs: the FP64 pipes of every SM share the work (times at the kernels)
    fwn_leaf_kernel<<<(unsigned)((T + kStatThreads - 1) / kStatThreads), kStatThreads, 0, st>>>(tri9, T, f.idx[kPasses & 1], f.leaf, f.cells[0], f.box[0]);
    for (int l = 1; l < 3; ++l) {
        GBSDF_COUNT_LAUNCH();
        fwn_level_kernel<<<(unsigned)((f.n[l - 1] + 31) / 32), 32, 0, st>>>(f.cells[l - 1], f.box[l - 1], f.n[l - 1],
                                                                           f.cells[l], f.box[l]);
    }
}

void launch_winding(const Fwn* f, const float* tri9, long long T, const Lattice& L, const long long* list,
                    long long list_cap, int consumer, int only_if, uint32_t* sbits, long long* recheck,
                    long long recheck_cap, const float* dist, int dist_sq, float surf_tol_vox, DevState* ds,
                    int num_sms, cudaStream_t st) {
    if (!f) {
        launch_gwn(tri9, T, L, list, list_cap, consumer, only_if, sbits, recheck, recheck_cap, dist, dist_sq,
                   surf_tol_vox, ds, num_sms, st);
        return;
    }
    winding_query(*f, tri9, T, L, list, list_cap, consumer, only_if, sbits, recheck, recheck_cap, dist, dist_sq,
                  surf_tol_vox, ds, num_sms, st);
}

void launch_list_blocks(const uint32_t* ubits, const Lattice& L, long long* list, long long cap, DevState* ds,
                        int only_if, cudaStream_t st) {
    const int BB = block_bricks(L);
    const long long cols = (long long)L.wx * ((L.nb[1] + BB - 1) / BB) * ((L.nb[2] + BB - 1) / BB);
    const unsigned blocks = (unsigned)std::max<long long>(1, std::min<long long>((cols + 7) / 8, 152ll * 16));
    GBSDF_COUNT_LAUNCH();
    if (BB == 2) list_blocks_kernel<2><<<blocks, 256, 0, st>>>(ubits, L, list, cap, ds, only_if);
    else list_blocks_kernel<1><<<blocks, 256, 0, st>>>(ubits, L, list, cap, ds, only_if);
}

void launch_nearest(const Fwn& f, long long T, const Lattice& L, float* d2, cudaStream_t st) {
    const unsigned grid = (unsigned)std::min<long long>(L.nbricks, 1ll << 30);
    GBSDF_COUNT_LAUNCH();
    nearest_bricks_kernel<<<grid, kBqThreads, 0, st>>>(view_of(f, T), L, d2);
}

void launch_capped_blocks(const Fwn& f, long long B, const Lattice& L, const Crossings& X, uint32_t* ubits,
                          uint32_t* sbits, uint32_t* ebits, const long long* list, long long list_cap, int only_if,
                          const float* dist, int dist_sq, float surf_tol_vox, DevState* ds, int num_sms,
                          cudaStream_t st) {
    const int BB = block_bricks(L);
    const unsigned grid = (unsigned)std::min<long long>(block_count(L, BB), (long long)num_sms * 8);
    auto go = [&](auto kernel) {
        kernel<<<grid, kBqThreads, 0, st>>>(view_of(f, B), L, X, ubits, sbits, ebits, list, list_cap, only_if, dist, dist_sq,
                                            surf_tol_vox, ds, nullptr, 0);
    };
    GBSDF_COUNT_LAUNCH();
    if (BB == 2) go(winding_blocks_kernel<2, true>);
    else go(winding_blocks_kernel<1, true>);
}

void launch_winding_blocks(const Fwn& f, const float* tri9, long long T, const Lattice& L, uint32_t* ubits,
                           uint32_t* sbits, uint32_t* ebits, const long long* list, long long list_cap, int only_if,
                           long long* recheck, long long recheck_cap, const float* dist, int dist_sq,
                           float surf_tol_vox, DevState* ds, int num_sms, cudaStream_t st) {
    const int BB = block_bricks(L);
    const unsigned grid = (unsigned)std::min<long long>(block_count(L, BB), (long long)num_sms * 8);
    auto go = [&](auto kernel) {
        kernel<<<grid, kBqThreads, 0, st>>>(view_of(f, T), L, Crossings{}, ubits, sbits, ebits, list, list_cap, only_if, dist,
                                            dist_sq, surf_tol_vox, ds, f.fb2, f.fb_cap);
    };
    GBSDF_COUNT_LAUNCH();
    if (BB == 2) go(winding_blocks_kernel<2, false>);
    else go(winding_blocks_kernel<1, false>);
    winding_query(f, tri9, T, L, nullptr, 0, kGwnFixup, only_if, sbits, recheck, recheck_cap, dist, dist_sq, surf_tol_vox, ds,
                 num_sms, st);
}

}  // namespace gbsdf
