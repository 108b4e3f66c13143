// k_parity.cu — scanline parity signs [B], a strip of columns at a time.
//
// The reference runs one thread per (x, y) column, gathers up to 128 z-crossings
// of the jittered column ray from a host-built 4x4-supercell CSR, sorts them and
// writes one byte per voxel with column-strided stores (cuda_rasterizer.cu:279-368,
// CSR :824-882). Here a CTA owns a strip of 32 adjacent columns of one row: its warps
// test the strip's candidates 32 at a time, a crossing goes to its column as the first
// voxel above it, the columns' sides become toggles of one 32-bit word per z, and a
// prefix over z gives the sign words -- bit-packed signs (1 bit per voxel) instead of
// bytes.
//
// Candidate predicate per (column, triangle), identical to the reference: the
// column's supercell lies in the triangle's CSR supercell range and the jittered
// ray passes the triangle's XY AABB; then the 2D edge functions, the |area2| >=
// 1e-12 test and the barycentric hit height. An odd or overflowing (> 128) hit
// count marks the whole column unknown (exact winding later).
#include "gbsdf_device.cuh"
#include "gbsdf_internal.h"

namespace gbsdf {

namespace {

constexpr int kParThreads = 128, kParWarps = kParThreads / 32;
constexpr int kZTile = 1024;  // sign words formed at a time
// Exact-signs rays sit 1000x closer to the lattice point than the reference's jitter.
constexpr float kJXExact = 3.7e-4f;
constexpr float kJYExact = 5.1e-4f;

// SIGNED = 0: the reference's parity. SIGNED = 1: signed crossings -- a crossing whose
// projected triangle is clockwise in xy (entering an outward-oriented solid going up)
// counts +1, a counter-clockwise one -1; the running sum below a voxel is the winding
// number of a closed, consistently oriented mesh (overlapping shells included), inside
// iff nonzero; a column whose total is nonzero (a ray through a hole) or that overflows
// is unknown.
//
// Four warps share a strip, so that its list is walked four chunks at a time, and a crossing
// costs 4 bytes of shared memory per column slot, so that 44 warps fit an SM; the order of the
// list does not show. A chunk's triangles are walked by the warp, the lanes taking the columns,
// or, where they span few columns, taken by a lane each: whichever has fewer steps. Sign words
// are written where they are not zero (the grids are cleared before). Bound by latency: the
// lists' records, then the shared-memory counts. One warp a strip, its crossings' heights in
// 20 KB of shared memory, walking z voxel by voxel: 860 x 860 x 880 mug 2.70 ms, 640^3 blob 2.00,
// 150^3 sphere 0.18; this, with the grids' clearing, 0.20, 0.36 and 0.05.
template <int SIGNED>
__global__ void __launch_bounds__(kParThreads) parity_kernel(const ParTri* __restrict__ ptt,
                                                             const unsigned long long* __restrict__ off,
                                                             const unsigned* __restrict__ cnt,
                                                             const unsigned* __restrict__ list, Lattice L,
                                                             uint32_t* __restrict__ sbits,
                                                             uint32_t* __restrict__ ubits, DevState* ds) {
    __shared__ unsigned s_hit[kParityMaxHits][32];  // first voxel above a crossing; top bit: leaving
    __shared__ int s_n[32];
    __shared__ uint32_t s_tog[kZTile];
    __shared__ uint32_t s_unknown, s_any, s_scan[kParWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long strip = blockIdx.x;
    const int y = (int)(strip / L.nsx), sx = (int)(strip % L.nsx);
    const long long part = strip_list(y / kSup, L.nsx, sx);
    const unsigned long long o = off[part];
    const unsigned n = (unsigned)(off[part + kListSub - 1] - o) + cnt[part + kListSub - 1];
    if (n == 0 || ds->overflow) return;
    const int x0 = sx * kStrip, dz = L.dims[2];
    const float h = L.h, inv_h = 1.0f / h;
    constexpr float kOffX = SIGNED ? kJXExact : kJX;
    const float ry = ((float)(L.mn[1] + y) + (SIGNED ? kJYExact : kJY)) * h;
    const int supy = y >> 2;
    if (threadIdx.x < 32) s_n[threadIdx.x] = 0;
    __syncthreads();
    auto ray_x = [&](int c) { return ((float)(L.mn[0] + x0 + c) + kOffX) * h; };
    // the triangle of corners (a, b, q) against column c's ray
    auto cross = [&](const float4& a, const float4& b, float q, int c) {
        const float rx = ray_x(c);
        const float v[9] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, q};
        // the roundings of the reference's build (nvcc's default FMA contraction):
        // a*b - c*d as fma(a, b, -(c*d)), the hit height's sum as
        // fma(d0, z2, fma(d1, z0, d2*z1))
        const float d0 = __fmaf_rn(v[3] - v[0], ry - v[1], -((v[4] - v[1]) * (rx - v[0])));
        const float d1 = __fmaf_rn(v[6] - v[3], ry - v[4], -((v[7] - v[4]) * (rx - v[3])));
        const float d2 = __fmaf_rn(v[0] - v[6], ry - v[7], -((v[1] - v[7]) * (rx - v[6])));
        const bool pos = (d0 > 0.0f && d1 > 0.0f && d2 > 0.0f);
        const bool neg = (d0 < 0.0f && d1 < 0.0f && d2 < 0.0f);
        if (!pos && !neg) return;
        const float area2 = d0 + d1 + d2;
        if (fabsf(area2) < 1e-12f) return;
        const float zh = __fmaf_rn(d0, v[8], __fmaf_rn(d1, v[2], d2 * v[5])) / area2;
        // the first z whose voxel is above: zh < (mn + z) h, which never turns false going up
        int z = (int)fminf(fmaxf(floorf(zh * inv_h) - (float)L.mn[2] + 1.0f, 0.0f), (float)dz);
        while (z > 0 && zh < (float)(L.mn[2] + z - 1) * h) --z;
        while (z < dz && !(zh < (float)(L.mn[2] + z) * h)) ++z;
        const int k = atomicAdd(&s_n[c], 1);
        if (k < kParityMaxHits) s_hit[k][c] = (unsigned)z | ((SIGNED && !neg) ? 0x80000000u : 0u);
    };
    const int last = min(kStrip, L.dims[0] - x0) - 1;  // the strip's last column
    for (unsigned e0 = 32 * warp; e0 < n; e0 += kParThreads) {
        // The row part of the candidate test is the same for every column (one row y): each
        // lane tests one list entry. The test is the negated skip condition, so a NaN bound
        // passes as before.
        unsigned tri = 0;
        bool row = false;
        int c0 = 0, c1 = -1;  // columns the entry can cross, widened by the rounding of the ray and the quotient
        if (e0 + lane < n) {
            tri = list[o + e0 + lane];
            const int4 sr = *reinterpret_cast<const int4*>(&ptt[tri].sx0);
            const float4 ab = *reinterpret_cast<const float4*>(ptt[tri].xyab);
            if (!(supy < sr.z || supy > sr.w || ry < ab.y || ry > ab.w)) {
                const float base = (float)L.mn[0] + (float)x0, qa = ab.x * inv_h, qb = ab.z * inv_h;
                const float wide = 2.0f + 1e-6f * (fabsf(qa) + fabsf(qb) + fabsf(base) + (float)x0);
                c0 = max(max(0, sr.x * kSup - x0), (int)fminf(fmaxf(floorf(qa - base - wide), -1.0f), 64.0f));
                c1 = min(min(last, sr.y * kSup + kSup - 1 - x0), (int)fminf(fmaxf(ceilf(qb - base + wide), -1.0f), 64.0f));
                row = c1 >= c0;
            }
        }
        unsigned rows = __ballot_sync(0xffffffffu, row);
        if (!rows) continue;
        const int most = __reduce_max_sync(0xffffffffu, row ? c1 - c0 + 1 : 0);
        if (most <= __popc(rows)) {  // a lane a triangle
            if (row) {
                const ParTri& p = ptt[tri];
                const float4 ab = *reinterpret_cast<const float4*>(p.xyab);
                const float4 a = *reinterpret_cast<const float4*>(p.v), b = *reinterpret_cast<const float4*>(p.v + 4);
                const float q = p.v[8];
                for (int c = c0; c <= c1; ++c) {
                    const float rx = ray_x(c);
                    if (rx < ab.x || rx > ab.z) continue;
                    cross(a, b, q, c);
                }
            }
            __syncwarp();
        } else {  // a lane a column
            const int supx = (x0 + lane) >> 2;
            const float rx = ray_x(lane);
            while (rows) {
                const int src = __ffs(rows) - 1;
                rows &= rows - 1;
                const ParTri& p = ptt[__shfl_sync(0xffffffffu, tri, src)];
                if (lane > last || supx < p.sx0 || supx > p.sx1) continue;
                const float4 ab = *reinterpret_cast<const float4*>(p.xyab);
                if (rx < ab.x || rx > ab.z) continue;
                cross(*reinterpret_cast<const float4*>(p.v), *reinterpret_cast<const float4*>(p.v + 4), p.v[8], lane);
            }
        }
    }
    __syncthreads();
    if (warp == 0) {  // a lane a column: unknown columns; the z at which the others change sides
        const int found = s_n[lane], nh = min(found, kParityMaxHits);
        bool unknown = found > kParityMaxHits;
        int m = nh;
        if (SIGNED) {
            int total = 0;
            for (int i = 0; i < nh; ++i) total += (s_hit[i][lane] >> 31) ? -1 : 1;
            unknown |= total != 0;
            if (unknown) m = 0;
            for (int i = 1; i < m; ++i) {  // by z (equal ones in any order)
                const unsigned key = s_hit[i][lane];
                int j = i - 1;
                while (j >= 0 && (s_hit[j][lane] & 0x7fffffffu) > (key & 0x7fffffffu)) {
                    s_hit[j + 1][lane] = s_hit[j][lane];
                    --j;
                }
                s_hit[j + 1][lane] = key;
            }
            int w = 0, out = 0;
            for (int i = 0; i < m; ++i) {
                const unsigned e = s_hit[i][lane];
                const int before = w;
                w += (e >> 31) ? -1 : 1;
                if ((before != 0) != (w != 0)) s_hit[out++][lane] = e & 0x7fffffffu;  // (two at one z cancel)
            }
            m = out;
        } else {
            unknown |= (nh & 1) != 0;
            if (unknown) m = 0;
        }
        s_n[lane] = m;
        const uint32_t uword = __ballot_sync(0xffffffffu, unknown), any = __ballot_sync(0xffffffffu, m > 0);
        if (lane == 0) {
            s_unknown = uword;
            s_any = any;
            if (uword) atomicAdd(&ds->unknown_columns, (unsigned long long)__popc(uword));
        }
    }
    __syncthreads();
    const uint32_t uword = s_unknown;
    const size_t zrow = (size_t)L.dims[1] * L.wx;
    const size_t wbase = (size_t)y * L.wx + sx;
    if (uword)
        for (int z = threadIdx.x; z < dz; z += kParThreads) ubits[(size_t)z * zrow + wbase] = uword;
    if (!s_any) return;
    const int m = s_n[lane];
    uint32_t carry = 0;  // the sides at the tile's first voxel
    for (int z0 = 0; z0 < dz; z0 += kZTile) {
        const int len = min(kZTile, dz - z0), per = (len + kParThreads - 1) / kParThreads;
        for (int i = threadIdx.x; i < len; i += kParThreads) s_tog[i] = 0;
        __syncthreads();
        for (int k = warp; k < m; k += kParWarps) {
            const int z = (int)s_hit[k][lane] - z0;
            if (z >= 0 && z < len) atomicXor(&s_tog[z], 1u << lane);
        }
        __syncthreads();
        const int i0 = threadIdx.x * per, i1 = min(len, i0 + per);
        uint32_t own = 0;
        for (int i = i0; i < i1; ++i) own ^= s_tog[i];
        uint32_t inc = own;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= d) inc ^= u;
        }
        if (lane == 31) s_scan[warp] = inc;
        __syncthreads();
        uint32_t word = carry ^ inc ^ own;
#pragma unroll
        for (int k = 0; k < kParWarps; ++k) {
            if (k < warp) word ^= s_scan[k];
            carry ^= s_scan[k];
        }
        for (int i = i0; i < i1; ++i) {
            word ^= s_tog[i];
            if (word) sbits[(size_t)(z0 + i) * zrow + wbase] = word;
        }
        __syncthreads();  // s_tog and s_scan are reused by the next tile
    }
}

}  // namespace

void launch_parity(const ParTri* ptt, const unsigned long long* strip_off, const unsigned* strip_count,
                   const unsigned* strip_list, const Lattice& L, uint32_t* sbits, uint32_t* ubits, DevState* ds,
                   int signed_crossings, cudaStream_t st) {
    cudaMemsetAsync(sbits, 0, (size_t)L.nwords * sizeof(uint32_t), st);
    cudaMemsetAsync(ubits, 0, (size_t)L.nwords * sizeof(uint32_t), st);
    GBSDF_COUNT_LAUNCH();
    if (signed_crossings)
        parity_kernel<1><<<(unsigned)L.nstrips, kParThreads, 0, st>>>(ptt, strip_off, strip_count, strip_list, L, sbits,
                                                                      ubits, ds);
    else
        parity_kernel<0><<<(unsigned)L.nstrips, kParThreads, 0, st>>>(ptt, strip_off, strip_count, strip_list, L, sbits,
                                                                      ubits, ds);
}

}  // namespace gbsdf
