// k_splat.cu — triangle preparation, binning (counting sorts) and the exact band splat [A] of
// the mesh-to-SDF path.
//
// The reference splats with one thread per (triangle, z-layer) and a CAS-loop
// atomicMin into the grid (cuda_rasterizer.cu:211-268). Here the clusters of eight triangles
// (k_fwn.cu) are binned to the 8^3 bricks their band can touch, and a warp takes a 4^3 octant
// of a brick: it keeps the clusters that can hold one of its voxels' nearest triangles, and
// each voxel skips clusters and triangles that lie beyond its best so far. The grid sees one
// plain store per band voxel and no atomics. The per-(voxel, triangle) predicates are the
// reference's own: the z-layer test, the clamped integer XY footprint, the AABB box test and
// d^2 <= band^2 (cuda_rasterizer.cu:225-266); they differ from d <= band only by rounding, so
// they are evaluated where d is near the band's edge, and every voxel's minimum is the
// reference's.
#include <algorithm>

#include "gwn_device.cuh"

namespace gbsdf {

namespace {

constexpr int kPrepThreads = 256;

__device__ __forceinline__ bool finite3(f3 a) { return isfinite(a.x) && isfinite(a.y) && isfinite(a.z); }

// Conservative plane test between a brick and a triangle's band: the plane
// distance from the brick centre lower-bounds the distance of every brick voxel
// to the triangle, so a brick whose centre is farther than band + half-diagonal
// (+ a relative margin far above FP32 rounding) can hold no band voxel of it.
__device__ __forceinline__ bool brick_may_hit(const float* v, const Lattice& L, int bx, int by, int bz, float bw) {
    float h = L.h;
    float cx = ((float)(L.mn[0] + bx * kBrick) + 3.5f) * h;
    float cy = ((float)(L.mn[1] + by * kBrick) + 3.5f) * h;
    float cz = ((float)(L.mn[2] + bz * kBrick) + 3.5f) * h;
    float ex = v[3] - v[0], ey = v[4] - v[1], ez = v[5] - v[2];
    float fx = v[6] - v[0], fy = v[7] - v[1], fz = v[8] - v[2];
    float nx = ey * fz - ez * fy, ny = ez * fx - ex * fz, nz = ex * fy - ey * fx;
    float nn = nx * nx + ny * ny + nz * nz;
    if (!(nn > 1e-30f)) return true;
    float dist = fabsf(nx * (cx - v[0]) + ny * (cy - v[1]) + nz * (cz - v[2])) * rsqrtf(nn);
    float reach = bw + 6.0621778f * h * 1.0001f + 1e-3f * (bw + 7.0f * h) + 1e-4f * fabsf(dist);
    return dist <= reach;
}

// Checks the coordinates and writes the parity pass's records and strip counts. Bound by the
// queues at the counters: one list per supercell row in parts, the totals through one atomic a
// block, and no FP64 divisions where the coordinates are plainly in range, 30k triangles on
// 150^3 56 -> 7.5 us.
__global__ void __launch_bounds__(kPrepThreads) prep_kernel(const float* __restrict__ tris12, long long T, Lattice L,
                                                            ParTri* __restrict__ pto,
                                                            unsigned* __restrict__ strip_count, DevState* ds) {
    __shared__ unsigned long long s_sum[2];
    if (threadIdx.x < 2) s_sum[threadIdx.x] = 0;
    __syncthreads();
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long csr = 0, pairs = 0;
    if (t < T) {
        float r[9];
        for (int k = 0; k < 9; ++k) r[k] = __ldg(tris12 + 12 * t + k);
        const f3 v0 = mk(r[0], r[1], r[2]), v1 = mk(r[3], r[4], r[5]), v2 = mk(r[6], r[7], r[8]);
        const float h = L.h;
        ParTri p;
        for (int k = 0; k < 9; ++k) p.v[k] = r[k];
        p.sx0 = 0;
        p.sx1 = -1;
        p.sy0 = 0;
        p.sy1 = -1;
        p.pad[0] = p.pad[1] = p.pad[2] = 0;
        // Bounds validation before any float->int grid arithmetic, |coordinate / h| < 1e9 in FP64;
        // coordinates well inside it need no division.
        bool ok = finite3(v0) && finite3(v1) && finite3(v2);
        if (ok) {
            const double lim = 1.0e9, hd = (double)h;
            const float inside = (float)(0.999 * lim * hd);
            for (int k = 0; k < 9; ++k)
                if (!(fabsf(r[k]) < inside) && !(fabs((double)r[k] / hd) < lim)) ok = false;
        }
        for (int k = 0; k < 4; ++k) p.xyab[k] = 0.0f;
        if (!ok) atomicAdd(&ds->invalid_tris, 1ull);
        if (ok) {
            // the reference's host CSR coverage, cuda_rasterizer.cu:837-860
            float minx = fminf(v0.x, fminf(v1.x, v2.x)), maxx = fmaxf(v0.x, fmaxf(v1.x, v2.x));
            float miny = fminf(v0.y, fminf(v1.y, v2.y)), maxy = fmaxf(v0.y, fmaxf(v1.y, v2.y));
            p.xyab[0] = minx;
            p.xyab[1] = miny;
            p.xyab[2] = maxx;
            p.xyab[3] = maxy;
            int sdx = (L.dims[0] + kSup - 1) / kSup, sdy = (L.dims[1] + kSup - 1) / kSup;
            int cx0 = (int)floorf(minx / h) - L.mn[0] - 1;
            int cx1 = (int)ceilf(maxx / h) - L.mn[0] + 1;
            int cy0 = (int)floorf(miny / h) - L.mn[1] - 1;
            int cy1 = (int)ceilf(maxy / h) - L.mn[1] + 1;
            int sx0 = max(0, cx0 / kSup), sx1 = min(sdx - 1, cx1 / kSup);
            int sy0 = max(0, cy0 / kSup), sy1 = min(sdy - 1, cy1 / kSup);
            p.sx0 = sx0;
            p.sx1 = sx1;
            p.sy0 = sy0;
            p.sy1 = sy1;
            if (sx1 >= sx0 && sy1 >= sy0) {
                csr = (unsigned long long)(sx1 - sx0 + 1) * (unsigned long long)(sy1 - sy0 + 1);
                const int xa = sx0 * kSup / kStrip, xb = min(L.dims[0] - 1, sx1 * kSup + kSup - 1) / kStrip;
                for (int y = sy0; y <= sy1; ++y)
                    for (int sx = xa; sx <= xb; ++sx)
                        atomicAdd(&strip_count[strip_list(y, L.nsx, sx) + threadIdx.x % kListSub], 1u);
                pairs = (unsigned long long)(sy1 - sy0 + 1) * (unsigned long long)(xb - xa + 1);
            }
        }
        pto[t] = p;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        csr += __shfl_down_sync(0xffffffffu, csr, o);
        pairs += __shfl_down_sync(0xffffffffu, pairs, o);
    }
    if ((threadIdx.x & 31) == 0 && csr) {
        atomicAdd(&s_sum[0], csr);
        atomicAdd(&s_sum[1], pairs);
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_sum[0]) {
        atomicAdd(&ds->csr_entries, s_sum[0]);
        atomicAdd(&ds->strip_pairs, s_sum[1]);
    }
}

// The strip lists of the parity pass. Bound by the latency of the atomics that hand out the
// slots, four in flight together; with lists per row and one counter each, 30k triangles on 150^3
// took 54 us, now 5.9.
__global__ void __launch_bounds__(kPrepThreads) strip_fill_kernel(
    const ParTri* __restrict__ ptt, long long T, Lattice L, const unsigned long long* __restrict__ strip_off,
    unsigned* __restrict__ strip_cur, unsigned* __restrict__ list, DevState* ds, unsigned long long cap_b,
    unsigned long long cap_s) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T) return;
    if (ds && (ds->brick_pairs > cap_b || ds->strip_pairs > cap_s)) {  // planned lists too small
        if (t == 0) ds->overflow = 1;
        return;
    }
    const int4 sr = *reinterpret_cast<const int4*>(&ptt[t].sx0);
    if (sr.y >= sr.x && sr.w >= sr.z) {
        const int xa = sr.x * kSup / kStrip, xb = min(L.dims[0] - 1, sr.y * kSup + kSup - 1) / kStrip;
        for (int sx = xa; sx <= xb; ++sx)
            for (int y = sr.z; y <= sr.w; y += 4) {
                unsigned long long at[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const long long b = strip_list(y + k, L.nsx, sx) + threadIdx.x % kListSub;
                    if (y + k <= sr.w) at[k] = strip_off[b] + atomicAdd(&strip_cur[b], 1u);
                }
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (y + k <= sr.w) list[at[k]] = (unsigned)t;
            }
    }
}

// Counts (list null) or fills the bricks' cluster lists: one warp per (cluster, slice), the lanes
// taking the bricks that the cluster's box widened by the band covers. A brick takes the
// cluster when one of its triangles' spheres and planes comes within the band of the brick's
// points (widened by far more than the rounding). A run of triangles that jumps (from one part of
// the mesh to another) has a wide box of mostly empty bricks: its triangles' boxes are
// taken one by one, a brick going to the first of them that meets it (the 860 x 860 x 880
// mug's widest cluster alone held its warp for 2.4 ms).
constexpr long long kWideBox = 2048;  // bricks
__global__ void __launch_bounds__(256) brick_bin_kernel(FwnView f, Lattice L, int slices, unsigned* __restrict__ count,
                                                        const unsigned long long* __restrict__ off,
                                                        unsigned* __restrict__ list, DevState* ds,
                                                        unsigned long long cap_b, unsigned long long cap_s) {
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const long long k = w / slices;
    const int sl = (int)(w - k * slices);
    if (k >= f.n[0]) return;
    if (list && (ds->brick_pairs > cap_b || ds->strip_pairs > cap_s)) return;  // strip_fill_kernel reports it
    const float h = L.h, bw = (float)kBandVoxels * h;
    const float4 blo = __ldg(&f.box[0][2 * k]), bhi = __ldg(&f.box[0][2 * k + 1]);
    const float slop = 4e-6f * (fabsf(blo.x) + fabsf(blo.y) + fabsf(blo.z) + fabsf(bhi.x) + fabsf(bhi.y) + fabsf(bhi.z)) +
                       1e-4f * bw;
    const float reach = bw + 6.0622f * h + slop + 1e-6f * h * (float)(L.dims[0] + L.dims[1] + L.dims[2]);
    const long long t0 = k * kFwnLeaf;
    const int m = (int)min((long long)kFwnLeaf, f.T - t0);
    int b0[3], nb[3];
    auto range = [&](const f3& lo, const f3& hi) -> long long {
        const float l3[3] = {lo.x, lo.y, lo.z}, h3[3] = {hi.x, hi.y, hi.z};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            // a brick holds points (mn + 8 b .. mn + 8 b + 7) h
            const float u = floorf((l3[a] - bw - slop) / h - (float)L.mn[a] - 8.0f) * 0.125f;
            const float v = ceilf((h3[a] + bw + slop) / h - (float)L.mn[a] + 1.0f) * 0.125f;
            const int i0 = (int)fminf(fmaxf(floorf(u), 0.0f), (float)(L.nb[a] - 1));
            const int i1 = (int)fminf(fmaxf(floorf(v), -1.0f), (float)(L.nb[a] - 1));
            b0[a] = i0;
            nb[a] = max(i1 - i0 + 1, 0);
        }
        return (long long)nb[0] * nb[1] * nb[2];
    };
    auto hits = [&](int t, const f3& c) {
        const float4* o = f.leaf + 5 * (t0 + t);
        const float4 g = __ldg(o), d = __ldg(o + 1);
        const float dx = g.x - c.x, dy = g.y - c.y, dz = g.z - c.z, r = reach + g.w;
        const float s = __fmaf_rn(d.z, dz, __fmaf_rn(d.y, dy, d.x * dx));
        return !(__fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx)) > r * r ||
                 s * s > reach * reach * 1.001f * __ldg(&o[4].y));
    };
    unsigned pairs = 0;
    // the bricks of the current range; `first`: the triangle they are taken for (-1: any)
    auto bricks = [&](long long n, int first) {
        for (long long i = (long long)sl * 32 + lane; i < n; i += (long long)slices * 32) {
            const int bx = b0[0] + (int)(i % nb[0]), by = b0[1] + (int)(i / nb[0] % nb[1]),
                      bz = b0[2] + (int)(i / ((long long)nb[0] * nb[1]));
            const f3 c = mk(lattice_mid(L.mn[0], bx * 8, 3.5f, h), lattice_mid(L.mn[1], by * 8, 3.5f, h),
                            lattice_mid(L.mn[2], bz * 8, 3.5f, h));
            if (box_dist_sq(f.box[0] + 2 * k, c) > reach * reach) continue;
            bool hit;
            if (first < 0) {
                hit = false;
                for (int t = 0; t < m && !hit; ++t) hit = hits(t, c);
            } else {
                hit = hits(first, c);
                for (int t = 0; t < first && hit; ++t) hit = !hits(t, c);
            }
            if (!hit) continue;
            const long long b = ((long long)bz * L.nb[1] + by) * L.nb[0] + bx;
            const unsigned pos = atomicAdd(&count[b], 1u);
            if (list) list[off[b] + pos] = (unsigned)k;
            ++pairs;
        }
    };
    const long long n = range(mk(blo.x, blo.y, blo.z), mk(bhi.x, bhi.y, bhi.z));
    if (n <= kWideBox) {
        bricks(n, -1);
    } else {
        for (int t = 0; t < m; ++t) {  // a sphere's box holds all bricks that hits() lets pass for t
            const float4 g = __ldg(f.leaf + 5 * (t0 + t));
            const float r = g.w + 6.1f * h;
            bricks(range(mk(g.x - r, g.y - r, g.z - r), mk(g.x + r, g.y + r, g.z + r)), t);
        }
    }
    if (!list) {
        const unsigned pw = __reduce_add_sync(0xffffffffu, pairs);
        if (lane == 0 && pw) atomicAdd(&ds->brick_pairs, (unsigned long long)pw);
    }
}

// Triangles per brick (a feature of the sign-risk model): those whose clamped footprint and plane
// can put a band voxel into the brick.
__global__ void __launch_bounds__(kPrepThreads) brick_tris_kernel(const float* __restrict__ tris12, long long T,
                                                                  Lattice L, unsigned* __restrict__ count) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T) return;
    const float* r = tris12 + 12 * t;
    float v[9];
    for (int k = 0; k < 9; ++k) v[k] = r[k];
    const float h = L.h, bw = (float)kBandVoxels * h;
    int a0[3], a1[3];
    for (int a = 0; a < 3; ++a) {
        const float lo = fminf(v[a], fminf(v[3 + a], v[6 + a])), hi = fmaxf(v[a], fmaxf(v[3 + a], v[6 + a]));
        if (a < 2) {  // splat footprint, cuda_rasterizer.cu:225-248
            a0[a] = max((int)ceilf((lo - bw) / h) - L.mn[a], 0);
            a1[a] = min((int)floorf((hi + bw) / h) - L.mn[a], L.dims[a] - 1);
        } else {  // conservative z range
            a0[a] = max((int)floorf((lo - bw) / h) - L.mn[a] - 1, 0);
            a1[a] = min((int)ceilf((hi + bw) / h) - L.mn[a] + 1, L.dims[a] - 1);
        }
        if (a1[a] < a0[a]) return;
    }
    for (int bz = a0[2] / kBrick; bz <= a1[2] / kBrick; ++bz)
        for (int by = a0[1] / kBrick; by <= a1[1] / kBrick; ++by)
            for (int bx = a0[0] / kBrick; bx <= a1[0] / kBrick; ++bx)
                if (brick_may_hit(v, L, bx, by, bz, bw))
                    atomicAdd(&count[((long long)bz * L.nb[1] + by) * L.nb[0] + bx], 1u);
}

// ---- exclusive scan (unsigned -> unsigned long long), three-phase, recursive on the host
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;  // 2048

template <typename Tin>
__global__ void __launch_bounds__(kScanThreads) scan_tile_kernel(const Tin* __restrict__ in,
                                                                 unsigned long long* __restrict__ out, long long n,
                                                                 unsigned long long* __restrict__ tile_sums) {
    __shared__ unsigned long long warp_tot[kScanThreads / 32];
    long long base = (long long)blockIdx.x * kScanTile + (long long)threadIdx.x * kScanItems;
    unsigned long long v[kScanItems];
    unsigned long long run = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        long long k = base + i;
        unsigned long long x = (k < n) ? (unsigned long long)in[k] : 0ull;
        v[i] = run;
        run += x;
    }
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned long long y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    unsigned long long wpre = 0;
    for (int w = 0; w < warp; ++w) wpre += warp_tot[w];
    unsigned long long excl = wpre + incl - run;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        long long k = base + i;
        if (k < n) out[k] = v[i] + excl;
    }
    if (threadIdx.x == kScanThreads - 1) tile_sums[blockIdx.x] = wpre + incl;
}

__global__ void scan_add_kernel(unsigned long long* __restrict__ out, long long n,
                                const unsigned long long* __restrict__ tile_off) {
    long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) out[k] += tile_off[k / kScanTile];
}

void scan_rec(const void* in, bool in_is_u64, unsigned long long* out, long long n, unsigned long long* tmp,
              cudaStream_t st) {
    long long tiles = (n + kScanTile - 1) / kScanTile;
    unsigned long long* sums = tmp;
    unsigned long long* rest = tmp + tiles;
    GBSDF_COUNT_LAUNCH();
    if (in_is_u64)
        scan_tile_kernel<unsigned long long><<<(unsigned)tiles, kScanThreads, 0, st>>>(
            (const unsigned long long*)in, out, n, sums);
    else
        scan_tile_kernel<unsigned><<<(unsigned)tiles, kScanThreads, 0, st>>>((const unsigned*)in, out, n, sums);
    if (tiles > 1) {
        unsigned long long* sums_scanned = rest;
        scan_rec(sums, true, sums_scanned, tiles, rest + tiles, st);
        GBSDF_COUNT_LAUNCH();
        scan_add_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(out, n, sums_scanned);
    }
}

constexpr int kSplatThreads = 256;
constexpr int kSplatCap = 512;  // clusters kept per octant before its voxels take them

// The bricks with binned clusters: those of more than `dense_cut` triangles (eight to a cluster)
// from the back of `active` (ds->dense_bricks of them, taken first), the others from the front
// (ds->active_bricks).
__global__ void active_bricks_kernel(const unsigned* __restrict__ cnt, long long nb, unsigned* __restrict__ active,
                                     DevState* ds, unsigned dense_cut) {
    const long long b = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned n = (b < nb) ? cnt[b] : 0u;
    const bool dense = n > dense_cut / kFwnLeaf, sparse = n > 0 && !dense;
    const unsigned ms = __ballot_sync(0xffffffffu, sparse), md = __ballot_sync(0xffffffffu, dense);
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    unsigned long long bs = 0, bd = 0;
    if (lane == 0) {
        if (ms) bs = atomicAdd(&ds->active_bricks, (unsigned long long)__popc(ms));
        if (md) bd = atomicAdd(&ds->dense_bricks, (unsigned long long)__popc(md));
    }
    bs = __shfl_sync(0xffffffffu, bs, 0);
    bd = __shfl_sync(0xffffffffu, bd, 0);
    if (sparse) active[bs + __popc(ms & below)] = (unsigned)b;
    if (dense) active[nb - 1 - (long long)(bd + __popc(md & below))] = (unsigned)b;
}

__global__ void fill_kernel(float4* __restrict__ g4, long long n4, float value) {
    long long stride = (long long)gridDim.x * blockDim.x;
    float4 v = make_float4(value, value, value, value);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += stride) g4[i] = v;
}
__global__ void fill_tail_kernel(float* __restrict__ g, long long from, long long n, float value) {
    long long i = from + threadIdx.x;
    if (i < n) g[i] = value;
}


// The reference's predicates of voxel (x, y, z) at p for a triangle (cuda_rasterizer.cu:225-266).
__device__ __forceinline__ bool splat_admits(const float4* __restrict__ leaf, const Lattice& L, int x, int y,
                                             const f3& p, float bw, float band_sq) {
    const float4 a = __ldg(leaf + 2), b = __ldg(leaf + 3);
    const float w = __ldg(&leaf[4].x), h = L.h;
    const float tx0 = fminf(a.x, fminf(a.w, b.z)), tx1 = fmaxf(a.x, fmaxf(a.w, b.z));
    const float ty0 = fminf(a.y, fminf(b.x, b.w)), ty1 = fmaxf(a.y, fmaxf(b.x, b.w));
    const float tz0 = fminf(a.z, fminf(b.y, w)), tz1 = fmaxf(a.z, fmaxf(b.y, w));
    if (x < (int)ceilf((tx0 - bw) / h) - L.mn[0] || x > (int)floorf((tx1 + bw) / h) - L.mn[0] ||
        y < (int)ceilf((ty0 - bw) / h) - L.mn[1] || y > (int)floorf((ty1 + bw) / h) - L.mn[1])
        return false;
    if (p.z < tz0 - bw || p.z > tz1 + bw) return false;
    const float dx = (p.x < tx0) ? (tx0 - p.x) : ((p.x > tx1) ? (p.x - tx1) : 0.0f);
    const float dy = (p.y < ty0) ? (ty0 - p.y) : ((p.y > ty1) ? (p.y - ty1) : 0.0f);
    const float dz = (p.z < tz0) ? (tz0 - p.z) : ((p.z > tz1) ? (p.z - tz1) : 0.0f);
    return dx * dx + dy * dy + dz * dz <= band_sq;
}

// One warp per octant (4^3 voxels, two a lane), the eight warps of a CTA taking one brick; bricks
// of many clusters first. With u the octant centre's distance to the triangles of the cluster
// whose box is nearest to it, no voxel of the octant is farther than u + rho from the mesh, and
// only triangles whose box and plane come within min(u + 2 rho, band + rho) of the centre can
// hold a voxel's nearest point in the band. Those are listed as clusters with a mask of their
// triangles (the lanes testing 32 clusters, then the near ones' triangles 32 at a time), and
// each voxel takes the listed ones whose boxes, the cluster's and then the triangle's, come
// within its best so far; the tests are widened by the rounding of both sides. Fine meshes are
// pruned by the cluster boxes, coarse ones by the masks and the triangle boxes. Bound by the
// FP32 work of the box tests and exact distances. Against one exact distance per (voxel,
// triangle binned to its brick), splat stage: 860 x 860 x 880 mug 9.8 -> 7.2 ms, 640^3 blob
// 21.4 -> 9.4, 512^3 vessel tree 10.2 -> 4.0, 128^3 mug 1.0 -> 0.39; summed over the kernels of
// a 16-mesh batch (2k to 150k triangles on 64^3 to 224^3) 27 -> 13.6 ms.
__global__ void __launch_bounds__(kSplatThreads, 4) splat_kernel(FwnView f, const unsigned long long* __restrict__ off,
                                                                 const unsigned* __restrict__ cnt,
                                                                 const unsigned* __restrict__ list,
                                                                 const unsigned* __restrict__ active, Lattice L,
                                                                 float* __restrict__ dist, DevState* ds) {
    __shared__ unsigned s_id[kSplatThreads / 32][kSplatCap];
    __shared__ unsigned char s_mask[kSplatThreads / 32][kSplatCap];
    if (ds->overflow) return;
    const long long nd = (long long)ds->dense_bricks, na = nd + (long long)ds->active_bricks;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float h = L.h, bw = (float)kBandVoxels * h, band_sq = bw * bw;
    const float inf = __int_as_float(0x7f800000);
    unsigned evals = 0, found = 0;
    for (long long i = blockIdx.x; i < na; i += gridDim.x) {
        const unsigned b = active[i < nd ? L.nbricks - 1 - i : i - nd];
        const int bx = (int)(b % (unsigned)L.nb[0]), by = (int)((b / (unsigned)L.nb[0]) % (unsigned)L.nb[1]),
                  bz = (int)(b / ((unsigned)L.nb[0] * (unsigned)L.nb[1]));
        const int x0 = bx * kBrick + (warp & 1) * 4, y0 = by * kBrick + (warp & 2) * 2, z0 = bz * kBrick + (warp & 4);
        if (x0 >= L.dims[0] || y0 >= L.dims[1] || z0 >= L.dims[2]) continue;
        const f3 oc = mk(lattice_mid(L.mn[0], x0, 1.5f, h), lattice_mid(L.mn[1], y0, 1.5f, h),
                         lattice_mid(L.mn[2], z0, 1.5f, h));
        const float slop = 2e-6f * (fabsf(oc.x) + fabsf(oc.y) + fabsf(oc.z) + bw);
        const float rho = 2.5981f * h * 1.0002f + slop;
        const float edge = fmaxf(bw * 0.9999f - 4.0f * slop, 0.0f), edge_sq = edge * edge;
        const unsigned* mine = list + off[b];
        const int n = (int)cnt[b];
        // the cluster nearest to the centre
        float bd = inf;
        int bk = 0x7fffffff;
        for (int e = lane; e < n; e += 32) {
            const int k = (int)mine[e];
            const float d = box_dist_sq(f.box[0] + 2 * (size_t)k, oc);
            if (d < bd || bk == 0x7fffffff) {
                bd = d;
                bk = k;
            }
        }
        const int kn = warp_argmin(bd, bk);
        const float out = (bw + rho) * 1.00002f + slop;  // beyond it: no band voxel
        if (box_dist_sq(f.box[0] + 2 * (size_t)kn, oc) > out * out) continue;
        const long long tn = (long long)kn * kFwnLeaf + (lane & 7);
        float u = tn < f.T ? sqrtf(leaf_dist_sq(f.leaf + 5 * tn, oc)) : inf;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) u = fminf(u, __shfl_xor_sync(0xffffffffu, u, o));
        int x[2], y[2], z[2];
        f3 p[2];
        float best[2], lim_sq[2], reach_sq;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int v = morton_voxel(k * 32 + lane);
            x[k] = x0 + (v & 7);
            y[k] = y0 + ((v >> 3) & 7);
            z[k] = z0 + (v >> 6);
            p[k] = lattice_point(L.mn[0], L.mn[1], L.mn[2], x[k], y[k], z[k], h);
        }
        auto take = [&](int m) {  // the listed clusters, voxel by voxel
            __syncwarp();
            for (int e = 0; e < m; ++e) {
                const size_t k0 = s_id[warp][e];
                unsigned tris = s_mask[warp][e];
                const bool near0 = !(box_dist_sq(f.box[0] + 2 * k0, p[0]) > lim_sq[0]),
                           near1 = !(box_dist_sq(f.box[0] + 2 * k0, p[1]) > lim_sq[1]);
                if (!__any_sync(0xffffffffu, near0 || near1)) continue;
                while (tris) {
                    const float4* o = f.leaf + 5 * (k0 * kFwnLeaf + (__ffs(tris) - 1));
                    tris &= tris - 1u;
                    const float4 a = __ldg(o + 2), c = __ldg(o + 3);
                    const float w = __ldg(&o[4].x);
                    const f3 lo = mk(min3f(a.x, a.w, c.z), min3f(a.y, c.x, c.w), min3f(a.z, c.y, w)),
                             hi = mk(max3f(a.x, a.w, c.z), max3f(a.y, c.x, c.w), max3f(a.z, c.y, w));
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const float dx = max3f(lo.x - p[k].x, p[k].x - hi.x, 0.0f),
                                    dy = max3f(lo.y - p[k].y, p[k].y - hi.y, 0.0f),
                                    dz = max3f(lo.z - p[k].z, p[k].z - hi.z, 0.0f);
                        if (__fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx)) > lim_sq[k]) continue;
                        const float d2 = ptd_sq(p[k], mk(a.x, a.y, a.z), mk(a.w, c.x, c.y), mk(c.z, c.w, w));
                        ++evals;
                        if (d2 < best[k] && d2 <= band_sq &&
                            (d2 <= edge_sq || splat_admits(o, L, x[k], y[k], p[k], bw, band_sq))) {
                            best[k] = d2;
                            const float lim = sqrtf(d2) * 1.00002f + slop;
                            lim_sq[k] = fminf(lim_sq[k], lim * lim);
                        }
                    }
                }
            }
            __syncwarp();
        };
        int nt = 0;
        auto list_tri = [&](long long t, bool on) {  // lane's triangle t of a group of eight
            if (on) {
                const float4* o = f.leaf + 5 * t;
                const float4 d = __ldg(o + 1), a = __ldg(o + 2), c = __ldg(o + 3);
                const float2 w = __ldg(reinterpret_cast<const float2*>(o + 4));
                const float dx = max3f(min3f(a.x, a.w, c.z) - oc.x, oc.x - max3f(a.x, a.w, c.z), 0.0f),
                            dy = max3f(min3f(a.y, c.x, c.w) - oc.y, oc.y - max3f(a.y, c.x, c.w), 0.0f),
                            dz = max3f(min3f(a.z, c.y, w.x) - oc.z, oc.z - max3f(a.z, c.y, w.x), 0.0f);
                const float s = __fmaf_rn(d.z, a.z - oc.z, __fmaf_rn(d.y, a.y - oc.y, d.x * (a.x - oc.x)));
                on = !(__fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx)) > reach_sq || s * s > w.y * 1.0001f * reach_sq);
            }
            const unsigned mask = (__ballot_sync(0xffffffffu, on) >> (lane & 24)) & 0xffu;
            const bool lead = (lane & 7) == 0 && mask;
            const unsigned bal = __ballot_sync(0xffffffffu, lead);
            if (lead) {
                const int slot = nt + __popc(bal & ((1u << lane) - 1u));
                s_id[warp][slot] = (unsigned)(t / kFwnLeaf);
                s_mask[warp][slot] = (unsigned char)mask;
            }
            nt += __popc(bal);
            if (nt > kSplatCap - 4) {
                take(nt);
                nt = 0;
            }
        };
        // The limits hold for the distances as computed, unless the triangle they come from is one
        // without area (it has no distance for some points) or a sliver: a voxel left above its
        // limit shows it, and the octant is taken again with the band as its only limit.
        for (;;) {
            const float reach = fminf((u + 2.0f * rho) * 1.00002f + slop, out);
            const float lim = fminf(u + rho, bw) * 1.00002f + slop, held = lim * lim;
            reach_sq = reach * reach;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                best[k] = inf;
                lim_sq[k] = held;
            }
            list_tri(tn, lane < 8 && tn < f.T);  // the nearest cluster first: it sets the voxels' limits
            for (int base = 0; base < n; base += 32) {
                const int e = base + lane;
                const unsigned k = e < n ? mine[e] : 0u;
                unsigned near = __ballot_sync(0xffffffffu, e < n && k != (unsigned)kn &&
                                                               !(box_dist_sq(f.box[0] + 2 * (size_t)k, oc) > reach_sq));
                while (near) {  // four clusters of eight triangles at a time
                    int src[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        src[q] = __ffs(near) - 1;
                        near &= near - 1u;
                    }
                    const int sl = lane < 8 ? src[0] : lane < 16 ? src[1] : lane < 24 ? src[2] : src[3];
                    const long long t = (long long)__shfl_sync(0xffffffffu, k, sl & 31) * kFwnLeaf + (lane & 7);
                    list_tri(t, sl >= 0 && t < f.T);
                }
            }
            take(nt);
            nt = 0;
            if (!(u + rho < bw) || !__any_sync(0xffffffffu, fmaxf(best[0], best[1]) > held)) break;
            u = inf;
        }
#pragma unroll
        for (int k = 0; k < 2; ++k)
            if (best[k] != inf && x[k] < L.dims[0] && y[k] < L.dims[1] && z[k] < L.dims[2]) {
                dist[((size_t)z[k] * L.dims[1] + y[k]) * L.dims[0] + x[k]] = sqrtf(best[k]);
                ++found;
            }
    }
    const unsigned fw = __reduce_add_sync(0xffffffffu, found), ew = __reduce_add_sync(0xffffffffu, evals);
    if (lane == 0) {
        if (fw) atomicAdd(&ds->band_voxels, (unsigned long long)fw);
        if (ew) atomicAdd(&ds->splat_evals, (unsigned long long)ew);
    }
}

// One warp per sample: the lanes split the triangles of the brick's clusters that come near
// the splat's distance, find the FP32 minimum (the splat's arithmetic), then evaluate in FP64
// only the triangles whose FP32 squared distance lies within 0.1% (plus 1e-6 h^2) of it -- the
// FP64 minimum is among them.
constexpr int kBandErrWarps = 4;
__global__ void __launch_bounds__(kBandErrWarps * 32)
    band_error_kernel(FwnView f, const unsigned long long* __restrict__ boff, const unsigned* __restrict__ bcount,
                      const unsigned* __restrict__ blist, Lattice L, const float* __restrict__ dist, DevState* ds) {
    const long long k = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (k >= kBandErrSamples || ds->overflow) return;
    // one voxel per stratum of N / kBandErrSamples, at a golden-ratio offset within it (an
    // offset common to all strata would put every sample in one x column when the stratum
    // is a multiple of the row length, as at 1024^3)
    const double off = (double)k * 0.6180339887498949 - floor((double)k * 0.6180339887498949);
    const long long v = (long long)(((double)k + off) * (double)L.N / (double)kBandErrSamples);
    if (v >= L.N) return;
    const float d = dist[v];
    if (!(d <= (float)kBandVoxels * L.h)) return;
    const int x = (int)(v % L.dims[0]);
    const long long r = v / L.dims[0];
    const int y = (int)(r % L.dims[1]), z = (int)(r / L.dims[1]);
    const long long b = ((long long)(z / kBrick) * L.nb[1] + y / kBrick) * L.nb[0] + x / kBrick;
    const f3 p = lattice_point(L.mn[0], L.mn[1], L.mn[2], x, y, z, L.h);
    const unsigned* mine = blist + boff[b];
    const unsigned n = bcount[b];
    // no triangle of a farther cluster has an FP32 squared distance within 0.1% of the minimum
    const float far = d * 1.002f + 2e-3f * L.h + 4e-6f * (fabsf(p.x) + fabsf(p.y) + fabsf(p.z) + d), far_sq = far * far;
    float m32 = 3.0e38f;
    double best = 1e300;
    for (int pass = 0; pass < 2; ++pass) {
        const float lim = m32 + m32 * 1e-3f + 1e-6f * L.h * L.h;
        for (unsigned base = 0; base < n; base += 32) {
            const unsigned e = base + lane;
            const unsigned k0 = e < n ? mine[e] : 0u;
            unsigned near = __ballot_sync(0xffffffffu, e < n && !(box_dist_sq(f.box[0] + 2 * (size_t)k0, p) > far_sq));
            while (near) {  // four clusters of eight triangles at a time
                int src[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    src[q] = __ffs(near) - 1;
                    near &= near - 1u;
                }
                const int s = src[0] < 0 ? -1 : (lane < 8 ? src[0] : lane < 16 ? src[1] : lane < 24 ? src[2] : src[3]);
                const long long t = (long long)__shfl_sync(0xffffffffu, k0, s & 31) * kFwnLeaf + (lane & 7);
                if (s < 0 || t >= f.T) continue;
                const float4* o = f.leaf + 5 * t;
                const float d2 = leaf_dist_sq(o, p);
                if (pass == 0) {
                    m32 = fminf(m32, d2);
                } else if (d2 <= lim) {
                    const float4 a = __ldg(o + 2), c = __ldg(o + 3);
                    const float v9[9] = {a.x, a.y, a.z, a.w, c.x, c.y, c.z, c.w, __ldg(&o[4].x)};
                    best = fmin(best, ptd_sq_f64(p.x, p.y, p.z, v9));
                }
            }
            __syncwarp();
        }
        for (int o = 16; o > 0; o >>= 1) m32 = fminf(m32, __shfl_xor_sync(0xffffffffu, m32, o));
    }
    for (int o = 16; o > 0; o >>= 1) best = fmin(best, __shfl_xor_sync(0xffffffffu, best, o));
    if (lane == 0) {
        const double err = fabs(sqrt(best) - (double)d) / (double)L.h;
        atomicMax(&ds->band_err_bits, (unsigned long long)__double_as_longlong(err));
        atomicAdd(&ds->band_err_n, 1ull);
    }
}

// warps per cluster: few clusters are large ones, whose bricks several warps share
int bin_slices(const Fwn& f) { return (int)std::max<long long>(1, std::min<long long>(64, 152ll * 64 / f.n[0])); }

}  // namespace

void launch_prep(const float* tris12, long long T, const Lattice& L, ParTri* pto, unsigned* strip_count, DevState* ds,
                 cudaStream_t st) {
    if (T <= 0) return;
    GBSDF_COUNT_LAUNCH();
    prep_kernel<<<(unsigned)((T + kPrepThreads - 1) / kPrepThreads), kPrepThreads, 0, st>>>(tris12, T, L, pto,
                                                                                          strip_count, ds);
}

long long scan_tmp_elems(long long n) {
    long long total = 0;
    while (n > 1) {
        long long tiles = (n + kScanTile - 1) / kScanTile;
        total += 2 * tiles;
        n = tiles;
    }
    return total + 2;
}

void launch_exclusive_scan(const unsigned* in, unsigned long long* out, long long n, unsigned long long* tmp,
                           long long tmp_elems, cudaStream_t st) {
    (void)tmp_elems;
    if (n <= 0) return;
    scan_rec(in, false, out, n, tmp, st);
}

void launch_strip_fill(const ParTri* ptt, long long T, const Lattice& L, const unsigned long long* strip_off,
                       unsigned* strip_cur, unsigned* strip_list, cudaStream_t st, DevState* ds,
                       unsigned long long cap_b, unsigned long long cap_s) {
    if (T <= 0) return;
    GBSDF_COUNT_LAUNCH();
    strip_fill_kernel<<<(unsigned)((T + kPrepThreads - 1) / kPrepThreads), kPrepThreads, 0, st>>>(
        ptt, T, L, strip_off, strip_cur, strip_list, ds, cap_b, cap_s);
}

void launch_brick_bins(const Fwn& f, long long T, const Lattice& L, unsigned* count, const unsigned long long* off,
                       unsigned* list, DevState* ds, cudaStream_t st, unsigned long long cap_b,
                       unsigned long long cap_s) {
    const int slices = bin_slices(f);
    GBSDF_COUNT_LAUNCH();
    brick_bin_kernel<<<(unsigned)((f.n[0] * slices + 7) / 8), 256, 0, st>>>(view_of(f, T), L, slices, count, off, list,
                                                                           ds, cap_b, cap_s);
}

void launch_brick_tris(const float* tris12, long long T, const Lattice& L, unsigned* count, cudaStream_t st) {
    GBSDF_COUNT_LAUNCH();
    brick_tris_kernel<<<(unsigned)((T + kPrepThreads - 1) / kPrepThreads), kPrepThreads, 0, st>>>(tris12, T, L, count);
}

void launch_active_bricks(const unsigned* brick_count, long long nbricks, unsigned* active, DevState* ds,
                          cudaStream_t st, unsigned dense_cut) {
    GBSDF_COUNT_LAUNCH();
    active_bricks_kernel<<<(unsigned)((nbricks + 255) / 256), 256, 0, st>>>(brick_count, nbricks, active, ds,
                                                                            dense_cut);
}

void launch_fill(float* g, long long n, float value, cudaStream_t st) {
    long long n4 = n / 4;
    if (n4 > 0) {
        long long blocks = std::min<long long>((n4 + 255) / 256, 152LL * 32);
        GBSDF_COUNT_LAUNCH();
        fill_kernel<<<(unsigned)blocks, 256, 0, st>>>(reinterpret_cast<float4*>(g), n4, value);
    }
    if (n4 * 4 < n) { GBSDF_COUNT_LAUNCH(); fill_tail_kernel<<<1, 4, 0, st>>>(g, n4 * 4, n, value); }
}

void launch_band_error(const Fwn& f, long long T, const unsigned long long* brick_off, const unsigned* brick_count,
                       const unsigned* brick_list, const Lattice& L, const float* dist, DevState* ds, cudaStream_t st) {
    if (L.N <= 0) return;
    GBSDF_COUNT_LAUNCH();
    band_error_kernel<<<(unsigned)((kBandErrSamples + kBandErrWarps - 1) / kBandErrWarps), kBandErrWarps * 32, 0,
                        st>>>(view_of(f, T), brick_off, brick_count, brick_list, L, dist, ds);
}

void launch_splat(const Fwn& f, long long T, const unsigned long long* brick_off, const unsigned* brick_count,
                  const unsigned* brick_list, const unsigned* active, long long n_bricks, const Lattice& L, float* dist,
                  DevState* ds, cudaStream_t st) {
    // one CTA a brick when the count is known, else a grid-stride over the device's count
    const long long blocks = n_bricks < 0 ? std::min<long long>(L.nbricks, 152ll * 32) : n_bricks;
    if (blocks <= 0) return;
    GBSDF_COUNT_LAUNCH();
    splat_kernel<<<(unsigned)blocks, kSplatThreads, 0, st>>>(view_of(f, T), brick_off, brick_count, brick_list, active,
                                                             L, dist, ds);
}

}  // namespace gbsdf
