// k_caps.cu — winding numbers of whole lattices from ray crossings and the mesh's boundary.
//
// A triangle soup's boundary is the chain of directed edges that no opposite edge cancels. Cap
// triangles with the opposite boundary close the mesh, and the winding number of the closed
// mesh at a point is the signed crossing number k of any ray from it, an integer. So
//     w(mesh) = k - w(caps),
// exactly, for any soup; a watertight mesh has no caps, and a scanned one with 1% of its
// triangles missing has a few caps for every hundred triangles, each as small as its hole.
// Where |w(caps)| < 1/2, a voxel is inside (|w| >= 1/2) iff k != 0: one bit, read off the
// crossings of its column. On the 512^3 vessel tree (2,062 triangles missing) it
// decides all but some hundred of 3.2M voxels; the fixup and the proposals' decisions fell
// from 61 ms with the clusters alone to 12, on the 181 x 141 x 171 mug (watertight) from 29 to 0.4.
//
// The caps: unmatched edges from a table of position-keyed undirected edges (exact comparison
// of the positions); connected components by union-find over the boundary's vertices (the
// boundary of a chain is closed, and so is each connected part of it); a fan from one vertex of
// each component.
//
// The crossings: a voxel's ray goes straight down its own column, moved by an infinitesimal
// (e, e^2) where it meets an edge, so that the crossing number below a voxel is the voxel's own and
// nothing has to be known about its distance to the mesh. The edge functions and the height are
// FP32 with a bound of their rounding, which grows with the triangle and not with the voxel, and
// FP64 where a sign or the voxel above is not certain within it (all but a few in 10^4; a sliver's
// height follows from its area by the same bound). The two triangles of an edge take its ends
// in one order, so they agree on its side. A voxel that a crossing's height cannot be told
// from even in FP64, and a column whose crossings do not sum to zero, are left out. Each
// crossing adds its sign at its height in an integer grid, and a pass up the columns sums it.
#include <algorithm>

#include "gwn_device.cuh"

namespace gbsdf {

namespace {

__device__ __forceinline__ uint32_t coord_bits(float v) {
    return __float_as_uint(v == 0.0f ? 0.0f : v);  // -0 is +0's position
}

struct Pos {
    uint32_t x, y, z;
};
__device__ __forceinline__ Pos vertex_pos(const float* __restrict__ t9, long long t, int k) {
    const float* v = t9 + 9 * t + 3 * k;
    return Pos{coord_bits(v[0]), coord_bits(v[1]), coord_bits(v[2])};
}
__device__ __forceinline__ bool same_pos(const Pos& a, const Pos& b) { return a.x == b.x && a.y == b.y && a.z == b.z; }
__device__ __forceinline__ bool less_pos(const Pos& a, const Pos& b) {
    return a.x != b.x ? a.x < b.x : (a.y != b.y ? a.y < b.y : a.z < b.z);
}
__device__ __forceinline__ uint32_t mix32(uint32_t h) {
    h ^= h >> 16;
    h *= 0x7feb352du;
    h ^= h >> 15;
    h *= 0x846ca68bu;
    return h ^ (h >> 16);
}
__device__ __forceinline__ uint32_t hash_pos(uint32_t seed, const Pos& p) {
    return mix32(mix32(mix32(seed ^ p.x) + p.y * 0x9e3779b9u) ^ (p.z * 0x85ebca6bu));
}

// The table of undirected edges: a slot's first edge (3 t + k + 1), the signed count of its
// directions (+ from the lesser position to the greater) and its least edge number.
__global__ void edge_table_kernel(const float* __restrict__ t9, long long T, unsigned* __restrict__ rep,
                                  int* __restrict__ sum, unsigned* __restrict__ least, unsigned mask,
                                  unsigned long long* __restrict__ counts) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 3 * T) return;
    const long long t = i / 3;
    const int k = (int)(i - 3 * t);
    const Pos a = vertex_pos(t9, t, k), b = vertex_pos(t9, t, k == 2 ? 0 : k + 1);
    const bool finite = (a.x & 0x7f800000u) != 0x7f800000u && (a.y & 0x7f800000u) != 0x7f800000u &&
                        (a.z & 0x7f800000u) != 0x7f800000u;
    if (!finite) counts[1] = 1ull;
    if (same_pos(a, b)) return;
    const bool up = less_pos(a, b);
    const Pos lo = up ? a : b, hi = up ? b : a;
    unsigned s = hash_pos(hash_pos(0x2545f491u, lo), hi) & mask;
    for (unsigned probe = 0; probe <= mask; ++probe, s = (s + 1) & mask) {
        unsigned r = rep[s];
        if (r == 0u) r = atomicCAS(&rep[s], 0u, (unsigned)i + 1u);
        if (r != 0u) {
            const long long rt = (r - 1u) / 3u;
            const int rk = (int)((r - 1u) - 3u * (unsigned)rt);
            const Pos c = vertex_pos(t9, rt, rk), d = vertex_pos(t9, rt, rk == 2 ? 0 : rk + 1);
            if (!((same_pos(c, lo) && same_pos(d, hi)) || (same_pos(c, hi) && same_pos(d, lo)))) continue;
        }
        atomicAdd(&sum[s], up ? 1 : -1);
        atomicMin(&least[s], (unsigned)i);
        return;
    }
}

// The unmatched edges, |count| times each: (least edge number, 1 when the mesh runs it from the
// lesser position to the greater). Only counted while `edges` is null.
__global__ void boundary_edges_kernel(const int* __restrict__ sum, const unsigned* __restrict__ least, long long cap,
                                      uint2* __restrict__ edges, unsigned long long* __restrict__ counts) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < cap; s += stride) {
        const int c = sum[s];
        if (c == 0) continue;
        const unsigned n = (unsigned)abs(c);
        const unsigned long long at = atomicAdd(&counts[edges ? 2 : 0], (unsigned long long)n);
        if (edges)
            for (unsigned k = 0; k < n; ++k) edges[at + k] = make_uint2(least[s], c > 0 ? 1u : 0u);
    }
}

// Boundary edge j's ends in the order the mesh runs it.
__device__ __forceinline__ void edge_ends(const float* __restrict__ t9, uint2 e, const float*& a, const float*& b) {
    const long long t = e.x / 3u;
    const int k = (int)(e.x - 3u * (unsigned)t), k1 = k == 2 ? 0 : k + 1;
    const bool up = less_pos(vertex_pos(t9, t, k), vertex_pos(t9, t, k1));
    const bool keep = up == (e.y != 0u);
    a = t9 + 9 * t + 3 * (keep ? k : k1);
    b = t9 + 9 * t + 3 * (keep ? k1 : k);
}

// Vertex (edge j, side) in the table of boundary vertices; its slot goes to vslot[2 j + side].
__global__ void vertex_table_kernel(const float* __restrict__ t9, const uint2* __restrict__ edges, long long B,
                                    unsigned* __restrict__ rep, unsigned mask, unsigned* __restrict__ vslot) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2 * B) return;
    const float *a, *b;
    edge_ends(t9, edges[i >> 1], a, b);
    const float* v = (i & 1) ? b : a;
    const Pos p{coord_bits(v[0]), coord_bits(v[1]), coord_bits(v[2])};
    unsigned s = hash_pos(0x9d2c5681u, p) & mask;
    for (unsigned probe = 0; probe <= mask; ++probe, s = (s + 1) & mask) {
        unsigned r = rep[s];
        if (r == 0u) r = atomicCAS(&rep[s], 0u, (unsigned)i + 1u);
        if (r != 0u) {
            const float *c, *d;
            edge_ends(t9, edges[(r - 1u) >> 1], c, d);
            const float* q = ((r - 1u) & 1u) ? d : c;
            if (!same_pos(p, Pos{coord_bits(q[0]), coord_bits(q[1]), coord_bits(q[2])})) continue;
        }
        vslot[i] = s;
        return;
    }
}

__device__ __forceinline__ unsigned root_of(volatile unsigned* parent, unsigned v) {
    unsigned p = parent[v];
    while (p != v) {  // parents only ever decrease, so the walk ends
        const unsigned g = parent[p];
        if (g != p) parent[v] = g;
        v = p;
        p = g;
    }
    return v;
}

__global__ void iota_u32_kernel(unsigned* __restrict__ a, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = (unsigned)i;
}

// Joins the two ends of every boundary edge: the greater root is hooked under the lesser.
__global__ void join_kernel(long long B, const unsigned* __restrict__ vslot, unsigned* parent) {
    const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= B) return;
    unsigned a = root_of(parent, vslot[2 * j]), b = root_of(parent, vslot[2 * j + 1]);
    while (a != b) {
        const unsigned hi = a > b ? a : b, lo = a > b ? b : a;
        const unsigned was = atomicCAS(&parent[hi], hi, lo);
        if (was == hi) break;
        a = root_of(parent, was);
        b = root_of(parent, lo);
    }
}

// Each component's apex: its vertex of the least edge number (and side).
__global__ void apex_kernel(const uint2* __restrict__ edges, long long B, const unsigned* __restrict__ vslot,
                            unsigned* parent, unsigned long long* __restrict__ apex) {
    const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= B) return;
    // (least edge number, list place): the place only names the edge, equal numbers are one edge
    atomicMin(&apex[root_of(parent, vslot[2 * j])], ((unsigned long long)edges[j].x << 32) | (unsigned long long)j);
}

// The caps: (apex, b, a) for a boundary edge the mesh runs from a to b.
__global__ void caps_kernel(const float* __restrict__ t9, const uint2* __restrict__ edges, long long B,
                            const unsigned* __restrict__ vslot, unsigned* parent,
                            const unsigned long long* __restrict__ apex, float* __restrict__ out9) {
    const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= B) return;
    const float *a, *b, *p, *q;
    edge_ends(t9, edges[j], a, b);
    edge_ends(t9, edges[(unsigned)apex[root_of(parent, vslot[2 * j])]], p, q);
    float* o = out9 + 9 * j;
    for (int k = 0; k < 3; ++k) {
        o[k] = p[k];
        o[3 + k] = b[k];
        o[6 + k] = a[k];
    }
}

// Edge function of a column (x, y) and the directed edge (a, b) in xy: d, the magnitude m of its
// terms (its rounding is within 4e-16 m), and the side s of the column moved by (e, e^2), 0 for an
// edge without extent. Differences of FP32 coordinates and their products are exact in FP64 but for
// far apart magnitudes; with the ends in order both triangles of an edge get the same.
struct EdgeFn {
    double d, m;
    int s;
};
__device__ __forceinline__ EdgeFn edge_fn(const float* a, const float* b, double x, double y) {
    const bool turn = b[0] < a[0] || (b[0] == a[0] && b[1] < a[1]);
    const float *lo = turn ? b : a, *hi = turn ? a : b;
    const double ux = (double)hi[0] - lo[0], uy = (double)hi[1] - lo[1], wx = x - lo[0], wy = y - lo[1];
    const double p = ux * wy, q = uy * wx, d = p - q;
    int s = (d > 0.0) - (d < 0.0);
    if (s == 0) s = (uy < 0.0) - (uy > 0.0);
    if (s == 0) s = (ux > 0.0) - (ux < 0.0);
    return turn ? EdgeFn{-d, fabs(p) + fabs(q), -s} : EdgeFn{d, fabs(p) + fabs(q), s};
}

// One warp per (triangle, row slice): the lanes take the columns of the triangle's xy box. A
// crossing adds its sign to its column's sum and, at the first voxel above it, to the grid.
__global__ void __launch_bounds__(256) crossings_kernel(const float* __restrict__ t9, long long T, Lattice L,
                                                        int slices, int* __restrict__ grid, int* __restrict__ colsum,
                                                        unsigned* __restrict__ colbad, uint32_t* __restrict__ unsure) {
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const long long t = w / slices;
    const int sl = (int)(w - t * slices);
    if (t >= T) return;
    const float* v = t9 + 9 * t;
    const float h = L.h;
    const int dz = L.dims[2];
    const float x0 = fminf(v[0], fminf(v[3], v[6])), x1 = fmaxf(v[0], fmaxf(v[3], v[6]));
    const float y0 = fminf(v[1], fminf(v[4], v[7])), y1 = fmaxf(v[1], fmaxf(v[4], v[7]));
    const float z0 = fminf(v[2], fminf(v[5], v[8])), z1 = fmaxf(v[2], fmaxf(v[5], v[8]));
    const float zabs = fmaxf(fabsf(z0), fabsf(z1));
    // the columns in the box, at least one more on each side for the rounding
    auto column = [&](float c, int a, float side) {
        const float q = c / h, far = 1.0f + 3e-7f * (fabsf(q) + fabsf((float)L.mn[a]));
        return fminf(fmaxf(floorf(q - (float)L.mn[a] + side * far), -1.0f), (float)L.dims[a]);
    };
    const int ix0 = max(0, (int)column(x0, 0, -1.0f)), ix1 = min(L.dims[0] - 1, (int)column(x1, 0, 1.0f));
    const int iy0 = max(0, (int)column(y0, 1, -1.0f)), iy1 = min(L.dims[1] - 1, (int)column(y1, 1, 1.0f));
    if (ix1 < ix0 || iy1 < iy0) return;
    const int nx = ix1 - ix0 + 1;
    const long long n = (long long)nx * (iy1 - iy0 + 1);
    auto height = [&](int z) { return (float)(L.mn[2] + z) * h; };
    auto above = [&](auto zh) {  // the first voxel higher than zh
        int z = (int)fminf(fmaxf(floorf((float)zh / h) - (float)L.mn[2], 0.0f), (float)dz);
        while (z > 0 && height(z - 1) > zh) --z;
        while (z < dz && height(z) <= zh) ++z;
        return z;
    };
    for (long long c = (long long)sl * 32 + lane; c < n; c += (long long)slices * 32) {
        const int x = ix0 + (int)(c % nx), y = iy0 + (int)(c / nx);
        const float qx = (float)(L.mn[0] + x) * h, qy = (float)(L.mn[1] + y) * h;
        if (qx < x0 || qx > x1 || qy < y0 || qy > y1) continue;
        int pos = 0, neg = 0;
        float df[3], e = 0.0f;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            // four roundings of each product at most (2^-24 each), of FP32 inputs taken as exact
            const float *a = v + 3 * k, *b = v + 3 * (k == 2 ? 0 : k + 1);
            const float ux = b[0] - a[0], uy = b[1] - a[1], wx = qx - a[0], wy = qy - a[1];
            const float q = uy * wx, d = __fmaf_rn(ux, wy, -q);
            const float ek = __fmaf_rn(4e-7f, fabsf(ux * wy) + fabsf(q), 1e-36f);
            pos += d > ek;
            neg += d < -ek;
            df[k] = d;
            e += ek;
        }
        if (pos && neg) continue;
        const size_t col = (size_t)y * L.dims[0] + x;
        auto voxel = [&](int z) { return ((size_t)z * L.dims[1] + y) * L.dims[0] + x; };
        if (pos == 3 || neg == 3) {  // inside for certain (FP64 issues at 1/64 of FP32's rate here)
            const float sum = df[0] + df[1] + df[2], area = fabsf(sum);
            const float zh = __fmaf_rn(df[0], v[8], __fmaf_rn(df[1], v[2], df[2] * v[5])) / sum;
            // the weights are off by e in all, of a true sum of at least area / 2
            const float ez = 2.1f * e * (z1 - z0) / area + 6e-7f * zabs;
            const int z = above(zh);
            if (e < 0.4f * area && (z == dz || height(z) - zh > ez) && (z == 0 || zh - height(z - 1) > ez)) {
                const int sg = neg ? 1 : -1;
                atomicAdd(&colsum[col], sg);
                if (z < dz) atomicAdd(&grid[voxel(z)], sg);
                continue;
            }
        }
        const EdgeFn f0 = edge_fn(v, v + 3, qx, qy), f1 = edge_fn(v + 3, v + 6, qx, qy), f2 = edge_fn(v + 6, v, qx, qy);
        if (f0.s == 0 || f0.s != f1.s || f0.s != f2.s) continue;
        const double sum = f0.d + f1.d + f2.d;
        const double zh = (f0.d * v[8] + f1.d * v[2] + f2.d * v[5]) / sum;
        const double ez = 1e-15 * ((f0.m + f1.m + f2.m) * ((double)z1 - z0) / fabs(sum) + zabs);
        if (!(ez < 0.25 * h)) {
            atomicOr(&colbad[col >> 5], 1u << (col & 31));
            continue;
        }
        const int sg = f0.s < 0 ? 1 : -1, z = above(zh);
        atomicAdd(&colsum[col], sg);
        if (z < dz) atomicAdd(&grid[voxel(z)], sg);
        auto leave = [&](int k) { atomicOr(&unsure[word_of(L, x, y, k)], 1u << (x & 31)); };
        for (int k = z; k < dz && height(k) - zh <= ez; ++k) leave(k);
        for (int k = z - 1; k >= 0 && zh - height(k) <= ez; --k) leave(k);
    }
}

// Sums the crossings up the columns: a warp takes 32 columns of a row. K: the voxels with a
// nonzero crossing number; the columns to leave out (bad, or not summing to zero) go to colbad.
// HBM-bound: 4 bytes a voxel, eight planes in flight (640^3: 0.22 ms, 4.7 TB/s).
__global__ void __launch_bounds__(128) crossing_bits_kernel(const int* __restrict__ grid,
                                                            const int* __restrict__ colsum,
                                                            unsigned* __restrict__ colbad, Lattice L,
                                                            uint32_t* __restrict__ K) {
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= (long long)L.wx * L.dims[1]) return;
    const int xw = (int)(w % L.wx), y = (int)(w / L.wx), x = xw * 32 + lane;
    const bool on = x < L.dims[0];
    const size_t col = (size_t)y * L.dims[0] + x, plane = (size_t)L.dims[0] * L.dims[1];
    if (on && colsum[col] != 0) atomicOr(&colbad[col >> 5], 1u << (col & 31));
    int k = 0;
    constexpr int kAhead = 8;
    for (int z0 = 0; z0 < L.dims[2]; z0 += kAhead) {
        int g[kAhead];
#pragma unroll
        for (int i = 0; i < kAhead; ++i) g[i] = (on && z0 + i < L.dims[2]) ? __ldcs(&grid[(z0 + i) * plane + col]) : 0;
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
            if (z0 + i >= L.dims[2]) break;
            k += g[i];
            const uint32_t word = __ballot_sync(0xffffffffu, on && k != 0);
            if (lane == 0) K[((size_t)(z0 + i) * L.dims[1] + y) * L.wx + xw] = word;
        }
    }
}

unsigned pow2_at_least(long long n) {
    unsigned long long p = 1024;
    while (p < (unsigned long long)n) p <<= 1;
    return (unsigned)p;
}

size_t up256(size_t b) { return (b + 255) & ~size_t(255); }

}  // namespace

size_t edge_table_bytes(long long T) { return 256 + 3 * up256((size_t)pow2_at_least(6 * T) * 4); }

void launch_edge_table(const float* tri9, long long T, void* table, cudaStream_t st) {
    const long long cap = pow2_at_least(6 * T);
    char* p = static_cast<char*>(table);
    auto* counts = reinterpret_cast<unsigned long long*>(p);
    const size_t part = up256((size_t)cap * 4);
    auto* rep = reinterpret_cast<unsigned*>(p + 256);
    auto* sum = reinterpret_cast<int*>(p + 256 + part);
    auto* least = reinterpret_cast<unsigned*>(p + 256 + 2 * part);
    cudaMemsetAsync(p, 0, 256 + 2 * part, st);
    cudaMemsetAsync(least, 0xff, part, st);
    GBSDF_COUNT_LAUNCH();
    edge_table_kernel<<<(unsigned)((3 * T + 255) / 256), 256, 0, st>>>(tri9, T, rep, sum, least, (unsigned)(cap - 1),
                                                                       counts);
    GBSDF_COUNT_LAUNCH();
    boundary_edges_kernel<<<152 * 8, 256, 0, st>>>(sum, least, cap, nullptr, counts);
}

size_t caps_bytes(long long B) {
    const size_t vt = (size_t)pow2_at_least(4 * B);
    return up256((size_t)B * 8) + up256((size_t)B * 8) + 2 * up256(vt * 4) + up256(vt * 8) + up256((size_t)B * 36);
}

const float* launch_caps(const float* tri9, long long T, const void* table, long long B, void* scratch,
                         cudaStream_t st) {
    const long long cap = pow2_at_least(6 * T);
    char* tp = static_cast<char*>(const_cast<void*>(table));
    auto* counts = reinterpret_cast<unsigned long long*>(tp);
    const size_t part = up256((size_t)cap * 4);
    auto* sum = reinterpret_cast<const int*>(tp + 256 + part);
    auto* least = reinterpret_cast<const unsigned*>(tp + 256 + 2 * part);
    const unsigned vt = pow2_at_least(4 * B);
    char* p = static_cast<char*>(scratch);
    auto take = [&](size_t b) {
        char* q = p;
        p += up256(b);
        return q;
    };
    auto* edges = reinterpret_cast<uint2*>(take((size_t)B * 8));
    auto* vslot = reinterpret_cast<unsigned*>(take((size_t)B * 8));
    auto* rep = reinterpret_cast<unsigned*>(take((size_t)vt * 4));
    auto* parent = reinterpret_cast<unsigned*>(take((size_t)vt * 4));
    auto* apex = reinterpret_cast<unsigned long long*>(take((size_t)vt * 8));
    auto* out9 = reinterpret_cast<float*>(take((size_t)B * 36));
    cudaMemsetAsync(&counts[2], 0, 8, st);
    cudaMemsetAsync(rep, 0, (size_t)vt * 4, st);
    cudaMemsetAsync(apex, 0xff, (size_t)vt * 8, st);
    const unsigned bb = (unsigned)((B + 255) / 256), bv = (unsigned)((2 * B + 255) / 256);
    GBSDF_COUNT_LAUNCH();
    boundary_edges_kernel<<<152 * 8, 256, 0, st>>>(sum, least, cap, edges, counts);
    GBSDF_COUNT_LAUNCH();
    iota_u32_kernel<<<(vt + 255) / 256, 256, 0, st>>>(parent, vt);
    GBSDF_COUNT_LAUNCH();
    vertex_table_kernel<<<bv, 256, 0, st>>>(tri9, edges, B, rep, vt - 1, vslot);
    GBSDF_COUNT_LAUNCH();
    join_kernel<<<bb, 256, 0, st>>>(B, vslot, parent);
    GBSDF_COUNT_LAUNCH();
    apex_kernel<<<bb, 256, 0, st>>>(edges, B, vslot, parent, apex);
    GBSDF_COUNT_LAUNCH();
    caps_kernel<<<bb, 256, 0, st>>>(tri9, edges, B, vslot, parent, apex, out9);
    return out9;
}

size_t crossing_bytes(const Lattice& L) {
    const size_t cols = (size_t)L.dims[0] * L.dims[1];
    return up256(cols * 4) + up256((cols + 31) / 32 * 4) + 2 * up256((size_t)L.nwords * 4);
}

Crossings launch_crossings(const float* tri9, long long T, const float* caps9, long long B, const Lattice& L,
                           int* grid, void* scratch, cudaStream_t st) {
    const size_t cols = (size_t)L.dims[0] * L.dims[1];
    char* p = static_cast<char*>(scratch);
    auto* colsum = reinterpret_cast<int*>(p);
    auto* colbad = reinterpret_cast<unsigned*>(p + up256(cols * 4));
    const size_t zeroed = up256(cols * 4) + up256((cols + 31) / 32 * 4) + up256((size_t)L.nwords * 4);
    auto* unsure = reinterpret_cast<uint32_t*>(p + up256(cols * 4) + up256((cols + 31) / 32 * 4));
    auto* K = reinterpret_cast<uint32_t*>(p + zeroed);
    cudaMemsetAsync(p, 0, zeroed, st);
    cudaMemsetAsync(grid, 0, (size_t)L.N * 4, st);
    auto cross = [&](const float* t9, long long n) {
        // few triangles are large ones: several warps share a triangle's columns
        const int slices = (int)std::max<long long>(1, std::min<long long>(64, 152ll * 64 / n));
        GBSDF_COUNT_LAUNCH();
        crossings_kernel<<<(unsigned)((n * slices + 7) / 8), 256, 0, st>>>(t9, n, L, slices, grid, colsum, colbad,
                                                                             unsure);
    };
    cross(tri9, T);
    if (B > 0) cross(caps9, B);
    const long long warps = (long long)L.wx * L.dims[1];
    GBSDF_COUNT_LAUNCH();
    crossing_bits_kernel<<<(unsigned)((warps + 3) / 4), 128, 0, st>>>(grid, colsum, colbad, L, K);
    return Crossings{K, unsure, colbad};
}

}  // namespace gbsdf
