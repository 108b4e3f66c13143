// k_iso.cu — iso-surface extraction (marching cubes) straight from a device-resident grid.
//
// Reference: CudaRasterizer::extract_iso_surface (cuda_marching_cubes.cu:829-951) with
// gpu_mc_seal_border_kernel (:312-332), dev_mc_cube_index (:334-360), the count pass
// (:362-413), gpu_mc_emit_vertices_kernel (:415-489) and gpu_mc_emit_triangles_kernel
// (:491-555). The reference takes the grid as a host vector and uploads it (2.6 GB for
// the 860 x 860 x 880 grid); here the grid may be the engine's device output, read in
// place. Its rules are kept:
//   * boundary voxels read below iso + h read as iso + h (the seal; the caller's grid is
//     not written);
//   * a corner is inside when value - iso <= 0; one vertex per grid edge whose ends
//     differ, at p0 + t h along the edge, t = (v0 / (v0 - v1)) clamped to [0.001, 0.999]
//     (0.5 when |v0 - v1| <= 1e-7), each operation rounded once (-fmad=false);
//   * triangles connect the vertices on a cube's edges, outward (towards values above iso).
// What differs:
//   * order: the reference numbers vertices and triangles with atomic counters (the order
//     changes from run to run); here vertices follow the voxel order (x, y, z edges of a
//     voxel in turn) and triangles the cube order, by scans;
//   * the triangle table: the reference's is a hand-written table; this one is generated
//     (mc_table_init) from one rule: on each cube face the crossing edges pair up so that
//     inside corners are cut off separately -- on a face with two inside corners on a
//     diagonal they stay apart -- and the resulting loops are triangulated without chords
//     across a cube face. Both cubes that share a face see its four corners alike, so they
//     pair its edges alike and the surface is closed and consistently oriented for any grid
//     (the reference's table can pair an ambiguous face differently in the two cubes). On
//     ambiguous cubes the vertices may be connected differently from the reference's table.
//
// Passes:
//   1. inside bits of the grid, words of 32 voxels along x;
//   2. count: vertices and triangles per word and per block of 256 words; the words that hold
//      any are listed;
//   3. a scan of the blocks' totals;
//   4. emission of the listed words' vertices and triangles; a cube's edge vertex is its owner
//      word's first vertex plus the crossings before it in the word.
#include <math_constants.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

#include "../../include/gbsdf.h"
#include "gbsdf_internal.h"

namespace gbsdf {
namespace {

// Cube corners (x, y, z bits as in the reference's corner order), edges (corner pairs)
// and faces (corners in cyclic order).
constexpr int kCorner[8][3] = {{0, 0, 0}, {1, 0, 0}, {1, 1, 0}, {0, 1, 0}, {0, 0, 1}, {1, 0, 1}, {1, 1, 1}, {0, 1, 1}};
constexpr int kEdge[12][2] = {{0, 1}, {1, 2}, {3, 2}, {0, 3}, {4, 5}, {5, 6}, {7, 6}, {4, 7}, {0, 4}, {1, 5}, {2, 6}, {3, 7}};
constexpr int kFace[6][4] = {{0, 1, 2, 3}, {4, 5, 6, 7}, {0, 1, 5, 4}, {3, 2, 6, 7}, {0, 3, 7, 4}, {1, 2, 6, 5}};

// The table on the device, a case a word: 4 bits an edge from the low end, the number of
// triangles in the top 4. Read with divergent per-lane cases: global memory, L1-cached.
__device__ unsigned long long c_tri[256];

int8_t g_tri[256][16];
std::once_flag g_tri_once;

int edge_of(int a, int b) {
    for (int e = 0; e < 12; ++e)
        if ((kEdge[e][0] == a && kEdge[e][1] == b) || (kEdge[e][0] == b && kEdge[e][1] == a)) return e;
    return -1;
}

// The triangle table from the face rule above. Per case: on each face, pair the crossing
// edges (cutting inside corners off separately) into segments directed so that the inside
// corners lie on their left seen from outside the cube; follow the segments into closed
// loops (every crossing edge lies on two faces) and walk each loop backwards, which turns
// its triangles outward (from the inside corners to the outside ones). The two cubes that
// share a face direct its segments oppositely, so the surface is closed and consistently
// oriented. A loop of more than 3 edges is split by the first triangulation (in a fixed
// enumeration) none of whose diagonals joins two edges of one cube face: such a chord would
// also be drawn by the neighbouring cube and leave an edge with four triangles. Every loop
// of the 256 cases has one; at most 5 triangles per case.
bool on_face(int e, const int* f) {
    bool a = false, b = false;
    for (int k = 0; k < 4; ++k) {
        a |= f[k] == kEdge[e][0];
        b |= f[k] == kEdge[e][1];
    }
    return a && b;
}

bool share_face(int e0, int e1) {
    for (const auto& f : kFace)
        if (on_face(e0, f) && on_face(e1, f)) return true;
    return false;
}

// all triangulations of the polygon p[0..n-1]: triangle (p0, pk, p(n-1)) plus the two sides
void triangulations(const std::vector<int>& p, std::vector<std::vector<std::array<int, 3>>>& out) {
    const int n = (int)p.size();
    out.clear();
    if (n < 3) {
        out.push_back({});
        return;
    }
    for (int k = 1; k + 1 < n; ++k) {
        std::vector<std::vector<std::array<int, 3>>> L, R;
        triangulations(std::vector<int>(p.begin(), p.begin() + k + 1), L);
        triangulations(std::vector<int>(p.begin() + k, p.end()), R);
        for (const auto& l : L)
            for (const auto& r : R) {
                std::vector<std::array<int, 3>> t = l;
                t.insert(t.end(), r.begin(), r.end());
                t.push_back({p[0], p[k], p[n - 1]});
                out.push_back(t);
            }
    }
}

void mc_table_init() {
    std::memset(g_tri, -1, sizeof(g_tri));
    static const int kNormal[6][3] = {{0, 0, -1}, {0, 0, 1}, {0, -1, 0}, {0, 1, 0}, {-1, 0, 0}, {1, 0, 0}};
    auto mid = [](int e, int c) { return 0.5 * (kCorner[kEdge[e][0]][c] + kCorner[kEdge[e][1]][c]); };
    for (int cs = 0; cs < 256; ++cs) {
        int in[8];
        for (int i = 0; i < 8; ++i) in[i] = (cs >> i) & 1;
        int nxt[12];
        for (int e = 0; e < 12; ++e) nxt[e] = -1;
        auto segment = [&](int a, int b, const double* c, const int* fn) {
            double pq[3], pc[3];
            for (int k = 0; k < 3; ++k) {
                pq[k] = mid(b, k) - mid(a, k);
                pc[k] = c[k] - mid(a, k);
            }
            const double t = fn[0] * (pq[1] * pc[2] - pq[2] * pc[1]) + fn[1] * (pq[2] * pc[0] - pq[0] * pc[2]) +
                             fn[2] * (pq[0] * pc[1] - pq[1] * pc[0]);
            if (t < 0) std::swap(a, b);
            nxt[a] = b;
        };
        for (int fi = 0; fi < 6; ++fi) {
            const int* f = kFace[fi];
            int cross[4], nc = 0;
            for (int k = 0; k < 4; ++k)
                if (in[f[k]] != in[f[(k + 1) % 4]]) cross[nc++] = k;
            if (nc == 2) {
                double c[3] = {0, 0, 0};
                int ni = 0;
                for (int k = 0; k < 4; ++k)
                    if (in[f[k]]) {
                        for (int j = 0; j < 3; ++j) c[j] += kCorner[f[k]][j];
                        ++ni;
                    }
                for (int j = 0; j < 3; ++j) c[j] /= ni;
                segment(edge_of(f[cross[0]], f[(cross[0] + 1) % 4]), edge_of(f[cross[1]], f[(cross[1] + 1) % 4]), c,
                        kNormal[fi]);
            } else if (nc == 4) {  // two inside corners on a diagonal: cut each off
                for (int k = 0; k < 4; ++k)
                    if (in[f[k]]) {
                        const double c[3] = {(double)kCorner[f[k]][0], (double)kCorner[f[k]][1],
                                             (double)kCorner[f[k]][2]};
                        segment(edge_of(f[(k + 3) % 4], f[k]), edge_of(f[k], f[(k + 1) % 4]), c, kNormal[fi]);
                    }
            }
        }
        bool seen[12] = {false};
        int nt = 0;
        for (int s = 0; s < 12; ++s) {
            if (nxt[s] < 0 || seen[s]) continue;
            std::vector<int> loop;
            for (int cur = s; !seen[cur]; cur = nxt[cur]) {
                loop.push_back(cur);
                seen[cur] = true;
            }
            std::reverse(loop.begin() + 1, loop.end());  // walk backwards: outward triangles
            const int n = (int)loop.size();
            std::vector<std::vector<std::array<int, 3>>> all;
            triangulations(loop, all);
            for (const auto& tri : all) {
                bool chord = false;
                for (const auto& t : tri)
                    for (int k = 0; k < 3; ++k) {
                        const int a = t[k], b = t[(k + 1) % 3];
                        int ia = 0, ib = 0;
                        for (int i = 0; i < n; ++i) {
                            if (loop[i] == a) ia = i;
                            if (loop[i] == b) ib = i;
                        }
                        const int d = ia > ib ? ia - ib : ib - ia;
                        if (d != 1 && d != n - 1 && share_face(a, b)) chord = true;
                    }
                if (chord) continue;
                for (const auto& t : tri) {
                    if (nt == 5) break;
                    for (int k = 0; k < 3; ++k) g_tri[cs][3 * nt + k] = (int8_t)t[k];
                    ++nt;
                }
                break;
            }
        }
    }
}

// Work layout. The grid is read once, into one inside bit per voxel: words of 32 voxels along
// x, rows padded to whole words, row y + z dy. The mesh hangs on the bits alone -- an edge is
// crossed where neighbouring bits differ, a cube's case is eight bits -- so everything but the
// vertex positions works on 1/32 of the grid, and, past the count, only on the words that hold
// a vertex or a cut cube ("items"). 509 x 480 x 512: 0.32 ms a call (bits 88 us, count 40, scan 6,
// emission 74); three walks over the grid with 5 B per voxel of masks and vertex numbers between
// them took 2.40 ms.
constexpr int kIsoThreads = 256;
constexpr int kIsoWarps = kIsoThreads / 32;
constexpr int kIsoChunk = 8;  // words a warp reads at once

struct IsoGeom {
    int dx, dy, dz, wpr;  // wpr: words per row
    long long rows, nw;   // rows of the grid, words
    float iso, seal;
    bool sealed;          // no border voxel is inside
};

__device__ __forceinline__ long long div_u(long long a, long long range, int b) {  // a / b, a < range
    return (range >> 32) ? a / b : (long long)((unsigned)a / (unsigned)b);
}

// value relative to iso, with the reference's border seal
__device__ __forceinline__ float iso_rel(float v, bool border, const IsoGeom& G) {
    if (border && v < G.seal) v = G.seal;
    return v - G.iso;
}
__device__ __forceinline__ float iso_val(const float* __restrict__ g, int x, int y, int z, const IsoGeom& G) {
    const bool border = x == 0 || x == G.dx - 1 || y == 0 || y == G.dy - 1 || z == 0 || z == G.dz - 1;
    return iso_rel(__ldg(&g[((size_t)z * G.dy + y) * G.dx + x]), border, G);
}

// 1. inside bits: a warp takes rows, 8 words at a time, eight loads in flight per lane; blocks
// by (rows, plane), so that no index is divided. A border voxel reads as iso + h at least, so it is
// outside, unless the sum rounds to iso and nothing changes sides: the seal is a mask on the
// words. Bound by the read of the grid.
__global__ void __launch_bounds__(kIsoThreads, 8) iso_bits_kernel(const float* __restrict__ g, IsoGeom G,
                                                                  unsigned* __restrict__ bits,
                                                                  unsigned long long* __restrict__ n_items) {
    if ((blockIdx.x | blockIdx.y | threadIdx.x) == 0) *n_items = 0;
    const int lane = threadIdx.x & 31, step = gridDim.x * kIsoWarps;
    for (int z = blockIdx.y; z < G.dz; z += gridDim.y)
        for (int y = blockIdx.x * kIsoWarps + (threadIdx.x >> 5); y < G.dy; y += step) {
            const long long row = (long long)z * G.dy + y;
            const float* p = g + (size_t)row * G.dx + lane;
            unsigned* out = bits + row * G.wpr + lane;
            const bool sealed_row = G.sealed && (y == 0 || y == G.dy - 1 || z == 0 || z == G.dz - 1);
            for (int w0 = 0; w0 < G.wpr; w0 += kIsoChunk, p += 32 * kIsoChunk, out += kIsoChunk) {
                const int left = sealed_row ? 0 : G.dx - 32 * w0 - lane;  // voxels of the row from this lane's first
                float v[kIsoChunk];
                unsigned mine = 0;
#pragma unroll
                for (int j = 0; j < kIsoChunk; ++j) v[j] = 32 * j < left ? __ldg(p + 32 * j) : CUDART_NAN_F;
#pragma unroll
                for (int j = 0; j < kIsoChunk; ++j) {
                    const unsigned b = __ballot_sync(0xffffffffu, v[j] - G.iso <= 0.0f);
                    if (lane == j) mine = b;
                }
                if (lane < kIsoChunk && w0 + lane < G.wpr) {
                    if (G.sealed && w0 + lane == 0) mine &= ~1u;
                    if (G.sealed && w0 + lane == G.wpr - 1) mine &= ~(1u << ((G.dx - 1) & 31));
                    *out = mine;
                }
            }
        }
}

// bits of the voxels with a neighbour at x + 1, among the word's 32
__device__ __forceinline__ unsigned has_next(const IsoGeom& G, int w) {
    const int n = G.dx - 1 - 32 * w;
    return n >= 32 ? ~0u : (1u << n) - 1u;
}
__device__ __forceinline__ unsigned shift_in(unsigned s, unsigned next) { return (s >> 1) | (next << 31); }

// case (reference corner order) of the cube at bit l: lo[r][k] the bits of the row y + r,
// plane z + k, hi the same one voxel on
__device__ __forceinline__ int cube_case(const unsigned lo[2][2], const unsigned hi[2][2], int l) {
    auto bit = [l](unsigned s) { return (int)((s >> l) & 1u); };
    return bit(lo[0][0]) | bit(hi[0][0]) << 1 | bit(hi[1][0]) << 2 | bit(lo[1][0]) << 3 | bit(lo[0][1]) << 4 |
           bit(hi[0][1]) << 5 | bit(hi[1][1]) << 6 | bit(lo[1][1]) << 7;
}

// 2. count: a thread a word. Vertices of a word and cut cubes by bit operations; the block's
// items are packed in order and a thread counts each one's triangles, cube by cube (most words
// hold a few cubes: with a warp an item, a lane a cube, 58 us at 509 x 480 x 512, this 40). Writes the
// word's first vertex (within the block of 256 words), the items (word, first triangle within
// the block; in the order the blocks come -- an item carries all that its emission needs) and
// the block's totals. Bound by the loads of the bits, which come from L2.
struct IsoItem {
    unsigned block, rest;  // rest: word of the block | first triangle << 8 (at most 256 x 160)
};

__global__ void __launch_bounds__(kIsoThreads) iso_count_kernel(IsoGeom G, const unsigned* __restrict__ bits,
                                                                uint16_t* __restrict__ vpre,
                                                                uint2* __restrict__ totals,
                                                                IsoItem* __restrict__ items,
                                                                unsigned long long* __restrict__ n_items) {
    __shared__ unsigned s_lo[4][kIsoThreads], s_hi[4][kIsoThreads], s_cut[kIsoThreads];
    __shared__ unsigned s_warp[2][kIsoWarps];
    __shared__ uint8_t s_list[kIsoThreads];
    __shared__ unsigned long long s_base;
    const int t = threadIdx.x, lane = t & 31, wp = t >> 5;
    const long long i = (long long)blockIdx.x * kIsoThreads + t;
    unsigned nv = 0, cut = 0;
    if (i < G.nw) {
        const long long row = div_u(i, G.nw, G.wpr);
        const int w = (int)(i - row * G.wpr);
        const int z = (int)div_u(row, G.rows, G.dy), y = (int)(row - (long long)z * G.dy);
        const unsigned nx = has_next(G, w);
        const bool ny = y + 1 < G.dy, nz = z + 1 < G.dz, nw = w + 1 < G.wpr;
        unsigned lo[2][2], hi[2][2];
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const unsigned* p = bits + i + (r && ny ? G.wpr : 0) + (k && nz ? (long long)G.dy * G.wpr : 0);
                lo[r][k] = __ldg(p);
                hi[r][k] = shift_in(lo[r][k], nw ? __ldg(p + 1) : 0u);
                s_lo[r + 2 * k][t] = lo[r][k];
                s_hi[r + 2 * k][t] = hi[r][k];
            }
        // (past the last row or plane the neighbour is the row itself, past the last voxel both
        // bits are 0: no crossing)
        nv = __popc((lo[0][0] ^ hi[0][0]) & nx) + __popc(lo[0][0] ^ lo[1][0]) + __popc(lo[0][0] ^ lo[0][1]);
        const unsigned any = lo[0][0] | lo[1][0] | lo[0][1] | lo[1][1] | hi[0][0] | hi[1][0] | hi[0][1] | hi[1][1];
        const unsigned all = lo[0][0] & lo[1][0] & lo[0][1] & lo[1][1] & hi[0][0] & hi[1][0] & hi[0][1] & hi[1][1];
        if (ny && nz) cut = any & ~all & nx;
    }
    s_cut[t] = cut;
    // prefixes of the vertices and the items over the block, in word order
    const unsigned act = __ballot_sync(0xffffffffu, nv || cut);
    unsigned inc = nv;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    if (lane == 31) {
        s_warp[0][wp] = inc;
        s_warp[1][wp] = __popc(act);
    }
    __syncthreads();
    unsigned vb = 0, ab = 0, vt = 0, na = 0;
#pragma unroll
    for (int k = 0; k < kIsoWarps; ++k) {
        if (k < wp) {
            vb += s_warp[0][k];
            ab += s_warp[1][k];
        }
        vt += s_warp[0][k];
        na += s_warp[1][k];
    }
    if (na == 0) {
        if (t == 0) totals[blockIdx.x] = make_uint2(0u, 0u);
        return;
    }
    if (i < G.nw) vpre[i] = (uint16_t)(vb + inc - nv);
    if (nv || cut) s_list[ab + __popc(act & ((1u << lane) - 1u))] = (uint8_t)t;
    __syncthreads();
    unsigned nt = 0;
    if ((unsigned)t < na) {  // a thread an item
        const int l = s_list[t];
        const unsigned lo[2][2] = {{s_lo[0][l], s_lo[2][l]}, {s_lo[1][l], s_lo[3][l]}};
        const unsigned hi[2][2] = {{s_hi[0][l], s_hi[2][l]}, {s_hi[1][l], s_hi[3][l]}};
        for (unsigned c = s_cut[l]; c; c &= c - 1)
            nt += (unsigned)(__ldg(&c_tri[cube_case(lo, hi, __ffs(c) - 1)]) >> 60);
    }
    inc = nt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    if (lane == 31) s_warp[0][wp] = inc;  // (its readers are past the barriers above)
    __syncthreads();
    unsigned tb = 0, tt = 0;
#pragma unroll
    for (int k = 0; k < kIsoWarps; ++k) {
        if (k < wp) tb += s_warp[0][k];
        tt += s_warp[0][k];
    }
    if (t == 0) {
        s_base = atomicAdd(n_items, (unsigned long long)na);
        totals[blockIdx.x] = make_uint2(vt, tt);
    }
    __syncthreads();
    if ((unsigned)t < na) items[s_base + t] = IsoItem{blockIdx.x, (unsigned)s_list[t] | (tb + inc - nt) << 8};
}

// 3. the blocks' first vertex and triangle, and the mesh's totals (sum[0], sum[1]). At most one
// CTA per SM; each adds up the blocks before its own share itself, which at 15,360 blocks (509 x
// 480 x 512) is 15 loads a thread against a second launch or a wait on its neighbours (one CTA
// over all blocks: 16 us).
constexpr int kScanThreads = 1024;
__device__ __forceinline__ unsigned long long warp_inclusive(unsigned long long v) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long u = __shfl_up_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) >= o) v += u;
    }
    return v;
}
__global__ void __launch_bounds__(kScanThreads) iso_scan_kernel(const uint2* __restrict__ totals, long long n,
                                                                long long share, ulonglong2* __restrict__ first,
                                                                unsigned long long* __restrict__ sum) {
    __shared__ unsigned long long s_w[2][32];
    const int t = threadIdx.x, lane = t & 31, wp = t >> 5;
    const long long begin = blockIdx.x * share, end = min(n, begin + share);
    unsigned long long cv = 0, ct = 0;  // before the share
    for (long long i = t; i < begin; i += kScanThreads) {
        const uint2 q = __ldg(&totals[i]);
        cv += q.x;
        ct += q.y;
    }
    // inclusive over the CTA; the last one of s_w is the total
    auto scan = [&](unsigned long long& v, unsigned long long& u) {
        v = warp_inclusive(v);
        u = warp_inclusive(u);
        __syncthreads();  // s_w's last readers
        if (lane == 31) {
            s_w[0][wp] = v;
            s_w[1][wp] = u;
        }
        __syncthreads();
        if (wp < 2) s_w[wp][lane] = warp_inclusive(s_w[wp][lane]);
        __syncthreads();
        if (wp) {
            v += s_w[0][wp - 1];
            u += s_w[1][wp - 1];
        }
    };
    scan(cv, ct);
    cv = s_w[0][31];
    ct = s_w[1][31];
    for (long long b0 = begin; b0 < end; b0 += kScanThreads) {
        const long long i = b0 + t;
        const uint2 q = i < end ? __ldg(&totals[i]) : make_uint2(0u, 0u);
        unsigned long long v = q.x, u = q.y;
        scan(v, u);
        if (i < end) first[i] = make_ulonglong2(cv + v - q.x, ct + u - q.y);
        cv += s_w[0][31];
        ct += s_w[1][31];
    }
    if (t == 0 && end == n) {
        sum[0] = cv;
        sum[1] = ct;
    }
}

// 4. emission: a thread an item, the vertices in blocks of their own (blockIdx.y). The bits around the word (rows y .. y + 2, planes z .. z + 2)
// give the crossing masks of the words that own its cubes' edges, and these, with the words'
// first vertices, every edge's vertex number. Most words hold a few cubes in a row of 32, which
// is why a thread walks them: a warp an item, a lane a voxel, spent 800 instructions an item and
// 346 us at 509 x 480 x 512, this 74 (88 with both kinds in one thread). Bound by latency: two rounds of loads, then the grid's values at the
// crossings.
constexpr int kEmitThreads = 128;
__global__ void __launch_bounds__(kEmitThreads) iso_emit_kernel(const float* __restrict__ g, IsoGeom G, float h,
                                                                float ox, float oy, float oz,
                                                                const unsigned* __restrict__ bits,
                                                                const uint16_t* __restrict__ vpre,
                                                                const ulonglong2* __restrict__ first,
                                                                const IsoItem* __restrict__ items, long long n_items,
                                                                float* __restrict__ out_v,
                                                                uint32_t* __restrict__ out_i) {
    __shared__ unsigned s_id[12][kEmitThreads];  // a cube's vertex numbers, by edge
    const int t = threadIdx.x;
    const long long it = (long long)blockIdx.x * kEmitThreads + t;
    if (it >= n_items) return;
    const IsoItem item = items[it];
    const long long i = (long long)item.block * kIsoThreads + (item.rest & 0xffu);
    const long long row = div_u(i, G.nw, G.wpr);
    const int w = (int)(i - row * G.wpr);
    const int z = (int)div_u(row, G.rows, G.dy), y = (int)(row - (long long)z * G.dy);
    const int ry = G.dy - 1 - y, rz = G.dz - 1 - z;  // rows and planes past this one
    const unsigned nx = has_next(G, w);
    // the word r rows and k planes on (past the last, the last one's own)
    auto at = [&](int r, int k) { return i + min(r, ry) * (long long)G.wpr + min(k, rz) * ((long long)G.dy * G.wpr); };
    auto word = [&](int r, int k, int n) { return w + n < G.wpr ? __ldg(&bits[at(r, k) + n]) : 0u; };
    auto number = [&](int r, int k, int n) {  // fewer than 2^32 vertices; unused where the word has none
        const long long j = at(r, k) + n;
        return w + n < G.wpr ? (unsigned)first[j / kIsoThreads].x + vpre[j] : 0u;
    };
    if (blockIdx.y == 0) {  // vertices: this word's own edges, in voxel order
        const unsigned s = word(0, 0, 0);
        const unsigned mx = (s ^ shift_in(s, word(0, 0, 1))) & nx, my = s ^ word(1, 0, 0), mz = s ^ word(0, 1, 0);
        const float py = oy + (float)y * h, pz = oz + (float)z * h;
        float* o = out_v + 3ull * number(0, 0, 0);
        for (unsigned m = mx | my | mz; m; m &= m - 1) {
            const int l = __ffs(m) - 1, x = 32 * w + l;
            const float px = ox + (float)x * h;
            const float v0 = iso_val(g, x, y, z, G);
            auto cross = [&](float v1) {
                const float den = v0 - v1;
                return (fabsf(den) > 1e-7f) ? fminf(fmaxf(v0 / den, 0.001f), 0.999f) : 0.5f;
            };
            if ((mx >> l) & 1u) {
                o[0] = px + cross(iso_val(g, x + 1, y, z, G)) * h;
                o[1] = py;
                o[2] = pz;
                o += 3;
            }
            if ((my >> l) & 1u) {
                o[0] = px;
                o[1] = py + cross(iso_val(g, x, y + 1, z, G)) * h;
                o[2] = pz;
                o += 3;
            }
            if ((mz >> l) & 1u) {
                o[0] = px;
                o[1] = py;
                o[2] = pz + cross(iso_val(g, x, y, z + 1, G)) * h;
                o += 3;
            }
        }
        return;
    }
    // triangles
    if (ry == 0 || rz == 0) return;
    unsigned lo[2][2], hi[2][2], mx[2][2], my[2][2], mz[2][2], f[2][2];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            lo[r][k] = word(r, k, 0);
            hi[r][k] = shift_in(lo[r][k], word(r, k, 1));
            f[r][k] = number(r, k, 0);
        }
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            mx[r][k] = (lo[r][k] ^ hi[r][k]) & nx;
            my[r][k] = lo[r][k] ^ (r ? word(2, k, 0) : lo[1][k]);
            mz[r][k] = lo[r][k] ^ (k ? word(r, 2, 0) : lo[r][1]);
        }
    const unsigned any = lo[0][0] | lo[1][0] | lo[0][1] | lo[1][1] | hi[0][0] | hi[1][0] | hi[0][1] | hi[1][1];
    const unsigned all = lo[0][0] & lo[1][0] & lo[0][1] & lo[1][1] & hi[0][0] & hi[1][0] & hi[0][1] & hi[1][1];
    uint32_t* o = out_i + 3ull * (first[item.block].y + (item.rest >> 8));
    for (unsigned m = any & ~all & nx; m; m &= m - 1) {
        const int l = __ffs(m) - 1;
        const unsigned below = (1u << l) - 1u;
        unsigned c[2][2], bx[2][2], by[2][2], c1[2][2], bx1[2][2], by1[2][2];  // first vertices of voxels l, l + 1
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                c[r][k] = f[r][k] + __popc(mx[r][k] & below) + __popc(my[r][k] & below) + __popc(mz[r][k] & below);
                bx[r][k] = (mx[r][k] >> l) & 1u;
                by[r][k] = (my[r][k] >> l) & 1u;
                if (r == 1 && k == 1) continue;
                c1[r][k] = c[r][k] + bx[r][k] + by[r][k] + ((mz[r][k] >> l) & 1u);
                bx1[r][k] = (mx[r][k] >> l >> 1) & 1u;  // (l = 31: below)
                by1[r][k] = (my[r][k] >> l >> 1) & 1u;
            }
        if (l == 31) {  // voxel l + 1 is the next word's first
            const bool next_x = 32 * w + 33 < G.dx;
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    if (r == 1 && k == 1) continue;
                    const unsigned n = word(r, k, 1);
                    c1[r][k] = number(r, k, 1);
                    bx1[r][k] = next_x ? (n ^ (n >> 1)) & 1u : 0u;
                    by1[r][k] = (n ^ word(r + 1, k, 1)) & 1u;
                }
        }
        s_id[0][t] = c[0][0];
        s_id[1][t] = c1[0][0] + bx1[0][0];
        s_id[2][t] = c[1][0];
        s_id[3][t] = c[0][0] + bx[0][0];
        s_id[4][t] = c[0][1];
        s_id[5][t] = c1[0][1] + bx1[0][1];
        s_id[6][t] = c[1][1];
        s_id[7][t] = c[0][1] + bx[0][1];
        s_id[8][t] = c[0][0] + bx[0][0] + by[0][0];
        s_id[9][t] = c1[0][0] + bx1[0][0] + by1[0][0];
        s_id[10][t] = c1[1][0] + bx1[1][0] + by1[1][0];
        s_id[11][t] = c[1][0] + bx[1][0] + by[1][0];
        unsigned long long tri = __ldg(&c_tri[cube_case(lo, hi, l)]);
        for (unsigned j = 3 * (unsigned)(tri >> 60); j; --j, tri >>= 4) *o++ = s_id[tri & 15u][t];
    }
}

// ---- other consumers of the SDF: interior volume, default seed -----------------------
// CudaRasterizer::compute_sdf_interior_volume_gpu (cuda_viewport_gl.cu:702-741, kernel
// :84-112) and find_default_seed_gpu (cuda_viewport_packers.cu:304-384, kernel :235-276,
// min reduce cuda_rasterizer.cu:1632-1665): both read the grid in place here. Counts and
// minima are integer atomics, so the results do not depend on the launch.
__device__ __forceinline__ unsigned ordered_u32(float f) {  // order-preserving float key
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__global__ void sdf_inside_min_kernel(const float* __restrict__ g, long long n,
                                      unsigned long long* __restrict__ inside, unsigned* __restrict__ min_key) {
    unsigned long long c = 0;
    float mn = 1e30f;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float v = __ldg(&g[i]);
        c += (v <= 0.0f);
        if (v < mn) mn = v;
    }
    unsigned k = ordered_u32(mn);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        c += __shfl_down_sync(0xffffffffu, c, o);
        k = min(k, __shfl_down_sync(0xffffffffu, k, o));
    }
    if ((threadIdx.x & 31) == 0) {
        if (c) atomicAdd(inside, c);
        atomicMin(min_key, k);
    }
}

__global__ void sdf_seed_kernel(const float* __restrict__ g, int dx, int dy, int dz, int mx, int my, int mz, float h,
                                float minpz, float cx, float cy, float margin, unsigned long long* __restrict__ best) {
    const long long n = (long long)dx * dy * dz;
    unsigned long long b = ~0ull;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float d = __ldg(&g[i]);
        if (d > margin) continue;
        const int x = (int)(i % dx), y = (int)((i / dx) % dy), z = (int)(i / ((long long)dx * dy));
        const float px = (float)(mx + x) * h, py = (float)(my + y) * h, pz = (float)(mz + z) * h;
        const float ex = px - cx, ey = py - cy;
        const float xy = sqrtf(ex * ex + ey * ey);
        const float zh = fmaxf(0.0f, pz - minpz);
        const float score = zh * 10.0f + xy * 0.5f;
        const unsigned long long key = ((unsigned long long)ordered_u32(score) << 32) | (unsigned long long)(i & 0xffffffffLL);
        b = key < b ? key : b;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long t = __shfl_down_sync(0xffffffffu, b, o);
        b = t < b ? t : b;
    }
    if ((threadIdx.x & 31) == 0 && b != ~0ull) atomicMin(best, b);
}

struct IsoErr {
    char* buf;
    size_t len;
    int set(int status, const char* fmt, ...) {
        if (buf && len > 0) {
            va_list ap;
            va_start(ap, fmt);
            vsnprintf(buf, len, fmt, ap);
            va_end(ap);
        }
        return status;
    }
};

// Per-device scratch kept across calls (grow-only, one allocation, carved 256-byte
// aligned): the query call and the emit call that follows it, and repeated extractions of
// one lattice, allocate nothing. Calls on one device hold its lock for their duration.
struct IsoCache {
    std::mutex mu;
    bool table = false;    // the device holds the triangle table
    void* base = nullptr;  // scratch
    size_t bytes = 0;
    void* out = nullptr;   // library-owned mesh (gbsdf_extract_iso_surface_device)
    size_t out_bytes = 0;
};
IsoCache g_iso[64];

struct IsoScratch {
    IsoCache& c;
    size_t need = 0;
    bool sizing = true;
    char* cur = nullptr;
    template <class T>
    T* get(size_t count, cudaError_t& err) {
        const size_t b = (std::max<size_t>(count, 1) * sizeof(T) + 255) & ~size_t(255);
        if (sizing) {
            need += b;
            return nullptr;
        }
        if (err != cudaSuccess) return nullptr;
        T* p = reinterpret_cast<T*>(cur);
        cur += b;
        return p;
    }
    cudaError_t commit() {  // after the sizing pass: grow the cache, start carving
        if (need > c.bytes) {
            if (c.base) cudaFree(c.base);
            c.base = nullptr;
            c.bytes = 0;
            const cudaError_t ce = cudaMalloc(&c.base, need);
            if (ce != cudaSuccess) return ce;
            c.bytes = need;
        }
        sizing = false;
        cur = static_cast<char*>(c.base);
        return cudaSuccess;
    }
};

bool table_to_device() {
    std::call_once(g_tri_once, mc_table_init);
    unsigned long long t[256];
    for (int cs = 0; cs < 256; ++cs) {
        unsigned long long n = 0;
        t[cs] = 0;
        while (n < 5 && g_tri[cs][3 * n] >= 0) {
            for (int k = 0; k < 3; ++k) t[cs] |= (unsigned long long)g_tri[cs][3 * n + k] << (4 * (3 * n + k));
            ++n;
        }
        t[cs] |= n << 60;
    }
    return cudaMemcpyToSymbol(c_tri, t, sizeof(t)) == cudaSuccess;
}

}  // namespace

void release_iso_workspace(int device) {
    if (device < 0 || device >= 64) return;
    std::lock_guard<std::mutex> lock(g_iso[device].mu);
    if (g_iso[device].base) cudaFree(g_iso[device].base);
    if (g_iso[device].out) cudaFree(g_iso[device].out);
    g_iso[device].base = g_iso[device].out = nullptr;
    g_iso[device].table = false;
    g_iso[device].bytes = g_iso[device].out_bytes = 0;
}

}  // namespace gbsdf

using namespace gbsdf;

// outputs: 0 caller's host arrays, 1 caller's device arrays, 2 library-owned device arrays
// (their addresses returned through *lib_v / *lib_i)
static int extract_iso(const float* grid, int32_t grid_on_device, const int32_t dims[3], float voxel_size,
                       const float origin[3], float iso_value, float* out_vertices, int64_t vertex_capacity,
                       uint32_t* out_indices, int64_t index_capacity, int outputs, float** lib_v, uint32_t** lib_i,
                       int64_t* n_vertices, int64_t* n_indices, int32_t device, char* err, size_t errlen) {
    IsoErr e{err, errlen};
    if (err && errlen) err[0] = 0;
    if (!n_vertices || !n_indices || !dims || !origin) return e.set(GBSDF_EINVAL, "null argument");
    *n_vertices = 0;
    *n_indices = 0;
    const int dx = dims[0], dy = dims[1], dz = dims[2];
    if (dx < 2 || dy < 2 || dz < 2) return GBSDF_OK;  // no cube: an empty mesh (cuda_marching_cubes.cu:842-845)
    if (!grid) return e.set(GBSDF_EINVAL, "null grid");
    if (!(voxel_size > 0.0f) || !std::isfinite(voxel_size)) return e.set(GBSDF_EINVAL, "voxel size must be positive");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) {
        cudaGetLastError();
        return e.set(GBSDF_ENODEV, "no CUDA device available");
    }
    if (device < 0 || device >= ndev || device >= 64)
        return e.set(GBSDF_ENODEV, "device %d out of range", device);
    if (cudaSetDevice(device) != cudaSuccess) {
        cudaGetLastError();
        return e.set(GBSDF_ECUDA, "cudaSetDevice failed");
    }
    const long long N = (long long)dx * dy * dz;
    const long long groups = (long long)((dy + 3) / 4) * dz;  // the call's limit on dims: groups of four rows
    if (groups > 0x7fffffffLL) return e.set(GBSDF_EINVAL, "lattice too large (%lld row groups)", groups);
    const int wpr = (dx + 31) / 32;
    const IsoGeom G{dx, dy, dz, wpr, (long long)dy * dz, (long long)dy * dz * wpr, iso_value, iso_value + voxel_size,
                    !(iso_value + voxel_size - iso_value <= 0.0f)};
    const long long blocks = (G.nw + kIsoThreads - 1) / kIsoThreads;
    cudaError_t ce = cudaSuccess;
    std::lock_guard<std::mutex> lock(g_iso[device].mu);
    if (!g_iso[device].table) {
        if (!table_to_device()) {
            cudaGetLastError();
            return e.set(GBSDF_ECUDA, "triangle table upload failed");
        }
        g_iso[device].table = true;
    }
    IsoScratch s{g_iso[device]};
    // two passes over the same carving: sizing, then placing
    const float* g = grid;
    float* d_up = nullptr;
    unsigned* d_bits = nullptr;
    uint16_t* d_vpre = nullptr;
    uint2* d_tot = nullptr;
    ulonglong2* d_first = nullptr;
    IsoItem* d_items = nullptr;
    unsigned long long* d_sum = nullptr;  // vertices, triangles, items
    for (int pass = 0; pass < 2; ++pass) {
        if (!grid_on_device) d_up = s.get<float>((size_t)N, ce);
        d_bits = s.get<unsigned>((size_t)G.nw, ce);
        d_vpre = s.get<uint16_t>((size_t)G.nw, ce);
        d_tot = s.get<uint2>((size_t)blocks, ce);
        d_first = s.get<ulonglong2>((size_t)blocks, ce);
        d_items = s.get<IsoItem>((size_t)G.nw, ce);
        d_sum = s.get<unsigned long long>(3, ce);
        if (pass == 0) ce = s.commit();
    }
    if (ce != cudaSuccess) {
        cudaGetLastError();
        return e.set(GBSDF_ENOMEM, "device allocation failed: %s", cudaGetErrorString(ce));
    }
    cudaStream_t st = 0;
    if (!grid_on_device) {  // the reference's path: the host grid is uploaded
        ce = cudaMemcpyAsync(d_up, grid, (size_t)N * 4, cudaMemcpyHostToDevice, st);
        if (ce != cudaSuccess) return e.set(GBSDF_ECUDA, "grid upload: %s", cudaGetErrorString(ce));
        g = d_up;
    }
    // about 64 CTAs per SM (16 read the grid 10% slower), one a plane at least
    const int by = std::min(dz, 65535), rows8 = (dy + kIsoWarps - 1) / kIsoWarps;
    const int bx = std::max(1, std::min(rows8, (152 * 64 + by - 1) / by));
    GBSDF_COUNT_LAUNCH();
    iso_bits_kernel<<<dim3(bx, by), kIsoThreads, 0, st>>>(g, G, d_bits, d_sum + 2);
    GBSDF_COUNT_LAUNCH();
    iso_count_kernel<<<(unsigned)blocks, kIsoThreads, 0, st>>>(G, d_bits, d_vpre, d_tot, d_items, d_sum + 2);
    GBSDF_COUNT_LAUNCH();
    const long long share = std::max<long long>((blocks + 151) / 152, kScanThreads);
    iso_scan_kernel<<<(unsigned)((blocks + share - 1) / share), kScanThreads, 0, st>>>(d_tot, blocks, share, d_first,
                                                                                      d_sum);
    ce = cudaGetLastError();  // launch errors are not reported by the synchronisation
    if (ce != cudaSuccess) return e.set(GBSDF_ECUDA, "iso-surface count launch: %s", cudaGetErrorString(ce));
    unsigned long long sum[3] = {0, 0, 0};
    cudaMemcpyAsync(sum, d_sum, sizeof(sum), cudaMemcpyDeviceToHost, st);
    ce = cudaStreamSynchronize(st);
    if (ce != cudaSuccess) return e.set(GBSDF_ECUDA, "iso-surface count: %s", cudaGetErrorString(ce));
    const long long V = (long long)sum[0], T = (long long)sum[1], n_items = (long long)sum[2];
    *n_vertices = V;
    *n_indices = 3 * T;
    if (V > 0xffffffffLL) return e.set(GBSDF_EINVAL, "%lld vertices exceed 32-bit indices", V);
    if (V == 0 || T == 0) {
        *n_vertices = 0;
        *n_indices = 0;
        return GBSDF_OK;
    }
    if (outputs == 2) {  // library-owned: grow the cache's mesh region
        IsoCache& c = g_iso[device];
        const size_t vb = ((size_t)V * 12 + 255) & ~size_t(255), need = vb + (size_t)T * 12;
        if (need > c.out_bytes) {
            if (c.out) cudaFree(c.out);
            c.out = nullptr;
            c.out_bytes = 0;
            ce = cudaMalloc(&c.out, need);
            if (ce != cudaSuccess) {
                cudaGetLastError();
                return e.set(GBSDF_ENOMEM, "device allocation failed: %s", cudaGetErrorString(ce));
            }
            c.out_bytes = need;
        }
        out_vertices = static_cast<float*>(c.out);
        out_indices = reinterpret_cast<uint32_t*>(static_cast<char*>(c.out) + vb);
        vertex_capacity = V;
        index_capacity = 3 * T;
        *lib_v = out_vertices;
        *lib_i = out_indices;
    }
    const bool outputs_on_device = outputs != 0;
    if (vertex_capacity < V || index_capacity < 3 * T || !out_vertices || !out_indices)
        return e.set(GBSDF_EINVAL, "outputs must hold %lld vertices and %lld indices", V, 3 * T);
    float* d_v = out_vertices;
    uint32_t* d_i = out_indices;
    void* stage = nullptr;  // host outputs: device staging of the mesh, per call
    if (!outputs_on_device) {
        ce = cudaMalloc(&stage, (size_t)V * 12 + (size_t)T * 12 + 256);
        if (ce != cudaSuccess) {
            cudaGetLastError();
            return e.set(GBSDF_ENOMEM, "device allocation failed: %s", cudaGetErrorString(ce));
        }
        d_v = static_cast<float*>(stage);
        d_i = reinterpret_cast<uint32_t*>(static_cast<char*>(stage) + (((size_t)V * 12 + 255) & ~size_t(255)));
    }
    struct FreeStage {
        void* p;
        ~FreeStage() {
            if (p) cudaFree(p);
        }
    } free_stage{stage};
    GBSDF_COUNT_LAUNCH();
    iso_emit_kernel<<<dim3((unsigned)((n_items + kEmitThreads - 1) / kEmitThreads), 2), kEmitThreads, 0, st>>>(
        g, G, voxel_size, origin[0], origin[1], origin[2], d_bits, d_vpre, d_first, d_items, n_items, d_v, d_i);
    ce = cudaGetLastError();
    if (ce == cudaSuccess && !outputs_on_device) {
        ce = cudaMemcpyAsync(out_vertices, d_v, (size_t)V * 12, cudaMemcpyDeviceToHost, st);
        if (ce == cudaSuccess) ce = cudaMemcpyAsync(out_indices, d_i, (size_t)T * 12, cudaMemcpyDeviceToHost, st);
    }
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(st);
    if (ce != cudaSuccess) return e.set(GBSDF_ECUDA, "iso-surface emit: %s", cudaGetErrorString(ce));
    return GBSDF_OK;
}


extern "C" {

int gbsdf_iso_surface_table(int8_t* out_table) {
    if (!out_table) return GBSDF_EINVAL;
    std::call_once(g_tri_once, mc_table_init);
    std::memcpy(out_table, g_tri, sizeof(g_tri));
    return GBSDF_OK;
}

int gbsdf_extract_iso_surface(const float* grid, int32_t grid_on_device, const int32_t dims[3], float voxel_size,
                              const float origin[3], float iso_value, float* out_vertices, int64_t vertex_capacity,
                              uint32_t* out_indices, int64_t index_capacity, int32_t outputs_on_device,
                              int64_t* n_vertices, int64_t* n_indices, int32_t device, char* err, size_t errlen) {
    return extract_iso(grid, grid_on_device, dims, voxel_size, origin, iso_value, out_vertices, vertex_capacity,
                       out_indices, index_capacity, outputs_on_device ? 1 : 0, nullptr, nullptr, n_vertices, n_indices,
                       device, err, errlen);
}

int gbsdf_extract_iso_surface_device(const float* grid, int32_t grid_on_device, const int32_t dims[3],
                                     float voxel_size, const float origin[3], float iso_value, float** vertices_dev,
                                     uint32_t** indices_dev, int64_t* n_vertices, int64_t* n_indices, int32_t device,
                                     char* err, size_t errlen) {
    if (!vertices_dev || !indices_dev) {
        if (err && errlen) std::snprintf(err, errlen, "null output pointers");
        return GBSDF_EINVAL;
    }
    *vertices_dev = nullptr;
    *indices_dev = nullptr;
    return extract_iso(grid, grid_on_device, dims, voxel_size, origin, iso_value, nullptr, 0, nullptr, 0, 2,
                       vertices_dev, indices_dev, n_vertices, n_indices, device, err, errlen);
}

// shared set-up of the two reductions: device, grid on the device, a small result block
struct SdfReduce {
    float* dgrid = nullptr;
    unsigned long long* res = nullptr;  // [0] inside count, [1] min key (low 32), [2] best seed key
    ~SdfReduce() {
        if (dgrid) cudaFree(dgrid);
        if (res) cudaFree(res);
    }
};

static int sdf_reduce_setup(const float* grid, int32_t on_dev, long long n, int32_t device, IsoErr& e,
                            SdfReduce& r, const float** g) {
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) {
        cudaGetLastError();
        return e.set(GBSDF_ENODEV, "no CUDA device available");
    }
    if (device < 0 || device >= ndev) return e.set(GBSDF_ENODEV, "device %d out of range", device);
    if (cudaSetDevice(device) != cudaSuccess) {
        cudaGetLastError();
        return e.set(GBSDF_ECUDA, "cudaSetDevice failed");
    }
    cudaError_t ce = cudaMalloc(&r.res, 3 * sizeof(unsigned long long));
    if (ce == cudaSuccess && !on_dev) {  // the reference's path: the host grid is uploaded
        ce = cudaMalloc(&r.dgrid, (size_t)n * 4);
        if (ce == cudaSuccess) ce = cudaMemcpy(r.dgrid, grid, (size_t)n * 4, cudaMemcpyHostToDevice);
    }
    if (ce != cudaSuccess) {
        cudaGetLastError();
        return e.set(ce == cudaErrorMemoryAllocation ? GBSDF_ENOMEM : GBSDF_ECUDA, "device set-up: %s",
                     cudaGetErrorString(ce));
    }
    *g = on_dev ? grid : r.dgrid;
    const unsigned long long init[3] = {0ull, 0xffffffffull, ~0ull};
    ce = cudaMemcpy(r.res, init, sizeof(init), cudaMemcpyHostToDevice);
    if (ce != cudaSuccess) return e.set(GBSDF_ECUDA, "device set-up: %s", cudaGetErrorString(ce));
    GBSDF_COUNT_LAUNCH();
    sdf_inside_min_kernel<<<152 * 8, 256>>>(*g, n, &r.res[0], reinterpret_cast<unsigned*>(&r.res[1]));
    return GBSDF_OK;
}

static float ordered_to_float(unsigned k) {
    const unsigned u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}

int gbsdf_interior_volume(const float* grid, int32_t grid_on_device, int64_t n_voxels, float voxel_size,
                          float* out_volume_mm3, int64_t* out_inside_voxels, int32_t device, char* err,
                          size_t errlen) {
    IsoErr e{err, errlen};
    if (err && errlen) err[0] = 0;
    if (!out_volume_mm3) return e.set(GBSDF_EINVAL, "null output");
    *out_volume_mm3 = 0.0f;
    if (out_inside_voxels) *out_inside_voxels = 0;
    if (!grid || n_voxels <= 0) return e.set(GBSDF_EINVAL, "empty grid");  // the reference returns false
    SdfReduce r;
    const float* g = nullptr;
    int rc = sdf_reduce_setup(grid, grid_on_device, n_voxels, device, e, r, &g);
    if (rc != GBSDF_OK) return rc;
    unsigned long long cnt = 0;
    const cudaError_t ce = cudaMemcpy(&cnt, &r.res[0], 8, cudaMemcpyDeviceToHost);
    if (ce != cudaSuccess) return e.set(GBSDF_ECUDA, "interior volume: %s", cudaGetErrorString(ce));
    const float vox = voxel_size * voxel_size * voxel_size;
    *out_volume_mm3 = (float)cnt * vox;
    if (out_inside_voxels) *out_inside_voxels = (int64_t)cnt;
    return GBSDF_OK;
}

int gbsdf_find_default_seed(const float* grid, int32_t grid_on_device, const int32_t dims[3],
                            const int32_t min_coord[3], float voxel_size, const float min_p[3], const float max_p[3],
                            float desired_margin, float out_seed[3], int32_t device, char* err, size_t errlen) {
    IsoErr e{err, errlen};
    if (err && errlen) err[0] = 0;
    if (!dims || !min_coord || !min_p || !max_p || !out_seed) return e.set(GBSDF_EINVAL, "null argument");
    const float cx = (min_p[0] + max_p[0]) * 0.5f, cy = (min_p[1] + max_p[1]) * 0.5f;
    out_seed[0] = cx;
    out_seed[1] = cy;
    out_seed[2] = min_p[2] + 2.0f * voxel_size;
    const long long n = (long long)dims[0] * dims[1] * dims[2];
    if (!grid || dims[0] <= 0 || dims[1] <= 0 || dims[2] <= 0) return e.set(GBSDF_EINVAL, "empty grid");
    SdfReduce r;
    const float* g = nullptr;
    int rc = sdf_reduce_setup(grid, grid_on_device, n, device, e, r, &g);
    if (rc != GBSDF_OK) return rc;
    unsigned long long mk = 0;
    cudaError_t ce = cudaMemcpy(&mk, &r.res[1], 8, cudaMemcpyDeviceToHost);
    if (ce != cudaSuccess) return e.set(GBSDF_ECUDA, "default seed: %s", cudaGetErrorString(ce));
    const float mn = std::min(1e30f, ordered_to_float((unsigned)mk));
    const float margin = (mn < 0.0f) ? std::max(desired_margin, mn * 0.65f) : (mn + voxel_size);
    GBSDF_COUNT_LAUNCH();
    sdf_seed_kernel<<<152 * 8, 256>>>(g, dims[0], dims[1], dims[2], min_coord[0], min_coord[1], min_coord[2],
                                      voxel_size, min_p[2], cx, cy, margin, &r.res[2]);
    unsigned long long best = ~0ull;
    ce = cudaMemcpy(&best, &r.res[2], 8, cudaMemcpyDeviceToHost);
    if (ce != cudaSuccess) return e.set(GBSDF_ECUDA, "default seed: %s", cudaGetErrorString(ce));
    if (best != ~0ull) {
        const long long i = (long long)(best & 0xffffffffull);
        if (i < n) {
            const int x = (int)(i % dims[0]), y = (int)((i / dims[0]) % dims[1]),
                      z = (int)(i / ((long long)dims[0] * dims[1]));
            out_seed[0] = (float)(min_coord[0] + x) * voxel_size;
            out_seed[1] = (float)(min_coord[1] + y) * voxel_size;
            out_seed[2] = (float)(min_coord[2] + z) * voxel_size;
        }
    }
    return GBSDF_OK;
}

}  // extern "C"
