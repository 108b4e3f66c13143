// tune.cu — the autotuner: sweep schedules per lattice class.
//
// The x sweep has six schedules and the y / z walks five, all with identical results
// (internal header, XSchedule / WSchedule). Which is fastest depends on the lattice (row
// length, CTAs per wave), the device and the field: the first round sweeps a band in a far
// field, where most updates are one-dimensional, later rounds a field where most warps
// need the 2D and 3D updates. The first build of a lattice class times each candidate on
// that build's own buffers on the field after the first round (phase 1) -- one warm-up and
// two timed launches each (x sweeps for the x schedules, z walks for the walk schedules),
// CUDA events on the build's stream -- and remembers the winners for the later rounds. The
// first round (phase 0) runs the default plan: timed on the band field alone the
// candidates' order did not hold over the round. A caller may still ask for a measured
// phase-0 plan (measure = true with phase 0). The exact eikonal has one plan per lattice
// (default_plan). A class is (device, row pitch a multiple of 16
// bytes, round(log2 voxels), round(log2 row length)). Timing writes only the destination
// copy, which the next sweep rewrites whole, and one change-flag slot.
#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <tuple>

#include "gbsdf_device.cuh"
#include "gbsdf_internal.h"

namespace gbsdf {
namespace {

using Key = std::tuple<int, int, int, int, int>;
std::mutex g_tune_mu;
std::map<Key, SweepPlan> g_tuned;

Key key_of(int device, const Lattice& L, int phase) {
    return Key{device, (L.px & 3) == 0 ? 1 : 0, (int)std::lround(std::log2((double)L.N)),
               (int)std::lround(std::log2((double)L.dims[0])), phase};
}

// The plan of a lattice without measurements: the first round of every build, a batch whose
// class no build has tuned, and every round of the exact eikonal, whose order is not that of
// the update the candidates are timed with. A schedule's narrow tiles run in place of the wide
// ones up to 1.5 wide tiles per SM, where those leave SMs idle or a nearly empty second wave.
// us per sweep, all six directions, wide -> narrow walks: 48^3 15.2 -> 11.0, 128^3 (32 tiles)
// 31.8 -> 19.9, 257 x 255 x 260 (144) 70.0 -> 53.0, 288^3 (162) 92 -> 74, 320^3 (200) 101 -> 90,
// 352^3 (242) 122.5 -> 121.4, 512^3 (512) 288 -> 298; then wide -> narrow x tiles: 128^3 (64
// tiles) 19.9 -> 19.0, 224^3 (196) 41.4 -> 38.8, 1024 x 64 x 64 (16) 50.9 -> 45.5, 257 x 255 x
// 260 (264) 53.0 -> 53.0, 320^3 (400) 89.5 -> 93.9. The exact update walks narrow everywhere:
// 128^3 73 -> 31, 257 x 255 x 260 146 -> 70, 400^3 285 -> 209, 512^3 430 -> 386 (its four
// chains per thread are branchy code that serialises).
SweepPlan default_plan(const Lattice& L, int rule, bool tma, bool wtma) {
    auto fills = [](int tiles) { return 2 * (long long)tiles <= 3 * 152; };
    const int dx = L.dims[0], dy = L.dims[1], dz = L.dims[2];
    SweepPlan p{kXCpAsync, kWCpAsync};
    if (tma) p.x = fills(((dy + 31) / 32) * ((dz + 7) / 8)) ? kXTmaNarrow : kXTmaPipe;
    if (wtma) p.w = rule != 0 || fills(((dx + 31) / 32) * ((std::max(dy, dz) + 15) / 16)) ? kWTmaNarrow : kWTmaVec2;
    return p;
}

}  // namespace

SweepPlan tuned_sweep_plan(int device, const Lattice& L, const float* src, float* dst, const GridMap* src_map,
                           const GridMap* dst_map,
                           DevState* ds, cudaStream_t st, bool measure, int phase, int rule) {
    const bool tma = src_map && src_map->valid, wtma = src_map && src_map->walk_valid;
    SweepPlan plan = default_plan(L, rule, tma, wtma);
    if ((!tma && !wtma) || rule != 0) return plan;
    const Key k = key_of(device, L, phase);
    {
        std::lock_guard<std::mutex> g(g_tune_mu);
        auto it = g_tuned.find(k);
        if (it != g_tuned.end()) return it->second;
    }
    if (!measure) return plan;
    cudaEvent_t a, b;
    if (cudaEventCreate(&a) != cudaSuccess) {
        cudaGetLastError();
        return plan;
    }
    if (cudaEventCreate(&b) != cudaSuccess) {
        cudaGetLastError();
        cudaEventDestroy(a);
        return plan;
    }
    const int slot = 63;  // a change-flag slot the reference round loop never uses
    // one warm-up and two timed launches of one directional sweep; < 0 on failure
    auto time_it = [&](int axis, int xs, int ws) -> float {
        launch_sweep(0, axis, 1, slot, src, dst, L, ds, st, src_map, dst_map, xs, ws);
        cudaEventRecord(a, st);
        for (int r = 0; r < 2; ++r) launch_sweep(0, axis, 1, slot, src, dst, L, ds, st, src_map, dst_map, xs, ws);
        cudaEventRecord(b, st);
        float ms = -1.0f;
        if (cudaEventSynchronize(b) != cudaSuccess || cudaEventElapsedTime(&ms, a, b) != cudaSuccess) {
            cudaGetLastError();
            return -1.0f;
        }
        return ms;
    };
    if (tma) {
        float best = 1e30f;
        for (int cand : {kXCpAsync, kXTmaRing, kXTmaPipe, kXTmaPipe2, kXTmaWide, kXTmaNarrow}) {
            const float ms = time_it(0, cand, plan.w);
            if (ms >= 0.0f && ms < best) {
                best = ms;
                plan.x = cand;
            }
        }
    }
    if (wtma) {
        float best = 1e30f;
        for (int cand : {kWCpAsync, kWTmaPipe, kWTmaVec, kWTmaVec2, kWTmaNarrow}) {
            const float ms = time_it(2, plan.x, cand);
            if (ms >= 0.0f && ms < best) {
                best = ms;
                plan.w = cand;
            }
        }
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    std::lock_guard<std::mutex> g(g_tune_mu);
    g_tuned[k] = plan;
    return plan;
}

}  // namespace gbsdf
