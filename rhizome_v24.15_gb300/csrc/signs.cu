// signs.cu — the host side of the exact sign decisions (signs.h).
#include <algorithm>

#include "gbsdf_device.cuh"
#include "signs.h"

namespace gbsdf {

#define SG_CK(call)                                  \
    do {                                             \
        const cudaError_t _e = (call);               \
        if (_e != cudaSuccess) return _e;            \
    } while (0)

cudaError_t ensure(Buf& b, size_t bytes) {
    if (bytes <= b.bytes && b.p) return cudaSuccess;
    release(b);
    const size_t want = bytes + bytes / 8 + 256;
    const cudaError_t err = cudaMalloc(&b.p, want);
    if (err != cudaSuccess) {
        cudaGetLastError();
        b.p = nullptr;
        return err;
    }
    b.bytes = want;
    return cudaSuccess;
}

void release(Buf& b) {
    if (b.p) cudaFree(b.p);
    b = Buf{};
}

namespace {

// Makes the crossings and caps of the build. Two kinds of mesh keep to their own clusters: those whose
// boundary is long (unwelded soups; more than one unmatched edge for every four triangles), whose
// caps are wide fans over one another and decide little, and those with more than one cap for
// every eight marked voxels, where a brick's caps cost more than its voxels' walks. So does a
// build that finds no memory for them. Without / with them, ms, every voxel of 64^3: sphere of 10k triangles,
// 8% missing (0.24 unmatched edges a triangle) 0.9 / 0.9, 12% 1.7 / 2.8, 20% 1.6 / 7.8, 40%
// 1.4 / 31; of 88k and 352k triangles, 8% missing, walks / caps and walks: 4.6 / 4.4 (13 voxels a
// cap), 6.9 / 11.6 (3.3).
cudaError_t make_capped(SignWork& w, long long marks) {
    CapScratch& s = *w.scratch;
    if (!w.counted) {
        w.counted = true;
        w.closable = false;
        if (w.T > (1ll << 26)) return cudaSuccess;  // the table is 12 bytes a slot, over six slots a triangle
        if (ensure(s.etab, edge_table_bytes(w.T)) != cudaSuccess) return cudaSuccess;
        launch_edge_table(w.t9, w.T, s.etab.p, w.st);
        unsigned long long counts[2] = {0, 0};
        SG_CK(cudaMemcpyAsync(counts, s.etab.p, sizeof(counts), cudaMemcpyDeviceToHost, w.st));
        SG_CK(cudaStreamSynchronize(w.st));
        w.B = (long long)counts[0];
        w.closable = counts[1] == 0 && w.B <= w.T / 4;
    }
    if (!w.closable || 8 * w.B > marks) return cudaSuccess;
    w.closable = false;  // (tried once)
    const float* caps9 = nullptr;
    if (w.B > 0) {
        if (ensure(s.caps, caps_bytes(w.B)) != cudaSuccess || ensure(s.cfw, fwn_bytes(w.B, 1)) != cudaSuccess)
            return cudaSuccess;
        caps9 = launch_caps(w.t9, w.T, s.etab.p, w.B, s.caps.p, w.st);
        w.capf = fwn_carve(s.cfw.p, w.B, 1);
        launch_fwn_build(caps9, w.B, w.L, w.capf, w.st);
    }
    if (ensure(s.cross, crossing_bytes(w.L)) != cudaSuccess) return cudaSuccess;
    w.x = launch_crossings(w.t9, w.T, caps9, w.B, w.L, w.grid, s.cross.p, w.st);
    SG_CK(cudaGetLastError());
    w.capped = true;
    return cudaSuccess;
}

}  // namespace

cudaError_t decide_marked(SignWork& w, uint32_t* E, bool patching) {
    const int only = patching ? 1 : 0;
    bool closed = false;  // the crossings and caps have decided what they can of these marks
    for (int pass = 0; pass < 1 << 20; ++pass) {
        SG_CK(cudaMemsetAsync(&w.ds->listed, 0, kPassCounters, w.st));
        if (w.fwn) launch_list_blocks(w.U, w.L, w.list, w.cap, w.ds, only, w.st);
        else launch_list_unknown(w.U, w.S, w.L, w.list, w.cap, w.ds, only, w.st, E);
        SG_CK(cudaMemcpyAsync(w.hs, w.ds, sizeof(DevState), cudaMemcpyDeviceToHost, w.st));
        SG_CK(cudaStreamSynchronize(w.st));
        const long long n = std::min<long long>((long long)w.hs->listed, w.cap);
        if (n <= 0) return cudaSuccess;
        if (w.fwn) {
            const long long marks = (long long)w.hs->listed_voxels;
            if (!w.capped && w.closable && marks >= caps_min_voxels(w.L.N)) SG_CK(make_capped(w, marks));
            if (w.capped && !closed) {
                launch_capped_blocks(w.capf, w.B, w.L, w.x, w.U, w.S, E, w.list, w.cap, only, w.dist, w.dist_sq, w.stol,
                                     w.ds, w.num_sms, w.st);
                SG_CK(cudaGetLastError());
                closed = true;
                continue;
            }
            if (by_voxels(marks, w.T)) {
                SG_CK(cudaMemsetAsync(&w.ds->listed, 0, kPassCounters, w.st));
                launch_list_unknown(w.U, w.S, w.L, w.list, w.cap, w.ds, only, w.st, E);
                launch_winding(w.fwn, w.t9, w.T, w.L, w.list, w.cap, kGwnFixup, only, w.S, w.recheck, w.cap, w.dist,
                               w.dist_sq, w.stol, w.ds, w.num_sms, w.st);
            } else {
                launch_winding_blocks(*w.fwn, w.t9, w.T, w.L, w.U, w.S, E, w.list, w.cap, only, w.recheck, w.cap, w.dist,
                                      w.dist_sq, w.stol, w.ds, w.num_sms, w.st);
            }
        } else if (n < 64 * 1024) {
            launch_gwn_small(w.t9, w.T, w.L, w.list, w.cap, kGwnFixup, w.S, w.recheck, w.cap, w.dist, w.dist_sq, w.stol,
                             w.ds, n, w.st);
        } else {
            launch_gwn(w.t9, w.T, w.L, w.list, w.cap, kGwnFixup, only, w.S, w.recheck, w.cap, w.dist, w.dist_sq, w.stol,
                       w.ds, w.num_sms, w.st);
        }
        launch_gwn_recheck(w.t9, w.T, w.L, w.recheck, w.cap, kGwnFixup, w.S, w.ds, w.num_sms, w.st);
        SG_CK(cudaGetLastError());
        // blocks: the leftovers of a pass can outgrow their list too (their voxels stay marked)
        if (w.hs->list_overflow == 0 && (!w.fwn || w.hs->listed_voxels <= (unsigned long long)w.cap)) return cudaSuccess;
    }
    return cudaErrorUnknown;
}

void enqueue_probe(SignWork& w, int gen, bool escalate) {
    launch_verify_prepare(w.L, gen, w.U, w.list, w.ds, w.st);
    launch_winding(w.fwn, w.t9, w.T, w.L, w.list, w.cap, kGwnVerify, 0, w.S, w.recheck, w.cap, w.dist, w.dist_sq, w.stol,
                   w.ds, w.num_sms, w.st);
    launch_gwn_recheck(w.t9, w.T, w.L, w.recheck, w.cap, kGwnVerify, w.S, w.ds, w.num_sms, w.st);
    launch_verify_plan(gen, w.ds, w.st, escalate ? 1 : 0);
}

cudaError_t finish_probes(SignWork& w, int gen, uint32_t* E) {
    while (w.hs->verify_state == 0 && w.hs->patching && ++gen < kProbeGens) {
        launch_patch_mark(w.L, w.U, w.ds, w.st);
        SG_CK(decide_marked(w, E, true));
        enqueue_probe(w, gen, false);
        SG_CK(cudaMemcpyAsync(w.hs, w.ds, sizeof(DevState), cudaMemcpyDeviceToHost, w.st));
        SG_CK(cudaStreamSynchronize(w.st));
    }
    return cudaSuccess;
}

}  // namespace gbsdf
