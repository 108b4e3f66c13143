// signs.h — the host side of the exact sign decisions, shared by single builds (engine.cu) and
// planned batches (batch.cu): decide every voxel marked in U, and run the stratified probes'
// patch rounds.
#pragma once
#include "gbsdf_internal.h"

namespace gbsdf {

// A grow-only device buffer.
struct Buf {
    void* p = nullptr;
    size_t bytes = 0;
};
cudaError_t ensure(Buf& b, size_t bytes);
void release(Buf& b);

// Scratch of the crossings and caps (edge table, caps, their clusters, crossing planes).
struct CapScratch {
    Buf etab, caps, cfw, cross;
};

// One build's sign state: where its arrays are, and the crossings and caps once they are made.
struct SignWork {
    const float* t9 = nullptr;
    long long T = 0;
    Lattice L{};
    const float* dist = nullptr;  // unsigned distances, squared when dist_sq
    int dist_sq = 0;
    float stol = 0.0f;            // voxels within this many voxels of the surface are inside
    int* grid = nullptr;          // an int per voxel, scratch
    uint32_t *U = nullptr, *S = nullptr;
    long long *list = nullptr, *recheck = nullptr;
    long long cap = 0;            // capacity of both
    DevState *ds = nullptr, *hs = nullptr;
    const Fwn* fwn = nullptr;     // null: every decision by the sum over every triangle
    int num_sms = 0;
    cudaStream_t st = nullptr;
    CapScratch* scratch = nullptr;
    bool tried = false, capped = false;
    long long B = 0;
    Fwn capf{};
    Crossings x{};
};

// Decides every voxel marked in U (its marks are cleared; E, when given, records them).
// `patching`: a patch round's marks. Returns a CUDA error, or cudaErrorUnknown when the passes
// do not drain the marks.
cudaError_t decide_marked(SignWork& w, uint32_t* E, bool patching);
// One generation of the stratified probes (no host round trip).
void enqueue_probe(SignWork& w, int gen, bool escalate);
// The rest of the probe generations after `gen` (whose plan is in *w.hs): patch rounds and
// probes until they come back clean or diverge; *w.hs holds the last state.
cudaError_t finish_probes(SignWork& w, int gen, uint32_t* E);

}  // namespace gbsdf
