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
    bool counted = false, closable = true;  // the mesh's boundary is counted; it can be closed by caps
    bool capped = false;
    long long B = 0;              // boundary edges, and caps
    Fwn capf{};
    Crossings x{};
};

// Whether `marks` voxels of a mesh of T triangles are walked one by one rather than taken by blocks
// of bricks. A block looks at its clusters once for all its voxels, which pays where they are many
// and the triangles in a brick few. Blocks / walks, ms (voxels marked): in columns through holes,
// vessel trees of 16k and 101k triangles 0.72 / 0.25 (3,840) and 1.73 / 0.45 (4,608), blob of 632k
// 13.2 / 1.3 (22,656) and 15.8 / 12.2 (234,496), sphere of 71k without a fifth of its triangles
// 5.2 / 7.5 (355,968), of 287k 35 / 12 (355,328) and 34 / 45 (1.5M); every voxel, sphere of 3k on
// 64^3 1.2 / 1.3 and on 96^3 2.5 / 4.5, of 90k 27 / 4.6 and 9.0 / 16, of 360k 248 / 23 (96^3) and
// 103 / 218 (200^3).
inline bool by_voxels(long long marks, long long T) { return marks <= (4 * T > (1ll << 18) ? 4 * T : (1ll << 18)); }

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
