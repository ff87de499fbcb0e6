// batch.h — the batched persistent renderer (batch.cu): many contexts, one
// launch.  Shared between batch.cu and capi.cu (which owns orn_context).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "ornament_cuda.h"
#include "pt_scene.h"

namespace orn {

constexpr uint32_t kMaxBatch = 64;   // scenes per launch (their views live in shared memory)

// One context's part of a batched frame: what orn_render would launch for
// it (all of this render()'s passes in one go).
struct BatchView {
    SceneDev scene;
    orn_constant_params cp;    // current_iteration = first pass of the frame
    uint32_t spp;              // passes this frame
    uint32_t pixel_begin;      // first pixel of this context in the frame's pixel space
    float4* acc;
    float4* fb;
    uint32_t* rng;
};

// Does the host side of orn_render for `ctx` (checks, targets, camera-dirty
// restart, current_iteration bookkeeping) and fills `view`; the batch stream
// is ordered after the context's queued work.  Returns an ORN_* status.
// With commit = false the context is left as it was (the autotuner's
// scratch frames).
int batch_prepare(orn_context* ctx, BatchView* view, bool* fast_slabs, uint32_t* semantics, int* device,
                  cudaStream_t batch_stream, bool commit);
// Orders the context's later work after `done` (recorded on the batch stream).
int batch_finish(orn_context* ctx, cudaEvent_t done);

struct BatchConfig {
    int block;           // 64, 128 or 192 threads
    int blocks_per_sm;   // resident blocks per SM the grid is sized for
    int shade_threshold; // ready lanes needed before a warp shades
};

// What every context of a batch allows: the exact slab test only, the FMNMX
// form, or the near-first trees (which imply that form).
enum { BATCH_EXACT = 0, BATCH_FAST = 1, BATCH_NEAR = 2 };

// What a batch walks: the near-first trees where all contexts have them and
// those that gain by it (NEAR_BATCH) have more to walk than the others.  (A
// context that does not gain loses up to 15 %, one that does gains 5 to 50; taken
// only when all gain, one SAH tree kept a batch of any others from it.)
struct BatchWalk {
    bool fast = true, near = true;
    double gain = 0.0, lose = 0.0;
    void add(const BatchView& v, bool fast_slabs) {
        fast = fast && fast_slabs;
        near = near && v.scene.near != NEAR_NONE;
        const double work = (double)v.cp.width * v.cp.height * v.spp * (1.0 + v.scene.visits);
        (v.scene.near >= NEAR_BATCH ? gain : lose) += work;
    }
    int slabs() const {
        if (!fast) return BATCH_EXACT;
        return near && gain > lose ? BATCH_NEAR : BATCH_FAST;
    }
};

// Launches one batched frame (views already in device memory).
cudaError_t launch_batch(const BatchView* views, uint32_t nviews, uint32_t total_pixels, uint32_t* work_counter,
                         uint32_t* error, int semantics, int slabs, const BatchConfig& cfg, cudaStream_t s);
// The largest resident block count per SM for a block size (0 if unknown).
int batch_max_blocks_per_sm(int block, int semantics, int slabs);

}  // namespace orn
