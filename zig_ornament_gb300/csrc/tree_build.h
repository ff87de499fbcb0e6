// tree_build.h — the node arrays and trees of a scene (tree_build.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "ornament_cuda.h"
#include "pt_scene.h"

namespace orn {

// What the device passes over the node arrays found.
struct NodeFacts {
    uint32_t huge;   // an inner box is not finite or reaches 1e30 (no FMNMX slab test, no near-first trees)
};

// Writes the kernels' node array (scene->nodes: TLAS, then BLAS, four
// float4 each) from the blob's nodes and transforms on the device, and behind
// it the near-first trees when the blob allows and memory lasts (scene->near).
// The array is appended to *allocs.  Everything runs on `s`, finished on return.
cudaError_t build_scene_trees(const orn_scene_blob* blob, const float4* d_xforms, SceneDev* scene, NodeFacts* facts,
                              std::vector<void*>* allocs, cudaStream_t s);

}  // namespace orn
