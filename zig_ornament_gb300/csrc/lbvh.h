// lbvh.h — GPU BLAS construction (lbvh.cu), called by the host builder
// (bvh_build.cpp) for orn_scene_desc.builder = ORN_BVH_LBVH.
#pragma once

#include <stdint.h>

#include "ornament_cuda.h"

namespace orn {

// One mesh: `tri` holds n triangles as 9 floats (v0, v1, v2, object space);
// its 2n - 1 nodes go to `out` in the reference's format (post-order, root
// last; child ids are node_offset + slot, triangle ids first_global + index).
struct LbvhJob {
    const float* tri;
    uint32_t n;
    uint32_t first_global, node_offset;
    orn_bvh_node* out;
};

// Builds the BLASes of `count` meshes on the current CUDA device.  Returns ORN_*.
int lbvh_build_all(const LbvhJob* jobs, size_t count);

}  // namespace orn
