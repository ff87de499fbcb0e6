// tree_build.cu — the device side of scene creation: the kernels' node array,
// and the trees that pt_near.cuh traverses.
//
//   1. The blob's nodes go to the device as they are.  A pass finds every node's
//      parent and checks what the near-first traversal's proof of equal results
//      needs: each stored box has its lower corner first and holds the boxes
//      stored below it, a triangle's box is that of its vertices, no node has
//      two parents, and no walk can need more than the reference's 64 stack
//      entries.  A blob without one of these (other builders' padding, shared
//      subtrees) keeps the reference's walk, and so does one whose new trees do
//      not fit in memory: nothing is allocated for good until they are decided.
//   2. Every triangle finds the mesh it belongs to by its parents; triangles
//      and TLAS leaves are sorted by (tree, Morton code of the box centre).
//   3. Binary trees by parallel locally-ordered clustering (Meister and
//      Bittner, "Parallel Locally-Ordered Clustering for Bounding Volume
//      Hierarchy Construction", TVCG 2018), all meshes and the TLAS in the
//      same passes: each cluster picks the neighbour within kRadius places of
//      the same tree whose union box has the least area; pairs that pick each
//      other merge.  The last kSmallClusters are merged by one block in
//      shared memory.
//   4. The kernels' node array (pt_scene.h) is written: the blob's nodes, in
//      place if they are all there is, and the new ones behind them as they are
//      numbered: leaves in Morton order, then inner nodes round by round.
//      (Treelets of eight stored together, top-down: 77.2 against 77.0 ms for 16
//      passes of the 1080p scene, and creation 5.6 against 4.5 ms, of a small
//      scene 1.3 against 0.6.)
//
// Results do not depend on these trees (pt_near.cuh has the exception), only
// speed does; near_level has who walks them.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_select.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "tree_build.h"

namespace orn {
namespace {

constexpr uint32_t kNone = 0xffffffffu;
constexpr uint32_t kTlasTree = 0x3fffffffu;   // tree id of the TLAS (meshes: their root's BLAS index)
// Cached frames of scenes of this many nodes (1 MB, more than an L1) are taken to
// spend more on walking than on shading, and keep the shading code of their own
// (SplitGeom).  Measured from 40 to 563 k nodes; on either side of the line what
// is taken there is the faster one or within 1 %.
constexpr uint32_t kLargeScene = 16384;
constexpr uint32_t kDepthLimit = 64;          // the reference's stack entries
constexpr int kRadius = 16;
constexpr int kNnBlock = 256;
constexpr uint32_t kSmallClusters = 2048;
constexpr int kSmallBlock = 1024;
constexpr uint32_t kChosenRounds = 64;   // then neighbours merge in pairs, whatever their boxes
constexpr uint32_t kRoundsPerSync = 4;
constexpr uint32_t kOwnBoxMark = 0x80000000u;   // a leaf's box is not its triangle's own
constexpr uint32_t kMostSlivers = 64;
constexpr float kSliver = 1024.0f;
// What triangle_pad and shapes_kernel allow for.
constexpr float kPadTriangle = 0x1p-20f, kPadMove = 0x1p-20f, kPadSphere = 0x1p-19f;
constexpr double kMostMiss = 0x1p-12, kMostTurn = 0x1p12;
constexpr uint32_t kNearDepthLimit = kNearStackSize;   // levels of TLAS and BLAS together (one entry each)

// Counters and flags of one build (device; read back between phases).
struct State {
    uint32_t bad;         // the blob lacks something the near-first traversal needs
    uint32_t huge;
    uint32_t slivers;
    uint32_t prims;       // triangles that belong to a mesh, and reachable TLAS leaves
    float turn;           // SceneDev::near_turn
    float reach;          // of SceneDev::near_reach, the shapes' share
    float slide;          // SceneDev::near_slide
    float world;          // largest |coordinate| of the TLAS leaves' boxes
    uint32_t trees;       // meshes with triangles, and the TLAS
    uint32_t blas_depth, tlas_depth;
    uint32_t next_node;   // inner nodes made
    uint32_t meshes;      // mesh leaves written
    uint32_t clusters;    // left to merge
    uint32_t near_depth[2];   // levels of the deepest BLAS, and of the TLAS
    uint32_t root;        // reference of the TLAS root
    uint32_t shapes_box[6];   // keys of the corners of the ordinary shapes' box (ordinary_kernel)
    uint32_t large_shapes;   // left out of it
    float visits[4];      // expected of a ray: the blob's TLAS and BLASes, the new ones
};

static_assert(sizeof(State) <= 256, "the space before the types");

// Adds a warp's half box areas (lanes without one: 0) to *sum.
__device__ __forceinline__ void add_area(float* sum, float a) {
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    if ((threadIdx.x & 31u) == 0u && a != 0.0f) atomicAdd(sum, a);
}
__device__ __forceinline__ float half_area(float x, float y, float z) { return x * y + y * z + z * x; }

__global__ void types_kernel(const orn_bvh_node* __restrict__ nodes, uint32_t n, uint8_t* __restrict__ types) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) types[i] = (uint8_t)nodes[i].node_type;
}

// The kernels' node array.  A triangle keeps its vertices as given, so
// triangles sharing an edge see the same floats (the watertight test relies
// on it), and the two edges the reference's test subtracts on the fly
// (bvh.hip.h:81-82) — the same single-precision subtractions.
// (`out` may be the blob's nodes themselves: a thread reads its own node, and of
// others the types only.)
__global__ void relayout_kernel(const orn_bvh_node* nodes, uint32_t T, uint32_t B, const uint8_t* __restrict__ types,
                                const float4* __restrict__ xforms, float4* out, State* st) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= T + B) return;
    const bool top = i < T;
    const orn_bvh_node n = nodes[i];
    auto ref = [&](uint32_t k) { return k | ((uint32_t)types[k] << 30); };
    const float* a = n.left_aabb_min_or_v0;
    const float* b = n.left_aabb_max_or_v1;
    const float* c = n.right_aabb_min_or_v2;
    const float* e = n.right_aabb_max_or_v3;
    float4* o = out + (size_t)i * 4;
    if (n.node_type == ORN_NODE_INTERNAL) {
        const uint32_t off = top ? 0u : T;
        o[0] = make_float4(a[0], a[1], a[2], __uint_as_float(ref(off + n.left_or_custom_id)));
        o[1] = make_float4(b[0], b[1], b[2], __uint_as_float(ref(off + n.right_or_material_index)));
        o[2] = make_float4(c[0], c[1], c[2], __uint_as_float(ORN_NODE_INTERNAL));
        o[3] = make_float4(e[0], e[1], e[2], 0.0f);
        bool ok = true;
        for (int k = 0; k < 3; ++k)
            ok = ok && fabsf(a[k]) < 1e30f && fabsf(b[k]) < 1e30f && fabsf(c[k]) < 1e30f && fabsf(e[k]) < 1e30f;
        if (!ok) st->huge = 1u;
    } else if (n.node_type == ORN_NODE_TRIANGLE) {
        o[0] = make_float4(a[0], a[1], a[2], __uint_as_float(n.left_or_custom_id));
        o[1] = make_float4(b[0], b[1], b[2], c[0] - a[0]);
        o[2] = make_float4(c[0], c[1], c[2], c[1] - a[1]);
        o[3] = make_float4(b[0] - a[0], b[1] - a[1], b[2] - a[2], c[2] - a[2]);
    } else {   // sphere / mesh leaf: inverse rows 0..2 inline
        const float4* m = xforms + (size_t)n.transform_id * 2 * 4;
        const float4 r0 = m[0], r1 = m[1], r2 = m[2];
        const uint32_t root = n.node_type == ORN_NODE_MESH ? ref(T + n.left_or_custom_id) : 0u;
        o[0] = r0;
        o[1] = r1;
        o[2] = make_float4(r2.x, r2.y, r2.z, __uint_as_float(n.node_type));
        o[3] = make_float4(r2.w, __uint_as_float(n.right_or_material_index), __uint_as_float(n.transform_id),
                           __uint_as_float(root));
    }
}

__device__ __forceinline__ void stored_box(const orn_bvh_node& n, bool right, float* lo, float* hi) {
    for (int k = 0; k < 3; ++k) {
        lo[k] = right ? n.right_aabb_min_or_v2[k] : n.left_aabb_min_or_v0[k];
        hi[k] = right ? n.right_aabb_max_or_v3[k] : n.left_aabb_max_or_v1[k];
    }
}
__device__ __forceinline__ void triangle_box(const orn_bvh_node& n, float* lo, float* hi) {
    for (int k = 0; k < 3; ++k) {
        const float a = n.left_aabb_min_or_v0[k], b = n.left_aabb_max_or_v1[k], c = n.right_aabb_min_or_v2[k];
        lo[k] = fminf(fminf(a, b), c);
        hi[k] = fmaxf(fmaxf(a, b), c);
    }
}

// Parents (bit 31: the right child) of the children of nodes[0..n), and the
// checks on their boxes.
__global__ void parents_kernel(const orn_bvh_node* __restrict__ nodes, uint32_t n, uint32_t* __restrict__ parent,
                               State* st) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const orn_bvh_node nd = nodes[i];
    if (nd.node_type != ORN_NODE_INTERNAL) return;
    bool ok = true;
    for (int side = 0; side < 2; ++side) {
        const uint32_t c = side ? nd.right_or_material_index : nd.left_or_custom_id;
        if (atomicExch(&parent[c], i | (side ? 0x80000000u : 0u)) != kNone) ok = false;
        float lo[3], hi[3];
        stored_box(nd, side != 0, lo, hi);
        // (a sphere of negative radius has its box the wrong way round: the slab
        // test takes it as it is, but no box above it holds it)
        for (int k = 0; k < 3; ++k) ok = ok && lo[k] <= hi[k] && lo[k] > -1e30f && hi[k] < 1e30f;
        const orn_bvh_node ch = nodes[c];
        if (ch.node_type == ORN_NODE_INTERNAL) {
            for (int s2 = 0; s2 < 2; ++s2) {
                float clo[3], chi[3];
                stored_box(ch, s2 != 0, clo, chi);
                for (int k = 0; k < 3; ++k) ok = ok && clo[k] >= lo[k] && chi[k] <= hi[k];
            }
        } else if (ch.node_type == ORN_NODE_TRIANGLE) {
            float tlo[3], thi[3];
            triangle_box(ch, tlo, thi);
            for (int k = 0; k < 3; ++k) ok = ok && tlo[k] == lo[k] && thi[k] == hi[k];
        }
    }
    if (!ok) st->bad = 1u;
}

__global__ void mark_roots_kernel(const orn_bvh_node* __restrict__ tlas, uint32_t T, uint8_t* __restrict__ is_root) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < T && tlas[i].node_type == ORN_NODE_MESH) is_root[tlas[i].left_or_custom_id] = 1;
}

__device__ __forceinline__ uint32_t spread3(uint32_t v) {   // 10 bits to every third bit
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    return (v | (v << 2)) & 0x09249249u;
}
__device__ __forceinline__ uint32_t morton30(const float* lo, const float* hi, const float* tlo, const float* thi) {
    uint32_t code = 0;
    for (int k = 0; k < 3; ++k) {
        const float ext = thi[k] - tlo[k];
        const float x = ext > 0.0f ? (0.5f * lo[k] + 0.5f * hi[k] - tlo[k]) / ext : 0.0f;
        code |= spread3((uint32_t)fminf(fmaxf(x * 1024.0f, 0.0f), 1023.0f)) << k;
    }
    return code;
}

// A triangle whose edges are so nearly parallel that its hit test can be off
// by far more than its distance to its box.
__device__ __forceinline__ bool is_sliver(const orn_bvh_node& n) {
    float e1[3], e2[3];
    for (int k = 0; k < 3; ++k) {
        e1[k] = n.left_aabb_max_or_v1[k] - n.left_aabb_min_or_v0[k];
        e2[k] = n.right_aabb_min_or_v2[k] - n.left_aabb_min_or_v0[k];
    }
    const float cx = e1[1] * e2[2] - e1[2] * e2[1], cy = e1[2] * e2[0] - e1[0] * e2[2], cz = e1[0] * e2[1] - e1[1] * e2[0];
    const float area = sqrtf(cx * cx + cy * cy + cz * cz);
    const float l1 = sqrtf(e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2]);
    const float l2 = sqrtf(e2[0] * e2[0] + e2[1] * e2[1] + e2[2] * e2[2]);
    return l1 * l2 > 0.0f && !(area * kSliver > l1 * l2);   // (a zero edge gives det = 0: never a hit)
}

// How far from the triangle, across the ray, the rounding of the reference's
// test can put a hit: 2^-22 of the triangle's extent over the sine between its
// edges, with a factor of 4 (what it is of the ray's length, the part of
// kNearMargin covers).
__device__ __forceinline__ float triangle_pad(const orn_bvh_node& n) {
    float lo[3], hi[3];
    triangle_box(n, lo, hi);
    double e1[3], e2[3], l1 = 0.0, l2 = 0.0, cc = 0.0;
    for (int k = 0; k < 3; ++k) {
        e1[k] = (double)n.left_aabb_max_or_v1[k] - n.left_aabb_min_or_v0[k];
        e2[k] = (double)n.right_aabb_min_or_v2[k] - n.left_aabb_min_or_v0[k];
        l1 += e1[k] * e1[k];
        l2 += e2[k] * e2[k];
    }
    for (int k = 0; k < 3; ++k) {
        const int a = (k + 1) % 3, b = (k + 2) % 3;
        const double c = e1[a] * e2[b] - e1[b] * e2[a];
        cc += c * c;
    }
    if (!(cc > 0.0)) return 0.0f;   // (no area: never hit)
    // (a sliver's box is its tree's, whatever its edges)
    return fmaxf(fmaxf(hi[0] - lo[0], hi[1] - lo[1]), hi[2] - lo[2]) * kPadTriangle *
           (float)fmin(sqrt(l1 * l2 / cc), (double)kSliver);
}

// Sort key and box of every primitive, by node index (BLAS, then TLAS).
__global__ void prims_kernel(const orn_bvh_node* __restrict__ tlas, uint32_t T, const orn_bvh_node* __restrict__ blas,
                             uint32_t B, const uint32_t* __restrict__ bparent, const uint32_t* __restrict__ tparent,
                             const uint8_t* __restrict__ is_root, unsigned long long* __restrict__ keys,
                             uint32_t* __restrict__ vals, float4* __restrict__ boxes, uint8_t* __restrict__ tree_used,
                             uint32_t* __restrict__ mesh_pad, State* st) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= B + T) return;
    keys[i] = 1ull << 60;   // after every tree: not a primitive of one
    vals[i] = i;
    const bool top = i >= B;
    const uint32_t self = top ? i - B : i;
    const orn_bvh_node nd = top ? tlas[self] : blas[self];
    if (nd.node_type == ORN_NODE_INTERNAL) return;
    float lo[3], hi[3], tlo[3], thi[3];
    uint32_t tree = kNone;
    uint32_t depth = 0;
    const uint32_t* parent = top ? tparent : bparent;
    uint32_t cur = self;
    for (;;) {   // up to the top: the tree is the one marked root on the way
        if (top ? cur == T - 1 : is_root[cur] != 0) {
            if (tree != kNone) st->bad = 1u;   // a mesh inside another
            tree = top ? kTlasTree : cur;
        }
        const uint32_t p = parent[cur];
        if (p == kNone) break;
        cur = p & 0x7fffffffu;
        if (tree == kNone) ++depth;
        if (depth > kDepthLimit) {
            st->bad = 1u;
            return;
        }
    }
    if (tree == kNone) return;   // not reachable from any shape
    uint32_t* deepest = top ? &st->tlas_depth : &st->blas_depth;
    if (depth > *(volatile uint32_t*)deepest) atomicMax(deepest, depth);
    const uint32_t p = parent[self];
    if (top) {
        if (self != T - 1) {
            stored_box(tlas[p & 0x7fffffffu], (p >> 31) != 0, lo, hi);
        } else {
            for (int k = 0; k < 3; ++k) {   // the only shape: its own node carries its box
                lo[k] = nd.left_aabb_min_or_v0[k];
                hi[k] = nd.left_aabb_max_or_v1[k];
            }
        }
        float ext = 0.0f;
        for (int k = 0; k < 3; ++k) ext = fmaxf(ext, fmaxf(fabsf(lo[k]), fabsf(hi[k])));
        if (!(ext < 1e30f)) st->bad = 1u;
        atomicMax((uint32_t*)&st->world, __float_as_uint(ext));
        const orn_bvh_node root = tlas[T - 1];
        if (T > 1) {
            float l2[3], h2[3];
            stored_box(root, false, tlo, thi);
            stored_box(root, true, l2, h2);
            for (int k = 0; k < 3; ++k) {
                tlo[k] = fminf(tlo[k], l2[k]);
                thi[k] = fmaxf(thi[k], h2[k]);
            }
        } else {
            for (int k = 0; k < 3; ++k) {
                tlo[k] = lo[k];
                thi[k] = hi[k];
            }
        }
    } else {
        triangle_box(nd, lo, hi);
        const orn_bvh_node root = blas[tree];
        if (root.node_type == ORN_NODE_INTERNAL) {
            float l2[3], h2[3];
            stored_box(root, false, tlo, thi);
            stored_box(root, true, l2, h2);
            for (int k = 0; k < 3; ++k) {
                tlo[k] = fminf(tlo[k], l2[k]);
                thi[k] = fmaxf(thi[k], h2[k]);
            }
        } else {
            for (int k = 0; k < 3; ++k) {
                tlo[k] = lo[k];
                thi[k] = hi[k];
            }
        }
        bool finite = true;
        for (int k = 0; k < 3; ++k) finite = finite && fabsf(lo[k]) < 1e30f && fabsf(hi[k]) < 1e30f;
        if (!finite) st->bad = 1u;
    }
    keys[i] = ((unsigned long long)tree << 30) | morton30(lo, hi, tlo, thi);
    float own_box = 0.0f;   // a mark: the box given here is not the triangle's own
    if (!top && tree != self && is_sliver(nd)) {   // visited wherever its mesh is
        atomicAdd(&st->slivers, 1u);
        own_box = __uint_as_float(kOwnBoxMark);
        for (int k = 0; k < 3; ++k) {
            lo[k] = tlo[k];
            hi[k] = thi[k];
        }
    }
    if (!top) {
        const uint32_t pad = __float_as_uint(triangle_pad(nd));
        if (pad > *(volatile uint32_t*)&mesh_pad[tree]) atomicMax(&mesh_pad[tree], pad);
    }
    boxes[2 * (size_t)i] = make_float4(lo[0], lo[1], lo[2], 0.0f);
    boxes[2 * (size_t)i + 1] = make_float4(hi[0], hi[1], hi[2], own_box);
    atomicAdd(&st->prims, 1u);
    uint8_t* used = top ? tree_used + B : tree_used + tree;
    if (*used == 0) *used = 1;
}

// How far the hits that the reference's tests compute in a shape may lie outside
// its box in the TLAS (the largest of all shapes, and of their axes, is
// SceneDev::near_reach): by the padding of its triangles or its ball, by the
// rounding of its inverse transform's translation, and because the box, a
// caller's, is not quite around it.  The rounding that grows with the ray's
// origin is near_turn's.  Boxes that miss their shapes altogether, and singular
// transforms, keep the blob's walk.
__global__ void shapes_kernel(const orn_bvh_node* __restrict__ tlas, uint32_t T,
                              const orn_bvh_node* __restrict__ blas, uint32_t B, const float4* __restrict__ xforms,
                              const unsigned long long* __restrict__ keys, const uint32_t* __restrict__ mesh_pad,
                              const float4* __restrict__ boxes, State* st) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= T || keys[B + (size_t)i] >> 60 != 0ull) return;
    const orn_bvh_node nd = tlas[i];
    double a[3][3], t[3], inv[3][3];
    for (int r = 0; r < 3; ++r) {
        const float4 row = xforms[(size_t)nd.transform_id * 8 + r];
        a[r][0] = row.x;
        a[r][1] = row.y;
        a[r][2] = row.z;
        t[r] = row.w;
    }
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) {
            const int a0 = (c + 1) % 3, a1 = (c + 2) % 3, b0 = (r + 1) % 3, b1 = (r + 2) % 3;
            inv[r][c] = a[a0][b0] * a[a1][b1] - a[a0][b1] * a[a1][b0];
        }
    const double det = a[0][0] * inv[0][0] + a[0][1] * inv[1][0] + a[0][2] * inv[2][0];
    const bool mesh = nd.node_type == ORN_NODE_MESH;
    double centre[3] = {0.0, 0.0, 0.0}, half[3] = {1.0, 1.0, 1.0}, pad[3] = {kPadSphere, kPadSphere, kPadSphere};
    if (mesh) {
        const orn_bvh_node root = blas[nd.left_or_custom_id];
        float lo[3], hi[3];
        if (root.node_type == ORN_NODE_TRIANGLE) {
            triangle_box(root, lo, hi);
        } else {
            float l2[3], h2[3];
            stored_box(root, false, lo, hi);
            stored_box(root, true, l2, h2);
            for (int k = 0; k < 3; ++k) {
                lo[k] = fminf(lo[k], l2[k]);
                hi[k] = fmaxf(hi[k], h2[k]);
            }
        }
        for (int k = 0; k < 3; ++k) {
            centre[k] = 0.5 * ((double)lo[k] + hi[k]);
            half[k] = 0.5 * ((double)hi[k] - lo[k]);
            pad[k] = __uint_as_float(mesh_pad[nd.left_or_custom_id]);
        }
    }
    const float4 blo = boxes[2 * ((size_t)B + i)], bhi = boxes[2 * ((size_t)B + i) + 1];
    const double box_lo[3] = {blo.x, blo.y, blo.z}, box_hi[3] = {bhi.x, bhi.y, bhi.z};
    double turn = 0.0, out = 0.0, slide = 0.0;
    bool ok = true;
    for (int r = 0; r < 3; ++r) {
        double at = 0.0, reach = 0.0, square = 0.0, move = 0.0, wide = 0.0, cond = 0.0;
        for (int c = 0; c < 3; ++c) {
            const double v = inv[r][c] / det, m = fabs(v);
            at += v * (centre[c] - t[c]);
            reach += m * half[c];
            square += m * m;
            move += m * fabs(t[c]);
            wide += m * pad[c];
            cond += m * (fabs(a[c][0]) + fabs(a[c][1]) + fabs(a[c][2]));
        }
        if (!mesh) reach = sqrt(square);   // (the box of the ball's image)
        if (mesh) slide = fmax(slide, wide * kNearSlide);
        wide += (move + fabs(at) + reach) * kPadMove;
        const double miss = fmax(at + reach - box_hi[r], box_lo[r] - (at - reach));
        // (the only shape's box is not tested)
        ok = ok && (T == 1 || miss <= kMostMiss * (fabs(box_lo[r]) + fabs(box_hi[r]) + move)) && cond < kMostTurn;
        out = fmax(out, wide + fmax(miss, 0.0));
        turn = fmax(turn, cond);
    }
    if (!ok) {   // (NaN among them)
        st->bad = 1u;
        return;
    }
    atomicMax((uint32_t*)&st->turn, __float_as_uint(__double2float_ru(turn * kPadMove)));
    atomicMax((uint32_t*)&st->slide, __float_as_uint(__double2float_ru(slide)));
    atomicMax((uint32_t*)&st->reach, __float_as_uint(__double2float_ru(T == 1 ? 0.0 : out)));
}

__global__ void count_trees_kernel(const uint8_t* __restrict__ used, uint32_t n, State* st) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned m = __ballot_sync(0xffffffffu, i < n && used[i] != 0);
    if ((threadIdx.x & 31u) == 0 && m) atomicAdd(&st->trees, (uint32_t)__popc(m));
}

// ---- binary trees ------------------------------------------------------------------------------
// Node k < n is the k-th primitive in sorted order; inner nodes follow.
// node_box[2k], [2k+1]: corners, the tree id in the first one's w, the levels
// below (or a leaf's kOwnBoxMark) in the second's.
__global__ void leaves_kernel(const unsigned long long* __restrict__ keys, const uint32_t* __restrict__ vals,
                              const float4* __restrict__ boxes, uint32_t n, float4* __restrict__ node_box,
                              uint32_t* __restrict__ cluster, State* st) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k == 0) st->clusters = n;
    if (k >= n) return;
    const uint32_t v = vals[k];
    float4 lo = boxes[2 * (size_t)v];
    lo.w = __uint_as_float((uint32_t)(keys[k] >> 30));
    node_box[2 * (size_t)k] = lo;
    node_box[2 * (size_t)k + 1] = boxes[2 * (size_t)v + 1];
    cluster[k] = k;
}

__device__ __forceinline__ float half_area(float4 lo, float4 hi) {
    const float x = hi.x - lo.x, y = hi.y - lo.y, z = hi.z - lo.z;
    return x * y + y * z + z * x;
}
__device__ __forceinline__ float4 min4(float4 a, float4 b) {
    return make_float4(fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z), a.w);
}
__device__ __forceinline__ float4 max4(float4 a, float4 b) {
    return make_float4(fmaxf(a.x, b.x), fmaxf(a.y, b.y), fmaxf(a.z, b.z), a.w);
}

// Each cluster's choice among its neighbours.  Pairs are ordered by (area,
// i xor j): the least pair of a tree is chosen from both sides, so every
// round merges something, and among equal boxes each index has another
// partner.
// (`bound`: clusters as the host last saw them; the kernels of a round read
// how many there are.)
__global__ void __launch_bounds__(kNnBlock)
neighbour_kernel(const uint32_t* __restrict__ cluster, const float4* __restrict__ node_box, uint32_t* __restrict__ nn,
                 const State* st) {
    const uint32_t m = st->clusters;
    __shared__ float4 slo[kNnBlock + 2 * kRadius], shi[kNnBlock + 2 * kRadius];
    const int first = (int)(blockIdx.x * kNnBlock) - kRadius;
    for (int t = threadIdx.x; t < kNnBlock + 2 * kRadius; t += kNnBlock) {
        const int g = first + t;
        float4 lo = make_float4(0, 0, 0, __uint_as_float(kNone)), hi = lo;
        if (g >= 0 && g < (int)m) {
            const uint32_t c = cluster[g];
            lo = node_box[2 * (size_t)c];
            hi = node_box[2 * (size_t)c + 1];
        }
        slo[t] = lo;
        shi[t] = hi;
    }
    __syncthreads();
    const uint32_t i = blockIdx.x * kNnBlock + threadIdx.x;
    if (i >= m) return;
    const int self = threadIdx.x + kRadius;
    const float4 lo = slo[self], hi = shi[self];
    const uint32_t tree = __float_as_uint(lo.w);
    uint32_t best = kNone;
    float area = 0.0f;
    for (int r = -kRadius; r <= kRadius; ++r) {
        if (r == 0 || __float_as_uint(slo[self + r].w) != tree) continue;
        const float a = half_area(min4(lo, slo[self + r]), max4(hi, shi[self + r]));
        const uint32_t j = i + r;
        if (best == kNone || a < area || (a == area && (i ^ j) < (i ^ best))) {
            best = j;
            area = a;
        }
    }
    nn[i] = best;
}

// For trees that merge too slowly: neighbours in pairs, from an even or odd place.
__global__ void pair_kernel(const uint32_t* __restrict__ cluster, const float4* __restrict__ node_box, uint32_t odd,
                            uint32_t* __restrict__ nn, const State* st) {
    const uint32_t m = st->clusters;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const uint32_t j = ((i + odd) & 1u) ? i - 1u : i + 1u;
    nn[i] = j < m && __float_as_uint(node_box[2 * (size_t)cluster[i]].w) ==
                         __float_as_uint(node_box[2 * (size_t)cluster[j]].w) ? j : kNone;
}

// The box above two others, with its levels.
__device__ __forceinline__ void join_boxes(float4 alo, float4 ahi, float4 blo, float4 bhi, float4* lo, float4* hi) {
    const uint32_t ha = __float_as_uint(ahi.w) & ~kOwnBoxMark, hb = __float_as_uint(bhi.w) & ~kOwnBoxMark;
    *lo = min4(alo, blo);
    *hi = max4(ahi, bhi);
    hi->w = __uint_as_float(max(ha, hb) + 1u);
}

__global__ void merge_kernel(uint32_t* __restrict__ cluster, uint32_t bound, const uint32_t* __restrict__ nn, uint32_t n,
                             float4* __restrict__ node_box, uint2* __restrict__ child, uint8_t* __restrict__ keep,
                             State* st) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= bound) return;
    const uint32_t m = st->clusters;
    const uint32_t j = i < m ? nn[i] : kNone;
    const bool pair = j != kNone && nn[j] == i;
    keep[i] = i < m && (!pair || i < j);
    if (!pair || i > j) return;
    const uint32_t a = cluster[i], b = cluster[j];
    const uint32_t id = n + atomicAdd(&st->next_node, 1u);
    float4 lo, hi;
    join_boxes(node_box[2 * (size_t)a], node_box[2 * (size_t)a + 1], node_box[2 * (size_t)b],
               node_box[2 * (size_t)b + 1], &lo, &hi);
    node_box[2 * (size_t)id] = lo;
    node_box[2 * (size_t)id + 1] = hi;
    child[id - n] = make_uint2(a, b);
    cluster[i] = id;
}

// The remaining rounds for at most kSmallClusters clusters, by one block with
// the boxes in shared memory; cluster[0..trees) is the trees' roots after it.
struct SmallClusters {
    float4 lo[kSmallClusters], hi[kSmallClusters];   // by slot; the list gives the slots in order
    uint32_t id[kSmallClusters];
    uint16_t list[2][kSmallClusters];
    uint16_t nn[kSmallClusters];
    uint32_t sums[kSmallBlock / 32];
};
__global__ void __launch_bounds__(kSmallBlock)
small_kernel(uint32_t* __restrict__ cluster, uint32_t trees, uint32_t n, float4* __restrict__ node_box,
             uint2* __restrict__ child, State* st) {
    extern __shared__ __align__(16) unsigned char small_smem[];
    SmallClusters& c = *reinterpret_cast<SmallClusters*>(small_smem);
    const uint32_t t = threadIdx.x;
    uint32_t m = st->clusters, next = st->next_node;
    for (uint32_t i = t; i < m; i += kSmallBlock) {
        const uint32_t id = cluster[i];
        c.id[i] = id;
        c.lo[i] = node_box[2 * (size_t)id];
        c.hi[i] = node_box[2 * (size_t)id + 1];
        c.list[0][i] = (uint16_t)i;
    }
    __syncthreads();
    uint32_t cur = 0;
    for (uint32_t round = 0; m > trees; ++round, cur ^= 1u) {
        const uint16_t* list = c.list[cur];
        for (uint32_t i = t; i < m; i += kSmallBlock) {
            const uint32_t s = list[i], tree = __float_as_uint(c.lo[s].w);
            uint32_t best = 0xffffu;
            float area = 0.0f;
            const bool chosen = round < kChosenRounds;
            const int from = chosen ? -kRadius : (((i + round) & 1u) ? -1 : 1), to = chosen ? kRadius : from;
            for (int r = from; r <= to; ++r) {
                const int j = (int)i + r;
                if (r == 0 || j < 0 || j >= (int)m) continue;
                const uint32_t q = list[j];
                if (__float_as_uint(c.lo[q].w) != tree) continue;
                const float a = half_area(min4(c.lo[s], c.lo[q]), max4(c.hi[s], c.hi[q]));
                if (best == 0xffffu || a < area || (a == area && (i ^ (uint32_t)j) < (i ^ best))) {
                    best = (uint32_t)j;
                    area = a;
                }
            }
            c.nn[i] = (uint16_t)best;
        }
        __syncthreads();
        // thread t takes places 2t and 2t + 1: what stays, what merges
        uint32_t stay = 0, made = 0;
        for (uint32_t k = 0; k < 2; ++k) {
            const uint32_t i = 2 * t + k;
            if (i >= m) continue;
            const uint32_t j = c.nn[i];
            const bool pair = j != 0xffffu && c.nn[j] == i;
            if (!pair || i < j) stay |= 1u << k;
            if (pair && i < j) made |= 1u << k;
        }
        // places in the next list and numbers of the new nodes: one scan of both counts
        uint32_t sum = (uint32_t)__popc(stay) | ((uint32_t)__popc(made) << 16);
        const uint32_t own = sum, lane = t & 31u;
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += v;
        }
        if (lane == 31u) c.sums[t >> 5] = sum;
        __syncthreads();
        if (t < 32u) {
            uint32_t v = c.sums[t];
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += u;
            }
            c.sums[t] = v;
        }
        __syncthreads();
        const uint32_t before = sum - own + (t >= 32u ? c.sums[(t >> 5) - 1] : 0u), total = c.sums[kSmallBlock / 32 - 1];
        uint32_t place = before & 0xffffu, number = before >> 16;
        for (uint32_t k = 0; k < 2; ++k) {
            const uint32_t i = 2 * t + k;
            if (!((stay >> k) & 1u)) continue;
            const uint32_t s = list[i];
            if ((made >> k) & 1u) {
                const uint32_t q = list[c.nn[i]], id = n + next + number;
                ++number;
                float4 lo, hi;
                join_boxes(c.lo[s], c.hi[s], c.lo[q], c.hi[q], &lo, &hi);
                child[id - n] = make_uint2(c.id[s], c.id[q]);
                node_box[2 * (size_t)id] = lo;
                node_box[2 * (size_t)id + 1] = hi;
                c.lo[s] = lo;
                c.hi[s] = hi;
                c.id[s] = id;
            }
            c.list[cur ^ 1u][place++] = (uint16_t)s;
        }
        m = total & 0xffffu;
        next += total >> 16;
        __syncthreads();
    }
    for (uint32_t i = t; i < m; i += kSmallBlock) cluster[i] = c.id[c.list[cur][i]];
    if (t == 0) {
        st->clusters = m;
        st->next_node = next;
    }
}

// ---- the node array ----------------------------------------------------------------------------
// What the writing kernels share.
struct Emit {
    uint32_t n, B, T;
    const float4* node_box;
    const uint2* child;
    const uint32_t* vals;      // primitive k's node index in the blob (BLAS, then TLAS)
    const float4* nodes;       // the kernels' node array (TLAS, then BLAS)
    float4* out;               // the same array: the new nodes go behind
    uint32_t first;            // index of the first new node
    uint32_t* root_of;         // by BLAS node index: the reference of a mesh's root
    uint32_t* mesh_place;      // places of the mesh leaves
    const uint32_t* mesh_pad;  // by BLAS node index: triangle_pad of a mesh
    State* st;
};

// Reference to tree node c.
__device__ __forceinline__ uint32_t node_ref(const Emit& e, uint32_t c) {
    const uint32_t at = e.first + c;
    if (c >= e.n) return at;   // ORN_NODE_INTERNAL == 0
    const uint32_t v = e.vals[c];
    if (v < e.B) return at | ((uint32_t)ORN_NODE_TRIANGLE << 30);
    const bool sphere = __float_as_uint(e.nodes[(size_t)(v - e.B) * 4 + 2].w) == ORN_NODE_SPHERE;
    return at | ((uint32_t)(sphere ? ORN_NODE_SPHERE : ORN_NODE_MESH) << 30);
}

// One cluster per tree is left: its root.
__global__ void levels_kernel(const float4* __restrict__ node_box, const uint32_t* __restrict__ cluster, uint32_t trees,
                              State* st) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= trees) return;
    const uint32_t c = cluster[i];
    const uint32_t levels = __float_as_uint(node_box[2 * (size_t)c + 1].w) & ~kOwnBoxMark;
    atomicMax(&st->near_depth[__float_as_uint(node_box[2 * (size_t)c].w) == kTlasTree ? 1 : 0], levels);
}
__global__ void roots_kernel(Emit e, const uint32_t* __restrict__ cluster, uint32_t trees) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= trees) return;
    const uint32_t c = cluster[i];
    const uint32_t tree = __float_as_uint(e.node_box[2 * (size_t)c].w);
    if (tree == kTlasTree) e.st->root = node_ref(e, c);
    else e.root_of[tree] = node_ref(e, c);
}

// ---- how much there is to walk -----------------------------------------------------------------
// Visits that a ray is expected to make: a box is visited with the chance of its
// area over that of the box of all shapes, a node in a mesh with that of its
// mesh's instances times its area over the mesh's own.  Shapes that take up more
// than a quarter of the scene (the ground, the walls of a room) would make all
// others look out of the way, where rays hardly are: they are left out of the box
// of all shapes, and no chance is more than one.
__device__ __forceinline__ float inner_area(const orn_bvh_node& nd) {   // of the box around both children's
    float lo[3], hi[3], l2[3], h2[3];
    stored_box(nd, false, lo, hi);
    stored_box(nd, true, l2, h2);
    return half_area(fmaxf(hi[0], h2[0]) - fminf(lo[0], l2[0]), fmaxf(hi[1], h2[1]) - fminf(lo[1], l2[1]),
                     fmaxf(hi[2], h2[2]) - fminf(lo[2], l2[2]));
}
__device__ __forceinline__ uint32_t order_key(float f) {   // order-preserving, for atomic maxima
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float key_float(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? k & 0x7fffffffu : ~k);
}
__global__ void ordinary_kernel(const orn_bvh_node* __restrict__ tlas, uint32_t T, uint32_t B,
                                const unsigned long long* __restrict__ keys, const float4* __restrict__ boxes, State* st) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= T || keys[B + (size_t)i] >> 60 != 0ull) return;
    const float4 lo = boxes[2 * ((size_t)B + i)], hi = boxes[2 * ((size_t)B + i) + 1];
    if (T > 1 && half_area(lo, hi) > 0.25f * inner_area(tlas[T - 1])) {
        atomicAdd(&st->large_shapes, 1u);
        return;
    }
    const float v[6] = {-lo.x, -lo.y, -lo.z, hi.x, hi.y, hi.z};
    for (int k = 0; k < 6; ++k) atomicMax(&st->shapes_box[k], order_key(v[k]));
}
__device__ __forceinline__ float shapes_area(const State* st, const orn_bvh_node& root) {
    float v[6];
    for (int k = 0; k < 6; ++k) {
        const uint32_t key = st->shapes_box[k];
        if (key == 0u) return inner_area(root);   // none
        v[k] = key_float(key);
    }
    return half_area(v[3] + v[0], v[4] + v[1], v[5] + v[2]);
}
__device__ __forceinline__ float chance_of(float area, float all) { return all > 0.0f ? fminf(area / all, 1.0f) : 1.0f; }
// Of each mesh (by its root): the sum over its instances.
__global__ void chances_kernel(const orn_bvh_node* __restrict__ tlas, uint32_t T, uint32_t B,
                               const unsigned long long* __restrict__ keys, const float4* __restrict__ boxes,
                               float* __restrict__ chance, const State* st) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= T || tlas[i].node_type != ORN_NODE_MESH || keys[B + (size_t)i] >> 60 != 0ull) return;
    const float all = T > 1 ? shapes_area(st, tlas[T - 1]) : 0.0f;
    atomicAdd(&chance[tlas[i].left_or_custom_id],
              chance_of(half_area(boxes[2 * ((size_t)B + i)], boxes[2 * ((size_t)B + i) + 1]), all));
}
__global__ void blob_visits_kernel(const orn_bvh_node* __restrict__ tlas, uint32_t T,
                                   const orn_bvh_node* __restrict__ blas, uint32_t B,
                                   const uint32_t* __restrict__ bparent, const uint8_t* __restrict__ is_root,
                                   const float* __restrict__ chance, State* st) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool top = i < T;
    float a = 0.0f;
    if (i < T + B && (top ? tlas[i] : blas[i - T]).node_type == ORN_NODE_INTERNAL) {
        const orn_bvh_node nd = top ? tlas[i] : blas[i - T];
        float all, times = 1.0f;
        if (top) {
            all = shapes_area(st, tlas[T - 1]);
        } else {
            uint32_t root = i - T;
            for (uint32_t level = 0; !is_root[root] && bparent[root] != kNone && level < kDepthLimit; ++level)
                root = bparent[root] & 0x7fffffffu;
            all = inner_area(blas[root]);
            times = is_root[root] ? chance[root] : 0.0f;
        }
        for (int side = 0; side < 2; ++side) {
            float lo[3], hi[3];
            stored_box(nd, side != 0, lo, hi);
            a += times * chance_of(half_area(hi[0] - lo[0], hi[1] - lo[1], hi[2] - lo[2]), all);
        }
    }
    add_area(&st->visits[0], top ? a : 0.0f);
    add_area(&st->visits[1], top ? 0.0f : a);
}
__global__ void near_visits_kernel(Emit e, uint32_t total, const orn_bvh_node* __restrict__ tlas,
                                   const orn_bvh_node* __restrict__ blas, const float* __restrict__ chance) {
    const uint32_t c = e.n + blockIdx.x * blockDim.x + threadIdx.x;
    float a = 0.0f;
    bool top = false;
    if (c < total) {
        const uint2 ch = e.child[c - e.n];
        const uint32_t tree = __float_as_uint(e.node_box[2 * (size_t)c].w);
        top = tree == kTlasTree;
        const float all = top ? shapes_area(e.st, tlas[e.T - 1]) : inner_area(blas[tree]);
        for (int side = 0; side < 2; ++side) {
            const uint32_t k = side ? ch.y : ch.x;
            a += chance_of(half_area(e.node_box[2 * (size_t)k], e.node_box[2 * (size_t)k + 1]), all);
        }
        if (!top) a *= chance[tree];
    }
    add_area(&e.st->visits[2], top ? a : 0.0f);
    add_area(&e.st->visits[3], top ? 0.0f : a);
}

__global__ void write_kernel(Emit e, uint32_t total) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= total) return;
    float4* o = e.out + 4 * (size_t)c;
    if (c >= e.n) {
        const uint2 ch = e.child[c - e.n];
        float4 llo = e.node_box[2 * (size_t)ch.x], lhi = e.node_box[2 * (size_t)ch.x + 1];
        float4 rlo = e.node_box[2 * (size_t)ch.y], rhi = e.node_box[2 * (size_t)ch.y + 1];
        llo.w = __uint_as_float(node_ref(e, ch.x));
        lhi.w = __uint_as_float(node_ref(e, ch.y));
        rlo.w = __uint_as_float(ORN_NODE_INTERNAL);
        rhi.w = 0.0f;
        o[0] = llo;
        o[1] = lhi;
        o[2] = rlo;
        o[3] = rhi;
        return;
    }
    const uint32_t v = e.vals[c];
    const float4* src = e.nodes + 4 * (size_t)(v < e.B ? e.T + v : v - e.B);
    float4 a = src[0];
    float4 mid = src[2];
    if (v < e.B && (__float_as_uint(e.node_box[2 * (size_t)c + 1].w) & kOwnBoxMark) != 0u)
        a.w = __uint_as_float(__float_as_uint(a.w) | kNearOwnBox);
    if (v >= e.B && __float_as_uint(mid.w) == ORN_NODE_MESH) {
        e.mesh_place[atomicAdd(&e.st->meshes, 1u)] = c;
        // (in the place of the type, which references carry)
        mid.w = __uint_as_float(e.mesh_pad[(__float_as_uint(src[3].w) & kRefIndexMask) - e.T]);
    }
    o[0] = a;
    o[1] = src[1];
    o[2] = mid;
    o[3] = src[3];
}

// Points the mesh leaves of the written array at their new roots.
__global__ void meshes_kernel(float4* __restrict__ out, uint32_t T, const uint32_t* __restrict__ root_of,
                              const uint32_t* __restrict__ mesh_place, const State* st) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= st->meshes) return;
    float4* o = out + 4 * (size_t)mesh_place[i];
    const uint32_t old = __float_as_uint(o[3].w) & kRefIndexMask;   // in the kernels' array: T + BLAS index
    o[3].w = __uint_as_float(root_of[old - T]);
}

inline unsigned blocks(size_t n, unsigned per) { return (unsigned)((n + per - 1) / per); }

// A bump allocator over one device allocation.
struct Arena {
    unsigned char* base = nullptr;
    size_t used = 0, size = 0;
    template <class T>
    T* take(size_t count) {
        used = (used + 255) & ~(size_t)255;
        T* p = (T*)(base + used);
        used += count * sizeof(T);
        return p;
    }
};

#define WB(call)                               \
    do {                                       \
        const cudaError_t e_ = (call);         \
        if (e_ != cudaSuccess) return e_;      \
    } while (0)

struct Build {
    const orn_scene_blob* blob;
    const float4* xforms;
    SceneDev* scene;
    cudaStream_t s;
    State* d_state = nullptr;
    State h{};
    orn_bvh_node *tlas = nullptr, *blas = nullptr;
    void *first = nullptr, *second = nullptr;   // arenas of near_trees
    // the new trees as near_trees leaves them to write_trees; no nodes: none
    Emit e{};
    uint32_t* cluster = nullptr;
    uint32_t trees = 0, total = 0;

    cudaError_t read_state() {
        WB(cudaMemcpyAsync(&h, d_state, sizeof(State), cudaMemcpyDeviceToHost, s));
        return cudaStreamSynchronize(s);
    }
    cudaError_t near_trees();
    cudaError_t write_trees(float4* nodes);
};

// Bytes of the first phase's arrays (all nodes), and of the second's (n primitives).
size_t first_bytes(size_t T, size_t B) {
    return 4 * (T + B) + 2 * (B + 1) + 24 * (T + B) + 32 * (T + B) + 8 * B + 32 * 256;
}
size_t second_bytes(size_t n, size_t T, size_t B, size_t temp) {
    return temp + 64 * n + 8 * n + 13 * n + 4 * (T + B) + 32 * 256;
}

// Who walks the near-first trees.  They take fewer visits, but a visit costs
// more: some 1.2 times as much in batches and the FP64 renderer, 1.5 times in the
// megakernel and the persistent wavefront.  So the lines lie at `blob`, the visits
// expected in the blob's trees, and at how many `times` those in the new ones that
// is.  Measured with 960 x 540 pixels, 16 passes, 58 scenes of 9 to 2 M nodes on
// the reference's median splits (1.0 to 2.0 times the visits), binned SAH (0.91 to
// 1.1) and linear trees (0.93 to 1.2); time on the blob's trees over time on the new:
//   * Ray lists, 1 to 1 M rays: 0.97 to 2.6, all scenes.
//   * Spheres and walls of two triangles, where little of the walk is in meshes,
//     and small meshes on a ground: shading counts for more, and the kernels on the
//     new trees have it in one sequence (shade_geom).  Megakernel 0.98 to 1.61
//     whatever the trees, batches 0.96 to 1.53; the wavefront, whose shading is the
//     same on either, 0.78 to 1.05.  With fewer than four visits there is nothing
//     to gain (five spheres: 1.0 to 1.09, batches 0.86 to 0.91).
//   * Others, megakernel: from 1.5 times and 50 visits on 1.01 to 1.21 (a closed
//     room of 64 instances 0.93); below that 0.64 to 1.25.
//   * Wavefront: from 1.5 times and 200 visits on 1.03 to 1.24, below 0.66 to 1.21.
//   * Batches: from 1.15 times on 1.0 to 1.6, below 0.88 to 1.25; FP64 likewise.
// (One line for all, and none below 16,384 nodes, had frames of SAH and linear
// trees there up to 1.35 times as long as on the blob's.)
uint32_t near_level(const State& h) {
    const float blob = h.visits[0] + h.visits[1], times = blob / (h.visits[2] + h.visits[3]);
    const float in_meshes = h.visits[1] / blob;
    if (!(blob >= 4.0f)) return NEAR_RAYS;
    if (in_meshes <= 0.45f || (in_meshes <= 0.7f && blob <= 30.0f && h.large_shapes == 1u)) return NEAR_MEGA;
    if (times >= 1.5f && blob >= 50.0f) return blob >= 200.0f ? NEAR_WAVE : NEAR_MEGA;
    return times >= 1.15f ? NEAR_BATCH : NEAR_RAYS;
}

// Decides whether the scene has near-first trees, and builds them up to their
// nodes.  Out of memory is an answer too: then it has none.
cudaError_t Build::near_trees() {
    const uint32_t T = blob->tlas_nodes_len, B = blob->blas_nodes_len, N = T + B;
    Arena a;
    a.size = first_bytes(T, B);
    WB(cudaMalloc((void**)&a.base, a.size));
    first = a.base;
    uint32_t* bparent = a.take<uint32_t>(B);
    uint32_t* tparent = a.take<uint32_t>(T);
    uint8_t* is_root = a.take<uint8_t>((size_t)B + 1);
    uint8_t* used = a.take<uint8_t>((size_t)B + 1);
    WB(cudaMemsetAsync(bparent, 0xff, (size_t)B * 4, s));
    WB(cudaMemsetAsync(tparent, 0xff, (size_t)T * 4, s));
    WB(cudaMemsetAsync(is_root, 0, (size_t)B + 1, s));
    WB(cudaMemsetAsync(used, 0, (size_t)B + 1, s));
    parents_kernel<<<blocks(T, 256), 256, 0, s>>>(tlas, T, tparent, d_state);
    if (B) parents_kernel<<<blocks(B, 256), 256, 0, s>>>(blas, B, bparent, d_state);
    if (B) mark_roots_kernel<<<blocks(T, 256), 256, 0, s>>>(tlas, T, is_root);
    unsigned long long* keys = a.take<unsigned long long>(N);
    unsigned long long* keys2 = a.take<unsigned long long>(N);
    uint32_t* vals = a.take<uint32_t>(N);
    uint32_t* vals2 = a.take<uint32_t>(N);
    float4* boxes = a.take<float4>(2 * (size_t)N);
    uint32_t* mesh_pad = a.take<uint32_t>(B);   // by mesh: the largest of its triangles' (float bits)
    float* chance = a.take<float>(B);           // by mesh: that a ray comes to it (chances_kernel)
    WB(cudaMemsetAsync(mesh_pad, 0, 4 * (size_t)B, s));
    WB(cudaMemsetAsync(chance, 0, 4 * (size_t)B, s));
    prims_kernel<<<blocks(N, 256), 256, 0, s>>>(tlas, T, blas, B, bparent, tparent, is_root, keys, vals, boxes, used,
                                                mesh_pad, d_state);
    shapes_kernel<<<blocks(T, 128), 128, 0, s>>>(tlas, T, blas, B, xforms, keys, mesh_pad, boxes, d_state);
    count_trees_kernel<<<blocks((size_t)B + 1, 256), 256, 0, s>>>(used, B + 1, d_state);
    WB(cudaGetLastError());
    WB(read_state());
    const uint32_t n = h.prims;
    trees = h.trees;
    if (h.bad || h.slivers > kMostSlivers || h.tlas_depth + h.blas_depth > kDepthLimit || n == 0 ||
        2 * (uint64_t)N > kRefIndexMask)
        return cudaSuccess;
    size_t sort_bytes = 0, select_bytes = 0;
    WB(cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, keys, keys2, vals, vals2, (int)N, 0, 61, s));
    WB(cub::DeviceSelect::Flagged(nullptr, select_bytes, vals, is_root, vals2, &d_state->clusters, (int)n, s));
    const size_t temp_bytes = std::max(sort_bytes, select_bytes);
    Arena a2;
    a2.size = second_bytes(n, T, B, temp_bytes);
    WB(cudaMalloc((void**)&a2.base, a2.size));
    second = a2.base;
    void* temp = a2.take<unsigned char>(temp_bytes);
    size_t tb = sort_bytes;
    WB(cub::DeviceRadixSort::SortPairs(temp, tb, keys, keys2, vals, vals2, (int)N, 0, 61, s));
    float4* node_box = a2.take<float4>(4 * (size_t)n);
    uint2* child = a2.take<uint2>(n);
    cluster = a2.take<uint32_t>(n);
    uint32_t* cluster2 = a2.take<uint32_t>(n);
    uint32_t* nn = a2.take<uint32_t>(n);
    uint8_t* keep_flag = a2.take<uint8_t>(n);
    leaves_kernel<<<blocks(n, 256), 256, 0, s>>>(keys2, vals2, boxes, n, node_box, cluster, d_state);
    WB(cudaGetLastError());
    uint32_t m = n;
    for (uint32_t round = 0; m > kSmallClusters && m > trees; ++round) {
        if (round < kChosenRounds) neighbour_kernel<<<blocks(m, kNnBlock), kNnBlock, 0, s>>>(cluster, node_box, nn, d_state);
        else pair_kernel<<<blocks(m, 256), 256, 0, s>>>(cluster, node_box, round & 1u, nn, d_state);
        merge_kernel<<<blocks(m, 256), 256, 0, s>>>(cluster, m, nn, n, node_box, child, keep_flag, d_state);
        WB(cudaGetLastError());
        size_t sb = select_bytes;
        WB(cub::DeviceSelect::Flagged(temp, sb, cluster, keep_flag, cluster2, &d_state->clusters, (int)m, s));
        std::swap(cluster, cluster2);
        if (round % kRoundsPerSync == kRoundsPerSync - 1) {
            WB(read_state());
            m = h.clusters;
        }
    }
    if (trees < kSmallClusters) {
        WB(cudaFuncSetAttribute(small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmallClusters)));
        small_kernel<<<1, kSmallBlock, sizeof(SmallClusters), s>>>(cluster, trees, n, node_box, child, d_state);
    }
    e.n = n;
    e.B = B;
    e.T = T;
    e.node_box = node_box;
    e.child = child;
    e.vals = vals2;
    e.root_of = a2.take<uint32_t>(B);
    e.mesh_place = a2.take<uint32_t>(T);
    e.mesh_pad = mesh_pad;
    e.st = d_state;
    e.first = N;
    const uint32_t all = 2 * n - trees;   // (no more than N: a binary tree of k leaves has 2k - 1 nodes here as there)
    levels_kernel<<<blocks(trees, 128), 128, 0, s>>>(node_box, cluster, trees, d_state);
    ordinary_kernel<<<blocks(T, 128), 128, 0, s>>>(tlas, T, B, keys, boxes, d_state);
    chances_kernel<<<blocks(T, 128), 128, 0, s>>>(tlas, T, B, keys, boxes, chance, d_state);
    blob_visits_kernel<<<blocks(N, 256), 256, 0, s>>>(tlas, T, blas, B, bparent, is_root, chance, d_state);
    if (all > n) near_visits_kernel<<<blocks(all - n, 256), 256, 0, s>>>(e, all, tlas, blas, chance);
    WB(cudaGetLastError());
    WB(read_state());
    if (h.near_depth[0] + h.near_depth[1] <= kNearDepthLimit) total = all;
    return cudaSuccess;
}

// Writes the new trees behind the blob's nodes.
cudaError_t Build::write_trees(float4* nodes) {
    e.nodes = nodes;
    e.out = nodes + 4 * (size_t)e.first;
    roots_kernel<<<blocks(trees, 128), 128, 0, s>>>(e, cluster, trees);
    write_kernel<<<blocks(total, 256), 256, 0, s>>>(e, total);
    meshes_kernel<<<blocks(e.T, 128), 128, 0, s>>>(e.out, e.T, e.root_of, e.mesh_place, d_state);
    WB(cudaGetLastError());
    WB(read_state());
    scene->nroot = h.root;
    scene->near_turn = h.turn;
    scene->near_slide = h.slide;
    scene->near_reach = h.reach + h.turn * h.world;
    scene->visits = h.visits[0] + h.visits[1];
    scene->near = near_level(h);
    return cudaSuccess;
}

}  // namespace

cudaError_t build_scene_trees(const orn_scene_blob* blob, const float4* d_xforms, SceneDev* scene, NodeFacts* facts,
                              std::vector<void*>* allocs, cudaStream_t s) {
    const uint32_t T = blob->tlas_nodes_len, B = blob->blas_nodes_len;
    const size_t N = (size_t)T + B;
    Build b;
    b.blob = blob;
    b.xforms = d_xforms;
    b.scene = scene;
    b.s = s;
    scene->near = 0u;
    scene->large = N >= kLargeScene ? 1u : 0u;
    void *raw = nullptr, *own = nullptr, *both = nullptr;   // the blob's nodes; State and types; nodes with new trees
    cudaError_t e = [&]() -> cudaError_t {
        WB(cudaMalloc(&raw, N * 64));
        WB(cudaMalloc(&own, 256 + N));
        b.d_state = (State*)own;
        uint8_t* types = (uint8_t*)own + 256;
        b.tlas = (orn_bvh_node*)raw;
        b.blas = b.tlas + T;
        // the transforms came through the default stream, which `s` does not wait for
        WB(cudaStreamSynchronize(nullptr));
        WB(cudaMemsetAsync(b.d_state, 0, sizeof(State), s));
        WB(cudaMemcpyAsync(b.tlas, blob->tlas_nodes, (size_t)T * 64, cudaMemcpyHostToDevice, s));
        if (B) WB(cudaMemcpyAsync(b.blas, blob->blas_nodes, (size_t)B * 64, cudaMemcpyHostToDevice, s));
        types_kernel<<<blocks(N, 256), 256, 0, s>>>(b.tlas, (uint32_t)N, types);
        WB(cudaGetLastError());
        cudaError_t grown = b.near_trees();
        if (grown == cudaSuccess && b.total != 0u) grown = cudaMalloc(&both, (N + b.total) * 64);
        if (grown == cudaErrorMemoryAllocation) {
            (void)cudaGetLastError();
            b.total = 0u;
        } else if (grown != cudaSuccess) {
            return grown;
        }
        float4* nodes = (float4*)(b.total != 0u ? both : raw);
        relayout_kernel<<<blocks(N, 256), 256, 0, s>>>(b.tlas, T, B, types, d_xforms, nodes, b.d_state);
        WB(cudaGetLastError());
        if (b.total != 0u) WB(b.write_trees(nodes));
        else WB(b.read_state());
        facts->huge = b.h.huge;
        scene->nodes = nodes;
        return cudaSuccess;
    }();
    if (e != cudaSuccess) cudaStreamSynchronize(s);
    void* kept = const_cast<float4*>(scene->nodes);
    if (e == cudaSuccess) allocs->push_back(kept);
    for (void* p : {raw, own, both, b.first, b.second}) {
        if (!p || (e == cudaSuccess && p == kept)) continue;
        const cudaError_t f = cudaFree(p);
        if (e == cudaSuccess) e = f;
    }
    return e;
}

}  // namespace orn
