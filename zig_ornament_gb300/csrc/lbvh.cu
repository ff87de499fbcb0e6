// lbvh.cu — BLAS construction on the GPU (a non-parity builder mode,
// ORN_BVH_LBVH): linear BVH after Karras, "Maximizing Parallelism in the
// Construction of BVHs, Octrees, and k-d Trees" (HPG 2012).
//
//   1. 30-bit Morton code of each triangle's centroid in the mesh's bounds,
//      with the triangle index as the low 32 bits of a 64-bit key (distinct
//      keys, deterministic order); keys sorted with CUB's radix sort.
//   2. Karras' per-node range and split search over the sorted keys gives
//      the n-1 internal nodes, their children and parents.
//   3. Bounds bottom-up: each leaf walks towards the root; at every internal
//      node the second arriving thread (an atomic counter) forms the union of
//      the children's boxes and continues.
//   4. Post-order relabelling: the reference's node format wants children
//      before parents (root last).  A subtree over leaves [a, b] occupies
//      2(b - a + 1) - 1 consecutive slots ending with its root; a node's first
//      slot is the sum of the sizes of the left siblings on its path to the
//      root.
//   5. Nodes written in the reference's layout (one triangle per leaf, raw
//      vertices, child ids global) and copied back to the host arrays.
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "lbvh.h"

namespace orn {
namespace {

constexpr uint32_t kLeafBit = 0x80000000u;
constexpr size_t kNodesAtOnce = 1u << 20;   // nodes of finished meshes that wait on the device (64 MB)

__device__ __forceinline__ uint32_t expand_bits(uint32_t v) {
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

// Order-preserving integers for floats (NaN aside), for atomic minima and maxima.
__device__ __forceinline__ uint32_t float_key(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float key_float(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? k & 0x7fffffffu : ~k);
}

// Centroid bounds: keys of the minima in bounds[0..3), of the maxima in [3..6).
// (A triangle whose first vertex is NaN stays out of them, as with std::min and
// std::max: fminf and fmaxf, which drop a NaN, would let its other vertices
// move every triangle's code.)
__global__ void centroid_kernel(const float* __restrict__ tri, uint32_t n, uint32_t* __restrict__ bounds) {
    uint32_t lo[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, hi[3] = {0u, 0u, 0u};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float* v = tri + (size_t)i * 9;
        for (int k = 0; k < 3; ++k) {
            float mn = v[k], mx = v[k];
            for (int j = 1; j < 3; ++j) {
                mn = v[3 * j + k] < mn ? v[3 * j + k] : mn;
                mx = v[3 * j + k] > mx ? v[3 * j + k] : mx;
            }
            const float c = 0.5f * (mn + mx);
            if (!(c == c)) continue;
            lo[k] = min(lo[k], float_key(c));
            hi[k] = max(hi[k], float_key(c));
        }
    }
    for (int k = 0; k < 3; ++k) {
        const uint32_t l = __reduce_min_sync(0xffffffffu, lo[k]), h = __reduce_max_sync(0xffffffffu, hi[k]);
        if ((threadIdx.x & 31u) == 0) {
            atomicMin(bounds + k, l);
            atomicMax(bounds + 3 + k, h);
        }
    }
}

__global__ void morton_kernel(const float* __restrict__ tri, uint32_t n, const uint32_t* __restrict__ bounds,
                              unsigned long long* __restrict__ keys) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float3 lo = make_float3(key_float(bounds[0]), key_float(bounds[1]), key_float(bounds[2]));
    const float3 e = make_float3(key_float(bounds[3]) - lo.x, key_float(bounds[4]) - lo.y, key_float(bounds[5]) - lo.z);
    const float3 scale = make_float3(e.x > 0 ? 1023.0f / e.x : 0.0f, e.y > 0 ? 1023.0f / e.y : 0.0f,
                                     e.z > 0 ? 1023.0f / e.z : 0.0f);
    const float* v = tri + (size_t)i * 9;
    float c[3];
    for (int k = 0; k < 3; ++k) {
        const float mn = fminf(fminf(v[k], v[3 + k]), v[6 + k]), mx = fmaxf(fmaxf(v[k], v[3 + k]), v[6 + k]);
        c[k] = 0.5f * (mn + mx);
    }
    const float fx = fminf(fmaxf((c[0] - lo.x) * scale.x, 0.0f), 1023.0f);
    const float fy = fminf(fmaxf((c[1] - lo.y) * scale.y, 0.0f), 1023.0f);
    const float fz = fminf(fmaxf((c[2] - lo.z) * scale.z, 0.0f), 1023.0f);
    const uint32_t m = (expand_bits((uint32_t)fx) << 2) | (expand_bits((uint32_t)fy) << 1) | expand_bits((uint32_t)fz);
    keys[i] = ((unsigned long long)m << 32) | i;
}

__device__ __forceinline__ int delta(const unsigned long long* keys, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    return __clzll(keys[i] ^ keys[j]);
}

// Karras 2012, section 4: node i's range, split and children.
__global__ void hierarchy_kernel(const unsigned long long* __restrict__ keys, int n, uint32_t* __restrict__ left,
                                 uint32_t* __restrict__ right, int* __restrict__ parent_int,
                                 int* __restrict__ parent_leaf, uint32_t* __restrict__ range_lo,
                                 uint32_t* __restrict__ range_hi) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const int d = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
    const int dmin = delta(keys, n, i, i - d);
    int lmax = 2;
    while (lmax < n && delta(keys, n, i, i + lmax * d) > dmin) lmax *= 2;   // (the bound keeps i + lmax*d from overflowing)
    int l = 0;
    for (int t = lmax / 2; t >= 1; t /= 2)
        if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
    const int j = i + l * d;
    const int dnode = delta(keys, n, i, j);
    int s = 0;
    for (int div = 2;; div *= 2) {
        const int t = (l + div - 1) / div;
        if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
        if (t <= 1) break;
    }
    const int gamma = i + s * d + min(d, 0);
    const int lo = min(i, j), hi = max(i, j);
    const uint32_t lc = (lo == gamma) ? (kLeafBit | (uint32_t)gamma) : (uint32_t)gamma;
    const uint32_t rc = (hi == gamma + 1) ? (kLeafBit | (uint32_t)(gamma + 1)) : (uint32_t)(gamma + 1);
    left[i] = lc;
    right[i] = rc;
    range_lo[i] = (uint32_t)lo;
    range_hi[i] = (uint32_t)hi;
    if (lc & kLeafBit) parent_leaf[lc & ~kLeafBit] = i;
    else parent_int[lc] = i;
    if (rc & kLeafBit) parent_leaf[rc & ~kLeafBit] = i;
    else parent_int[rc] = i;
}

__device__ __forceinline__ void tri_box(const float* tri, const unsigned long long* keys, uint32_t leaf, float* mn,
                                        float* mx) {
    const float* v = tri + (size_t)(uint32_t)(keys[leaf] & 0xFFFFFFFFull) * 9;
    for (int k = 0; k < 3; ++k) {
        mn[k] = fminf(fminf(v[k], v[3 + k]), v[6 + k]);
        mx[k] = fmaxf(fmaxf(v[k], v[3 + k]), v[6 + k]);
    }
}

__device__ __forceinline__ void child_box(uint32_t c, const float* tri, const unsigned long long* keys,
                                          const float* boxes, float* mn, float* mx) {
    if (c & kLeafBit) {
        tri_box(tri, keys, c & ~kLeafBit, mn, mx);
    } else {
        const volatile float* b = boxes + (size_t)c * 6;
        for (int k = 0; k < 3; ++k) {
            mn[k] = b[k];
            mx[k] = b[3 + k];
        }
    }
}

// Bounds bottom-up; the second thread to reach a node computes it.
__global__ void bounds_kernel(const float* __restrict__ tri, const unsigned long long* __restrict__ keys, int n,
                              const uint32_t* __restrict__ left, const uint32_t* __restrict__ right,
                              const int* __restrict__ parent_int, const int* __restrict__ parent_leaf,
                              uint32_t* __restrict__ arrivals, float* boxes) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    int p = parent_leaf[k];
    while (p >= 0) {
        __threadfence();
        if (atomicAdd(&arrivals[p], 1u) == 0u) return;   // the sibling's thread finishes this node
        float lmn[3], lmx[3], rmn[3], rmx[3];
        child_box(left[p], tri, keys, boxes, lmn, lmx);
        child_box(right[p], tri, keys, boxes, rmn, rmx);
        volatile float* b = boxes + (size_t)p * 6;
        for (int c = 0; c < 3; ++c) {
            b[c] = fminf(lmn[c], rmn[c]);
            b[3 + c] = fmaxf(lmx[c], rmx[c]);
        }
        p = parent_int[p];
    }
}

__device__ __forceinline__ uint32_t subtree_size(uint32_t c, const uint32_t* range_lo, const uint32_t* range_hi) {
    if (c & kLeafBit) return 1u;
    return 2u * (range_hi[c] - range_lo[c] + 1u) - 1u;
}

// Post-order slot of every node: first slot of its block (left siblings on
// the path to the root) plus its block size minus one.
__global__ void postorder_kernel(int n, const uint32_t* __restrict__ left, const uint32_t* __restrict__ range_lo,
                                 const uint32_t* __restrict__ range_hi, const int* __restrict__ parent_int,
                                 const int* __restrict__ parent_leaf, uint32_t* __restrict__ slot_int,
                                 uint32_t* __restrict__ slot_leaf) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 2 * n - 1) return;
    const bool leaf = t >= n - 1;
    const uint32_t self = leaf ? (kLeafBit | (uint32_t)(t - (n - 1))) : (uint32_t)t;
    uint32_t start = 0;
    uint32_t cur = self;
    int p = leaf ? parent_leaf[self & ~kLeafBit] : parent_int[self];
    while (p >= 0) {
        if (left[p] != cur) start += subtree_size(left[p], range_lo, range_hi);
        cur = (uint32_t)p;
        p = parent_int[p];
    }
    const uint32_t slot = start + subtree_size(self, range_lo, range_hi) - 1u;
    if (leaf) slot_leaf[self & ~kLeafBit] = slot;
    else slot_int[self] = slot;
}

__global__ void write_kernel(const float* __restrict__ tri, const unsigned long long* __restrict__ keys, int n,
                             const uint32_t* __restrict__ left, const uint32_t* __restrict__ right,
                             const float* __restrict__ boxes, const uint32_t* __restrict__ slot_int,
                             const uint32_t* __restrict__ slot_leaf, uint32_t first_global, uint32_t node_offset,
                             orn_bvh_node* __restrict__ out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 2 * n - 1) return;
    orn_bvh_node node;
    memset(&node, 0, sizeof(node));
    uint32_t slot;
    if (t >= n - 1) {
        const uint32_t k = (uint32_t)(t - (n - 1));
        const uint32_t tri_id = (uint32_t)(keys[k] & 0xFFFFFFFFull);
        const float* v = tri + (size_t)tri_id * 9;
        for (int c = 0; c < 3; ++c) {
            node.left_aabb_min_or_v0[c] = v[c];
            node.left_aabb_max_or_v1[c] = v[3 + c];
            node.right_aabb_min_or_v2[c] = v[6 + c];
        }
        node.left_or_custom_id = first_global + tri_id;
        node.node_type = ORN_NODE_TRIANGLE;
        slot = slot_leaf[k];
    } else {
        float mn[3], mx[3];
        child_box(left[t], tri, keys, boxes, mn, mx);
        for (int c = 0; c < 3; ++c) {
            node.left_aabb_min_or_v0[c] = mn[c];
            node.left_aabb_max_or_v1[c] = mx[c];
        }
        child_box(right[t], tri, keys, boxes, mn, mx);
        for (int c = 0; c < 3; ++c) {
            node.right_aabb_min_or_v2[c] = mn[c];
            node.right_aabb_max_or_v3[c] = mx[c];
        }
        const uint32_t l = left[t], r = right[t];
        node.left_or_custom_id = node_offset + ((l & kLeafBit) ? slot_leaf[l & ~kLeafBit] : slot_int[l]);
        node.right_or_material_index = node_offset + ((r & kLeafBit) ? slot_leaf[r & ~kLeafBit] : slot_int[r]);
        node.node_type = ORN_NODE_INTERNAL;
        slot = slot_int[t];
    }
    out[slot] = node;
}

}  // namespace

int lbvh_build_all(const LbvhJob* jobs, size_t count) {
    int devices = 0;
    size_t most = 0, nodes = 0;   // triangles of the largest mesh, nodes of all with more than one
    for (size_t j = 0; j < count; ++j) {
        if (jobs[j].n == 0) return ORN_ERR_EMPTY_SCENE;
        if (jobs[j].n >= (1u << 31)) return ORN_ERR_INVALID_ARGUMENT;   // node and sort indices are int
        most = std::max<size_t>(most, jobs[j].n);
        if (jobs[j].n > 1) nodes += 2 * (size_t)jobs[j].n - 1;
    }
    const size_t room = std::min(nodes, std::max(kNodesAtOnce, 2 * most));   // nodes that the device holds
    if (count && (cudaGetDeviceCount(&devices) != cudaSuccess || devices == 0)) return ORN_ERR_NO_DEVICE;
    int st = ORN_OK;
    auto ok = [&](cudaError_t e) {
        if (e != cudaSuccess && st == ORN_OK) st = e == cudaErrorMemoryAllocation ? ORN_ERR_OUT_OF_MEMORY : ORN_ERR_CUDA;
        return st == ORN_OK;
    };
    // One allocation for all meshes: the working arrays for the largest, used
    // by one mesh after another in stream order, and the nodes, which are copied
    // back once as many meshes are queued as there is room for (8 meshes of 35k
    // triangles: an allocation per array and a wait per mesh took the builder
    // 15.4 ms, this 11.1, with the host's share of both).
    size_t temp_bytes = 0;
    if (most > 1 && !ok(cub::DeviceRadixSort::SortKeys(nullptr, temp_bytes, (const unsigned long long*)nullptr,
                                                       (unsigned long long*)nullptr, (int)most, 0, 64)))
        return st;
    unsigned char* mem = nullptr;
    size_t used = 0;
    auto place = [&](size_t bytes) {
        const size_t at = used;
        used += (bytes + 255) / 256 * 256;
        return at;
    };
    const size_t a_tri = place(most * 36), a_keys = place(most * 8), a_keys2 = place(most * 8), a_left = place(most * 4),
                 a_right = place(most * 4), a_lo = place(most * 4), a_hi = place(most * 4), a_arr = place(most * 4),
                 a_slot_int = place(most * 4), a_slot_leaf = place(most * 4), a_pint = place(most * 4),
                 a_pleaf = place(most * 4), a_boxes = place(most * 24), a_bounds = place(24), a_temp = place(temp_bytes),
                 a_out = place(room * sizeof(orn_bvh_node));
    cudaStream_t s = nullptr;
    if (most > 1 && ok(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking)) && ok(cudaMalloc((void**)&mem, used))) {
        float* d_tri = (float*)(mem + a_tri);
        unsigned long long *d_keys = (unsigned long long*)(mem + a_keys), *d_keys2 = (unsigned long long*)(mem + a_keys2);
        uint32_t *d_left = (uint32_t*)(mem + a_left), *d_right = (uint32_t*)(mem + a_right),
                 *d_lo = (uint32_t*)(mem + a_lo), *d_hi = (uint32_t*)(mem + a_hi), *d_arr = (uint32_t*)(mem + a_arr),
                 *d_slot_int = (uint32_t*)(mem + a_slot_int), *d_slot_leaf = (uint32_t*)(mem + a_slot_leaf),
                 *d_bounds = (uint32_t*)(mem + a_bounds);
        int *d_pint = (int*)(mem + a_pint), *d_pleaf = (int*)(mem + a_pleaf);
        float* d_boxes = (float*)(mem + a_boxes);
        orn_bvh_node* const d_first = (orn_bvh_node*)(mem + a_out);
        orn_bvh_node* d_out = d_first;
        size_t back = 0;   // meshes before this one are copied back
        auto copy_back = [&](size_t end) {
            d_out = d_first;
            for (; back < end && st == ORN_OK; ++back) {
                if (jobs[back].n == 1) continue;
                const size_t k = 2 * (size_t)jobs[back].n - 1;
                ok(cudaMemcpyAsync(jobs[back].out, d_out, k * sizeof(orn_bvh_node), cudaMemcpyDeviceToHost, s));
                d_out += k;
            }
            d_out = d_first;
        };
        for (size_t j = 0; j < count && st == ORN_OK; ++j) {
            const size_t nn = jobs[j].n, ni = nn - 1;
            const uint32_t n = jobs[j].n;
            if (n == 1) continue;
            if ((size_t)(d_out - d_first) + 2 * nn - 1 > room) copy_back(j);
            const int B = 256;
            const unsigned gn = (unsigned)((nn + B - 1) / B), gall = (unsigned)((2 * nn - 1 + B - 1) / B);
            ok(cudaMemcpyAsync(d_tri, jobs[j].tri, nn * 36, cudaMemcpyHostToDevice, s));
            ok(cudaMemsetAsync(d_arr, 0, ni * 4, s));
            ok(cudaMemsetAsync(d_pint, 0xFF, ni * 4, s));   // root's parent = -1
            ok(cudaMemsetAsync(d_bounds, 0xFF, 12, s));
            ok(cudaMemsetAsync(d_bounds + 3, 0, 12, s));
            centroid_kernel<<<std::min(gn, 304u), B, 0, s>>>(d_tri, n, d_bounds);
            ok(cudaGetLastError());
            morton_kernel<<<gn, B, 0, s>>>(d_tri, n, d_bounds, d_keys);
            ok(cudaGetLastError());
            size_t tb = temp_bytes;
            ok(cub::DeviceRadixSort::SortKeys(mem + a_temp, tb, d_keys, d_keys2, (int)n, 0, 64, s));
            hierarchy_kernel<<<gn, B, 0, s>>>(d_keys2, (int)n, d_left, d_right, d_pint, d_pleaf, d_lo, d_hi);
            ok(cudaGetLastError());
            bounds_kernel<<<gn, B, 0, s>>>(d_tri, d_keys2, (int)n, d_left, d_right, d_pint, d_pleaf, d_arr, d_boxes);
            ok(cudaGetLastError());
            postorder_kernel<<<gall, B, 0, s>>>((int)n, d_left, d_lo, d_hi, d_pint, d_pleaf, d_slot_int, d_slot_leaf);
            ok(cudaGetLastError());
            write_kernel<<<gall, B, 0, s>>>(d_tri, d_keys2, (int)n, d_left, d_right, d_boxes, d_slot_int, d_slot_leaf,
                                            jobs[j].first_global, jobs[j].node_offset, d_out);
            ok(cudaGetLastError());
            d_out += 2 * nn - 1;
        }
        copy_back(count);
        ok(cudaStreamSynchronize(s));
    }
    if (s) {
        cudaStreamSynchronize(s);   // (an error above may have left work queued)
        cudaStreamDestroy(s);
    }
    if (mem) cudaFree(mem);
    for (size_t j = 0; j < count && st == ORN_OK; ++j) {
        if (jobs[j].n != 1) continue;
        orn_bvh_node node;
        std::memset(&node, 0, sizeof(node));
        std::memcpy(node.left_aabb_min_or_v0, jobs[j].tri, 12);
        std::memcpy(node.left_aabb_max_or_v1, jobs[j].tri + 3, 12);
        std::memcpy(node.right_aabb_min_or_v2, jobs[j].tri + 6, 12);
        node.left_or_custom_id = jobs[j].first_global;
        node.node_type = ORN_NODE_TRIANGLE;
        jobs[j].out[0] = node;
    }
    return st;
}

}  // namespace orn
