"""Device memory of scene creation: without near-first trees the blob's nodes
are all that stays, and a scene whose near-first trees find no memory is walked
over the blob's.  The library's own tree_build.cu.o is linked with counting
stand-ins of cudaMalloc and cudaFree."""
import ctypes as C
import subprocess

import numpy as np
import pytest

import test_gpu_near as near
from zig_ornament_gb300 import build, ornament

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cuda_runtime.h>
#include <map>
#include <vector>
#include "tree_build.h"

static int fail_at = -1, calls = 0;
static size_t live = 0, peak = 0;
static std::map<void*, size_t> sizes;

extern "C" cudaError_t __real_cudaMalloc(void**, size_t);
extern "C" cudaError_t __real_cudaFree(void*);
extern "C" cudaError_t __wrap_cudaMalloc(void** p, size_t n) {
    if (calls++ == fail_at) n = (size_t)1 << 60;   // more than there is: the runtime's own failure
    const cudaError_t e = __real_cudaMalloc(p, n);
    if (e == cudaSuccess) {
        sizes[*p] = n;
        live += n;
        peak = peak < live ? live : peak;
    }
    return e;
}
extern "C" cudaError_t __wrap_cudaFree(void* p) {
    live -= sizes[p];
    sizes.erase(p);
    return __real_cudaFree(p);
}

// out: status, last error, allocations tried, near, bytes that stay, peak
extern "C" void trees(const orn_scene_blob* blob, int fail, float* nodes, unsigned long long* out) {
    float4* x = nullptr;
    __real_cudaMalloc((void**)&x, blob->transforms_len * 64ull);
    cudaMemcpy(x, blob->transforms, blob->transforms_len * 64ull, cudaMemcpyHostToDevice);
    fail_at = fail;
    calls = 0;
    live = peak = 0;
    orn::SceneDev scene{};
    orn::NodeFacts facts{};
    std::vector<void*> allocs;
    out[0] = orn::build_scene_trees(blob, x, &scene, &facts, &allocs, nullptr);
    out[1] = cudaGetLastError();
    out[2] = calls;
    out[3] = scene.near;
    out[4] = live;
    out[5] = peak;
    if (out[0] == cudaSuccess)
        cudaMemcpy(nodes, scene.nodes, ((size_t)blob->tlas_nodes_len + blob->blas_nodes_len) * 64, cudaMemcpyDeviceToHost);
    for (void* p : allocs) __wrap_cudaFree(p);
    out[6] = live;
    __real_cudaFree(x);
}
"""


@pytest.fixture(scope="module")
def trees(tmp_path_factory):
    d = tmp_path_factory.mktemp("trees")
    (d / "t.cpp").write_text(SOURCE)
    subprocess.run([build._nvcc(), "-std=c++17", f"-I{build.INCLUDE}", f"-I{build.CSRC}", "-Xcompiler", "-fPIC", "-shared",
                    *build.ARCH, "-Xlinker", "--wrap=cudaMalloc", "-Xlinker", "--wrap=cudaFree", str(d / "t.cpp"),
                    str(build.BUILD / "tree_build.cu.o"), "-o", str(d / "t.so")], check=True)
    lib = C.CDLL(str(d / "t.so"))

    def run(bvh, fail=-1):
        blob, keep = bvh.blob()
        n = len(bvh.tlas_nodes) + len(bvh.blas_nodes)
        nodes = np.zeros((n, 16), np.uint32)
        out = (C.c_ulonglong * 7)()
        lib.trees(C.byref(blob), fail, C.c_void_p(nodes.ctypes.data), out)
        del keep
        return dict(zip(("status", "last", "calls", "near", "stays", "peak", "left"), out)), nodes
    return run


def _bvh():
    return ornament.Bvh(near.SCENES["instanced"]())


def test_what_stays(trees):
    bvh = _bvh()
    n = len(bvh.tlas_nodes) + len(bvh.blas_nodes)
    got, _ = trees(bvh)
    assert (got["status"], got["near"] > 0, got["left"]) == (0, True, 0)
    assert 64 * n < got["stays"] <= 2 * 64 * n
    inner = np.nonzero(bvh.blas_nodes["node_type"] == 0)[0]
    kinds = bvh.blas_nodes["node_type"][bvh.blas_nodes["left_or_custom_id"][inner]]
    bvh.blas_nodes["left_aabb_min_or_v0"][inner[kinds == 3][0]] -= 0.05   # (no near-first trees)
    got, _ = trees(bvh)
    assert (got["status"], got["near"], got["left"]) == (0, 0, 0)
    assert got["stays"] == 64 * n


def test_no_memory_for_the_trees(trees):
    bvh = _bvh()
    n = len(bvh.tlas_nodes) + len(bvh.blas_nodes)
    whole, nodes = trees(bvh)
    must = 0
    for k in range(whole["calls"]):
        got, again = trees(bvh, k)
        assert (got["last"], got["left"]) == (0, 0) or got["status"] == 2   # cudaErrorMemoryAllocation
        if got["status"] == 2:
            must += 1
            assert got["left"] == 0
        else:
            assert (got["status"], got["near"], got["stays"]) == (0, 0, 64 * n)
            assert np.array_equal(again, nodes)
    assert must <= 2   # the nodes, and a byte for each
    assert whole["calls"] >= must + 3
