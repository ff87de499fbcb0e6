"""Device memory of the GPU tree builder: by its largest mesh, not by all of
them.  The library's own lbvh.cu.o is linked with counting stand-ins of
cudaMalloc and cudaFree."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from zig_ornament_gb300 import build, ornament

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cuda_runtime.h>
#include <map>
#include "lbvh.h"

static size_t live = 0, peak = 0;
static std::map<void*, size_t> sizes;

extern "C" cudaError_t __real_cudaMalloc(void**, size_t);
extern "C" cudaError_t __real_cudaFree(void*);
extern "C" cudaError_t __wrap_cudaMalloc(void** p, size_t n) {
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

extern "C" int build_all(const orn::LbvhJob* jobs, size_t count, unsigned long long* out) {
    live = peak = 0;
    const int st = orn::lbvh_build_all(jobs, count);
    out[0] = peak;
    out[1] = live;
    return st;
}
"""


class Job(C.Structure):
    _fields_ = [("tri", C.c_void_p), ("n", C.c_uint32), ("first_global", C.c_uint32), ("node_offset", C.c_uint32),
                ("out", C.c_void_p)]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("lbvh")
    (d / "t.cpp").write_text(SOURCE)
    subprocess.run([build._nvcc(), "-std=c++17", f"-I{build.INCLUDE}", f"-I{build.CSRC}", "-Xcompiler", "-fPIC", "-shared",
                    *build.ARCH, "-Xlinker", "--wrap=cudaMalloc", "-Xlinker", "--wrap=cudaFree", str(d / "t.cpp"),
                    str(build.BUILD / "lbvh.cu.o"), "-o", str(d / "t.so")], check=True)
    return C.CDLL(str(d / "t.so"))


def _build(lib, sizes, alone):
    """Nodes of meshes of `sizes` triangles, and the peak of memory."""
    rs = np.random.default_rng(len(sizes))
    tris = [rs.uniform(-1, 1, (n, 9)).astype(np.float32) for n in sizes]
    out = [np.zeros(2 * n - 1, ornament.NODE_DTYPE) for n in sizes]
    first = np.concatenate([[0], np.cumsum(sizes)])
    jobs = (Job * len(sizes))(*[Job(t.ctypes.data, len(t), int(first[i]), int(2 * first[i] - i), o.ctypes.data)
                                for i, (t, o) in enumerate(zip(tris, out))])
    got, peak = (C.c_ulonglong * 2)(), 0
    for i in range(len(sizes) if alone else 1):
        assert lib.build_all(C.byref(jobs, i * C.sizeof(Job)), C.c_size_t(1 if alone else len(sizes)), got) == 0
        assert got[1] == 0
        peak = max(peak, got[0])
    return out, peak


@pytest.mark.parametrize("sizes", [[1], [2, 1, 3], [40_000] * 30, [1, 600_000, 5, 1, 400_000, 200_000, 70_000]])
def test_many_meshes(lib, sizes):
    want, least = _build(lib, sizes, True)
    got, peak = _build(lib, sizes, False)
    for a, b in zip(want, got):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
    # the largest mesh's working arrays, and 64 MB (2^20 nodes) of the others' nodes
    assert peak <= least + (64 << 20) + (1 << 20)
