"""Which trees a batch walks: by what most of its work gains from, not by its
one context that does not."""
import subprocess

import pytest

from zig_ornament_gb300 import build

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "batch.h"
// per context: who walks its near-first trees, passes, whether the FMNMX slab test will do
int main(int n, char** a) {
    orn::BatchWalk walk;
    for (int i = 1; i + 2 < n; i += 3) {
        orn::BatchView v{};
        v.cp.width = 100;
        v.cp.height = 50;
        v.scene.near = std::atoi(a[i]);
        v.spp = std::atoi(a[i + 1]);
        walk.add(v, std::atoi(a[i + 2]) != 0);
    }
    std::printf("%d", walk.slabs());
}
"""
EXACT, FAST, NEAR = 0, 1, 2


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("walk")
    (d / "t.cpp").write_text(SOURCE)
    subprocess.run([build._nvcc(), "-std=c++17", f"-I{build.INCLUDE}", f"-I{build.CSRC}", str(d / "t.cpp"), "-o", str(d / "t")],
                   check=True)
    return d / "t"


@pytest.mark.parametrize("contexts,walk", [
    ([(2, 4, 1)], NEAR), ([(1, 4, 1)], FAST), ([(0, 4, 1)], FAST), ([(2, 4, 0)], EXACT),
    ([(2, 4, 1), (2, 4, 1), (1, 4, 1)], NEAR),      # one that does not gain
    ([(2, 4, 1), (1, 16, 1)], FAST),                # most of the work does not
    ([(2, 40, 1), (0, 4, 1)], FAST),                # one without near-first trees
    ([(2, 40, 1), (1, 4, 0)], EXACT)])
def test_walk(program, contexts, walk):
    args = [str(x) for c in contexts for x in c]
    assert int(subprocess.run([str(program), *args], check=True, capture_output=True, text=True).stdout) == walk
