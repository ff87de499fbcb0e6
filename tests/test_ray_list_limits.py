"""The longest ray list that the persistent ray kernel takes: its 32-bit count of
rays handed out has to pass the end once for every resident warp without coming
round (the kernel would then begin at the first ray again, for ever)."""
import re
import subprocess

from zig_ornament_gb300 import build


def _most_rays(tmp_path):
    """The limit that orn_trace_rays compares its count with."""
    limit = re.search(r"bool near = .*?count (<=?) ([^;]+);", (build.CSRC / "capi.cu").read_text())
    (tmp_path / "t.cpp").write_text('#include <cstdio>\n#include "pt_kernels.h"\n'
                                    f'int main() {{ std::printf("%llu", (unsigned long long)({limit[2]})); }}\n')
    subprocess.run([build._nvcc(), "-std=c++17", f"-I{build.INCLUDE}", f"-I{build.CSRC}", str(tmp_path / "t.cpp"), "-o",
                    str(tmp_path / "t")], check=True)
    most = int(subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout)
    return most - (limit[1] == "<")


def test_the_count_of_rays_does_not_come_round(tmp_path):
    most = _most_rays(tmp_path)
    warps = 160 * 64   # more than any GPU of this kind holds
    for count in (most, most - 1, most - 12345):
        counter = count - 1000
        for _ in range(warps):
            exhausted = False
            for _ in range(64):   # (a warp takes up to 32 rays at a time until the end is reached)
                base, counter = counter, (counter + 32) % 2**32
                if (base + 32) % 2**32 >= count:
                    exhausted = True
                    break
            assert exhausted
