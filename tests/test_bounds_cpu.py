"""The bounds-checked build's element offsets (common.cuh, -DERF_B200_BOUNDS),
compiled for the host: an offset that leaves the array after a neighbour
level was added to it sets the status bit and reads element 0."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r'''
#include <cstdio>
#include "common.cuh"
using namespace erfb;
int main() {
    int flag = 0;
    Geo g{};
    g.nx = 4; g.ny = 3; g.nz = 5; g.sk = 12; g.ncell = 60; g.nzf = 72; g.oob = &flag;
    const uint32_t sk = 12;
    const Elem e{2u + 4u * 1u + sk * 4u, (uint32_t)g.nzf, g.oob};   // cell (2, 1, 4)
    const uint32_t up = e + sk, down = e - 4 * sk, two = e + (uint32_t)-2 * sk;
    printf("%u %u %u %d ", up, down, two, flag);
    const uint32_t above = e + 2 * sk;
    printf("%u %d ", above, flag & ST_BOUNDS);
    flag = 0;
    const uint32_t below = e - 5 * sk;
    printf("%u %d\n", below, flag & ST_BOUNDS);
    return 0;
}
'''


def test_offsets_added_to_an_element_are_checked(tmp_path):
    src, exe = tmp_path / "t.cu", tmp_path / "t"
    src.write_text(SRC)
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-std=c++17", "-DERF_B200_BOUNDS=1", "--expt-relaxed-constexpr", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-I", os.path.join(ROOT, "erf_b200", "csrc"), "-I",
                    os.path.join(ROOT, "include"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()
    bit = out[5]
    assert out[:4] == ["66", "6", "30", "0"], out
    assert out[4] == "0" and bit != "0" and out[6:] == ["0", bit], out
