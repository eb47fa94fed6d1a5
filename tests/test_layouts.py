"""The kernels' shared-memory layouts for every tile, lcg width and block shape that the entry points
accept: each area starts, and each warp's slice of it follows, on the alignment of the widest access made
through it, and the whole fits what the launch may ask for.  Host code of the kernels' own headers, run
without a GPU."""
import subprocess

from computational_physics_b200 import build


def _run(tmp_path, source):
    """Output lines of a host program compiled against csrc/."""
    src, exe = tmp_path / "layout.cu", tmp_path / "layout"
    src.write_text(source)
    subprocess.run([build.nvcc(), *build.ARCH, *build.NVCC_FLAGS, "-I", build.CSRC, "-o", str(exe), str(src)],
                   check=True, timeout=300)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=300).stdout.splitlines()


ASSIGN3 = r"""
#include "sw_3d.cuh"
#include <cstdio>
using namespace swb;
template <int W> void walk()
{
    for (uint32_t tx = 8; tx <= 32; tx *= 2)
        for (uint32_t ty = 1; ty <= 8; ++ty)
            for (uint32_t tz = 1; tz <= 8; ++tz) {
                uint32_t misaligned = 0, large = 0;
                for (uint32_t nx = 1; nx <= 32 / tx; ++nx)
                    for (uint32_t ny = 1; ny <= k3Rows / ty; ++ny)
                        for (uint32_t nz = 1; nz <= k3Layers / tz; ++nz) {
                            const Geo3 g = make_geo3(nx * tx, ny * ty, nz * tz, tx, ty, tz);
                            const Assign3Smem s = assign3_smem<W>(g);
                            // raw and scan: uint4; a piece's scan: two uint4 a row; work: uint2 a row; links:
                            // uint16; sums: int; pairs: uint2
                            misaligned += s.raw % 16 || s.scan % 16 || s.work % 8 || s.wcap % 2 || s.links % 2 ||
                                          s.sums % 4 || s.pairs % 8;
                            large += s.total > k3SmemMax || pieces3(g) * 32 > k3MaxThreads || s.wcap < 2 * s.rows;
                        }
                std::printf("%d %u %u %u %u %u\n", W, tx, ty, tz, misaligned, large);
            }
}
int main() { walk<8>(); walk<16>(); walk<32>(); }
"""


def test_3d_assign_layout(tmp_path):
    rows = [tuple(map(int, line.split())) for line in _run(tmp_path, ASSIGN3)]
    assert len(rows) == 3 * 3 * 8 * 8
    assert [r[:4] for r in rows if r[4]] == []  # (W, tile) with an area off its alignment
    assert [r[:4] for r in rows if r[5]] == []  # (W, tile) that does not fit
