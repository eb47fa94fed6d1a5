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


STRIPS = r"""
#include "sw_strip.cuh"
#include "sw_whole.cuh"
#include <cstdio>
using namespace swb;
int main()
{
    for (uint32_t W = 8; W <= 32; W *= 2) {
        const uint32_t most[2] = {strip_smem_max(W, 1), strip_smem_max(W, kBandsMax)};
        for (uint32_t tx = 8; tx <= 32; tx *= 2)
            for (uint32_t ty = 2; ty <= 32; ++ty) {
                uint32_t misaligned = 0, large = 0;
                for (uint32_t tbx = 1; tbx <= 128 / tx; ++tbx)
                    for (uint32_t tby = 1; tby == 1 || tby * ty <= 32; ++tby)
                        for (uint32_t bands = 1; bands <= kBandsMax; ++bands) {
                            const Geo g = make_geo(1024, 1024, tx, ty, tbx, tby);
                            const StripSmem s = strip_smem(g, W, bands);
                            // parent and words: uint4; last and pairs: uint2; draws, sums: 32 bits
                            misaligned += s.parent % 16 || s.words % 16 || s.last % 8 || s.draws % 4 || s.sums % 4 ||
                                          s.pairs % 8;
                            large += s.total > 48 * 1024 || (bands == 1 && s.total > most[0]) ||
                                     (bands == kBandsMax && s.total > most[1]);
                        }
                // the one-kernel form, where make_whole takes the lattice
                for (uint32_t L0 = 2; L0 <= 1056; L0 += L0 < 130 ? 2 : 62)
                    for (uint32_t L1 = 2; L1 <= 1056; L1 += L1 < 130 ? 2 : 62) {
                        const Whole w = make_whole(L0, L1, tx, ty);
                        if (!w.ctas)
                            continue;
                        const WholeSmem s = whole_smem(w, W);
                        // parent and scan: uint4; raw and pairs: uint2; the rest 32 bits
                        misaligned += w.pitch % 4 || s.raw % 8 || s.scan % 16 || s.pairs % 8 ||
                                      (s.spin | s.work | s.counts | s.edge | s.sums) % 4;
                        large += s.total > kWholeSmemMax;
                    }
                std::printf("%u %u %u %u %u\n", W, tx, ty, misaligned, large);
            }
    }
}
"""


def test_2d_assign_layouts(tmp_path):
    rows = [tuple(map(int, line.split())) for line in _run(tmp_path, STRIPS)]
    assert len(rows) == 3 * 3 * 31
    assert [r[:3] for r in rows if r[3]] == []  # (W, tile) with an area off its alignment
    assert [r[:3] for r in rows if r[4]] == []  # (W, tile) that does not fit
