"""Launch rules of the CUDA sources that are plain host functions, compiled here without a GPU."""
import os
import subprocess

from bbfmm_b200 import build

SRC = r"""
#include <cstdio>
#include "solver.cuh"
int main() {
  for (int level = 2; level <= 5; ++level)
    for (int nsets = 1; nsets <= 300; ++nsets)
      std::printf("%d %d %lld %d\n", level, nsets, (long long)bbfmm::tc2_ctas(bbfmm::tc2_tiles(level, nsets) / 8),
                  bbfmm::tc2_groups(level, nsets));
}
"""


def test_offset_groups_of_the_tensor_core_m2l_fit_the_gpu(tmp_path):
    """A level's groups times the CTAs of its launch (pairs of a class's tiles, one CTA an SM) stay
    within the 148 SMs, and one group more would not, up to the nine that are worth their partial
    sums."""
    (tmp_path / "t.cu").write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.run([build.nvcc(), "-std=c++17", "-Xcompiler", "-O1", "-I" + os.path.join(build.ROOT, "include"), "-I" + build.CSRC,
                    "-o", exe, str(tmp_path / "t.cu")], check=True)
    rows = [tuple(map(int, ln.split())) for ln in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()]
    assert len(rows) == 1200
    for level, nsets, ctas, g in rows:
        sets = {2: 32, 3: 4}.get(level, 1)  # stacked sets of a tile
        per_class = -(-nsets // sets) * (8 ** (level - 1) // 256 or 1)
        assert ctas == 16 * -(-per_class // 2), (level, nsets)
        assert 1 <= g <= 9 and (g == 1 or g * ctas <= 148), (level, nsets, ctas, g)
        assert g == 9 or (g + 1) * ctas > 148, (level, nsets, ctas, g)
