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

OPT_IN = r"""
#include <cstdio>
#include "smem_opt_in.h"
static int device = 0, calls[4] = {}, fail = 0;
extern "C" cudaError_t CUDARTAPI cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t CUDARTAPI cudaFuncSetAttribute(const void *, enum cudaFuncAttribute, int) {
  ++calls[device];
  return fail ? cudaErrorInvalidValue : cudaSuccess;
}
void kernel_a(int) {}
void kernel_b(int) {}
int main() {
  using bbfmm::smem_opt_in;
  for (device = 0; device < 3; ++device)
    for (int i = 0; i < 2; ++i) smem_opt_in<kernel_a>(100000);
  device = 0;
  smem_opt_in<kernel_b>(100000);
  std::printf("%d %d %d\n", calls[0], calls[1], calls[2]);
  device = 3;
  fail = 1;
  const int first = smem_opt_in<kernel_a>(100000) != cudaSuccess;
  fail = 0;
  const int second = smem_opt_in<kernel_a>(100000) == cudaSuccess;
  std::printf("%d %d %d\n", first, second, calls[3]);
}
"""


def test_every_device_opts_into_its_shared_memory(tmp_path):
    """The shared-memory attribute belongs to a kernel on one device: each device of a process sets it
    once per kernel, and a call that failed is made again. (The CUDA runtime is a stand-in here.)"""
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    (tmp_path / "t.cpp").write_text(OPT_IN)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-I" + build.CSRC, "-I" + (cuda if os.path.isdir(cuda) else "/usr/local/cuda/include"),
                    "-o", exe, str(tmp_path / "t.cpp")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()
    assert out == ["2", "1", "1", "1", "1", "2"]


def test_no_launcher_keeps_its_own_flag():
    """Every opt-in goes through that one function."""
    for f in os.listdir(build.CSRC):
        if f != "smem_opt_in.h" and f.endswith((".cu", ".cuh", ".h")):
            assert "cudaFuncSetAttribute" not in open(os.path.join(build.CSRC, f)).read(), f
