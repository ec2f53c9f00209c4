"""Order of the near-field work list (near_order in p2p.cu), which no entry point returns: a program
compiled from the sources prints the list before and after (-m gpu)."""
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "p2p.cu"
#include "tree.cu"
int bbfmm_set_cuda_error(cudaError_t e, const char *, const char *, int) { return e == cudaSuccess ? 0 : 2; }
int bbfmm_set_error(int code, const char *) { return code; }
using namespace bbfmm;
#define OK(x) do { if ((x) != 0) return 1; } while (0)
int main(int argc, char **argv) {  // maxlev, threads, then the particles of every leaf
  const int maxlev = atoi(argv[1]), threads = atoi(argv[2]);
  const int64_t nl = pow8i(maxlev);
  std::vector<int> ls(nl + 1, 0);
  for (int64_t m = 0, c; m < nl; ++m) {
    if (scanf("%ld", &c) != 1) return 1;
    ls[m + 1] = ls[m] + (int)c;
  }
  const int N = ls[nl];
  int *ls_d;
  void *work, *scratch;
  OK(cudaMalloc(&ls_d, 4 * (nl + 1)));
  OK(cudaMemcpy(ls_d, ls.data(), 4 * (nl + 1), cudaMemcpyHostToDevice));
  OK(cudaMalloc(&work, near_work_bytes(N, maxlev, 1)));
  for (int rep = 0; rep < 2; ++rep) {
    int n = 0, flag = 0;
    OK(near_work_build(N, ls_d, maxlev, 1, threads, work, 0, &n, &flag, nullptr, 0));
    OK(flag);
    std::vector<int2> a(n), b(n);
    const int2 *items = near_work_items(work, maxlev, 1);
    OK(cudaMemcpy(a.data(), items, 8 * (size_t)n, cudaMemcpyDeviceToHost));
    OK(cudaMalloc(&scratch, near_order_bytes(n)));
    OK(near_order(N, ls_d, maxlev, 1, threads, work, n, scratch, 0));
    OK(cudaDeviceSynchronize());
    OK(cudaFree(scratch));
    OK(cudaMemcpy(b.data(), items, 8 * (size_t)n, cudaMemcpyDeviceToHost));
    printf("%d\n", n);
    for (const auto *v : {&a, &b})
      for (const int2 &i : *v) printf("%d %d\n", i.x, i.y);
  }
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    from bbfmm_b200 import build
    d = tmp_path_factory.mktemp("near_order")
    (d / "t.cu").write_text(SRC)
    r = subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I" + os.path.join(build.ROOT, "include"),
                        "-I" + build.CSRC, "-o", str(d / "t"), str(d / "t.cu")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return str(d / "t")


def _cost(item, ls, maxlev, threads):
    from bbfmm_b200.fmm import morton_to_grid
    x, j = item
    if x >= 0:
        n = ls[64 * x + 64] - ls[64 * x]
        return -(-n // threads) * 27 * n / 64
    m = -x - 1
    n1 = 2 ** maxlev
    ix, iy, iz = (int(v) for v in morton_to_grid(m, maxlev))
    src = 0
    for a in (-1, 0, 1):
        for b in (-1, 0, 1):
            for c in (-1, 0, 1):
                g = (ix + a, iy + b, iz + c)
                if min(g) >= 0 and max(g) < n1:
                    k = sum(((g[0] >> t & 1) << 2 | (g[1] >> t & 1) << 1 | (g[2] >> t & 1)) << 3 * t for t in range(maxlev))
                    src += ls[k + 1] - ls[k]
    left = ls[m + 1] - ls[m] - j * threads
    return src / (threads // min(left, threads))


@pytest.mark.parametrize("threads", [64, 128, 256])
@pytest.mark.parametrize("kind", ["clustered", "uniform", "one leaf"])
def test_longest_items_first_and_neighbours_together(program, threads, kind):
    maxlev = 3
    rng = np.random.default_rng(threads)
    counts = {"clustered": rng.integers(0, 6, 512) + (rng.random(512) < 0.1) * rng.integers(0, 3000, 512),
              "uniform": rng.integers(4, 12, 512), "one leaf": np.eye(512, dtype=int)[77] * 5000}[kind]
    ls = np.concatenate([[0], np.cumsum(counts)])
    out = subprocess.run([program, str(maxlev), str(threads)], input=" ".join(map(str, counts)), capture_output=True, text=True)
    assert out.returncode == 0
    lines = out.stdout.splitlines()
    n = int(lines[0])
    assert int(lines[1 + 2 * n]) == n and lines[1 + n:1 + 2 * n] == lines[2 + 3 * n:2 + 4 * n]  # the same list again
    before = [tuple(map(int, s.split())) for s in lines[1:1 + n]]
    after = [tuple(map(int, s.split())) for s in lines[1 + n:1 + 2 * n]]
    assert sorted(before) == sorted(after)
    cost = np.array([_cost(i, ls, maxlev, threads) for i in after])
    # 32 buckets an octave: a later item is longer by less than one bucket
    assert np.all(np.log2(cost[1:] + 1) < np.log2(cost[:-1] + 1) + 1 / 32 + 1e-4)
    where = {i: k for k, i in enumerate(before)}
    place = np.array([where[i] for i in after])
    same = cost[1:] == cost[:-1]
    assert np.all(place[1:][same] > place[:-1][same])  # items of one cost keep the list's order
