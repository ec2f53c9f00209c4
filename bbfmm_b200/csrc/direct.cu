// FP64 direct O(N^2) sum on sampled targets (the reference's direct code, DirectCalc3D /
// EvaluateField, bbfmm.c:471-504 and 880-913): out[t] = q_i sum_{x_j != x_i} q_j / |x_j - x_i|
// for i = targets[t]. Used to state the error of every run against an exact sum.
//
// A cluster of eight CTAs takes 32 targets: CTA c streams the c-th eighth of the sources through
// shared memory in tiles of 256, and its eight warps take every eighth source of a tile for all 32
// targets (lane = target), so a few thousand targets fill the chip -- with one thread per target
// 4,096 of them were 32 CTAs, each walking all sources alone. Every thread keeps
// Neumaier-compensated FP64 sums; the 64 partial sums of a target are added in a fixed order, also
// compensated. Bound by FP64 issue: about 30 operations a pair (separation, rsqrt, compensation).
#include <cooperative_groups.h>

#include "common.cuh"

namespace bbfmm {

namespace cg = cooperative_groups;

namespace ds {
constexpr int TARGETS = 32, WARPS = 8, CTAS = 8, TILE = 256;
}

__device__ __forceinline__ void neumaier_add(double &s, double &c, double v) {
  const double y = s + v;
  c += (fabs(s) >= fabs(v)) ? ((s - y) + v) : ((v - y) + s);
  s = y;
}

// FIELD false: out = q_i pot_i. FIELD: the potential and its gradient at the targets, without the
// target-charge factor (the exact counterpart of bbfmm_b200_solve_fields): pot[t] = sum_{x_j != x_i}
// q_j / r_ij and field[3t + a] = sum q_j (x_j - x_i)_a / r_ij^3. The reference has no gradient code;
// this is the analytic derivative of its 1/r kernel.
template <bool FIELD>
__global__ void __cluster_dims__(1, ds::CTAS, 1) __launch_bounds__(32 * ds::WARPS)
    direct_kernel(int N, const double *__restrict__ xyz, const double *__restrict__ q, int nt,
                  const int *__restrict__ targets, double *__restrict__ pot, double *__restrict__ fld) {
  constexpr int NS = FIELD ? 4 : 1;  // sums per target
  __shared__ double sx[ds::TILE], sy[ds::TILE], sz[ds::TILE], sq[ds::TILE];
  __shared__ double part[ds::WARPS][2 * NS][ds::TARGETS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int t = blockIdx.x * ds::TARGETS + lane;
  const int i = t < nt ? targets[t] : 0;
  const double fx = xyz[3 * (int64_t)i], fy = xyz[3 * (int64_t)i + 1], fz = xyz[3 * (int64_t)i + 2];
  double s[NS], c[NS];
#pragma unroll
  for (int k = 0; k < NS; ++k) s[k] = c[k] = 0.0;
  const int c0 = (int)((int64_t)N * blockIdx.y / ds::CTAS), c1 = (int)((int64_t)N * (blockIdx.y + 1) / ds::CTAS);
  for (int j0 = c0; j0 < c1; j0 += ds::TILE) {
    const int n = min(ds::TILE, c1 - j0);
    __syncthreads();
    if (tid < n) {
      const int64_t j = j0 + tid;
      sx[tid] = xyz[3 * j]; sy[tid] = xyz[3 * j + 1]; sz[tid] = xyz[3 * j + 2]; sq[tid] = q[j];
    }
    __syncthreads();
#pragma unroll 4
    for (int e = warp; e < n; e += ds::WARPS) {
      const double dx = sx[e] - fx, dy = sy[e] - fy, dz = sz[e] - fz;
      const double rr = dx * dx + dy * dy + dz * dz;
      if (rr != 0.0) {
        const double ir = rsqrt(rr), v = sq[e] * ir;
        neumaier_add(s[0], c[0], v);
        if constexpr (FIELD) {
          const double v3 = v * ir * ir;
          neumaier_add(s[1], c[1], v3 * dx);
          neumaier_add(s[2], c[2], v3 * dy);
          neumaier_add(s[3], c[3], v3 * dz);
        }
      }
    }
  }
#pragma unroll
  for (int k = 0; k < NS; ++k) {
    part[warp][2 * k][lane] = s[k];
    part[warp][2 * k + 1][lane] = c[k];
  }
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  if (blockIdx.y == 0 && warp < NS) {  // warp k adds the partial sums of quantity k
    double ts = 0.0, tc = 0.0;
    for (int r = 0; r < ds::CTAS; ++r) {
      const double *p = cluster.map_shared_rank(&part[0][0][0], r);
      for (int w = 0; w < ds::WARPS; ++w) {
        neumaier_add(ts, tc, p[(w * 2 * NS + 2 * warp) * ds::TARGETS + lane]);
        tc += p[(w * 2 * NS + 2 * warp + 1) * ds::TARGETS + lane];
      }
    }
    if (t < nt) {
      if constexpr (!FIELD) pot[t] = q[i] * (ts + tc);
      else if (warp == 0) {
        if (pot) pot[t] = ts + tc;
      } else if (fld) {
        fld[3 * (int64_t)t + warp - 1] = ts + tc;
      }
    }
  }
  cluster.sync();  // the other CTAs' partial sums stay until they are read
}

int launch_direct_fp64(int N, const double *xyz, const double *q, int nt, const int *targets, double *out,
                       cudaStream_t s) {
  if (nt <= 0) return BBFMM_OK;
  direct_kernel<false><<<dim3((nt + ds::TARGETS - 1) / ds::TARGETS, ds::CTAS), 32 * ds::WARPS, 0, s>>>(N, xyz, q, nt, targets,
                                                                                                     out, nullptr);
  return bbfmm_set_cuda_error(cudaGetLastError(), "direct", __FILE__, __LINE__);
}

int launch_direct_field_fp64(int N, const double *xyz, const double *q, int nt, const int *targets, double *pot,
                             double *fld, cudaStream_t s) {
  if (nt <= 0) return BBFMM_OK;
  direct_kernel<true><<<dim3((nt + ds::TARGETS - 1) / ds::TARGETS, ds::CTAS), 32 * ds::WARPS, 0, s>>>(N, xyz, q, nt, targets,
                                                                                                    pot, fld);
  return bbfmm_set_cuda_error(cudaGetLastError(), "direct_field", __FILE__, __LINE__);
}

}  // namespace bbfmm
