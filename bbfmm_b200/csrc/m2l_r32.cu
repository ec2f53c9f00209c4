// M2L and U-projections for r = 32 (n = 4) on the FP64 tensor path (mma.sync m8n8k4 f64), FP64 or
// FP32 expansions, sums in FP64.
//
// One product is 32 x 32: a warp that holds all 32 outputs of its targets uses every multipole it
// loads for four output fragments at once, so the multipoles need no shared memory. A warp owns 16
// targets (two 2 x 2 x 2 blocks of one sibling class) and loads the sources of the next offset into
// registers while the current one is contracted: lane u of a target's four lanes takes the 8
// consecutive components 8u .. 8u + 7 (wide loads), k-slot u of step ks standing for component
// 8u + ks. The operators are packed once in that fragment order (8 KB an offset, pack32); the CTA's
// eight warps share them through a three-stage cp.async ring.
// Bound by the FP64 tensor rate: 8 KB of operators and 32 KB of multipoles per 128 x 32 x 32
// products. The CUDA-core kernel it replaces was bound by its shared-memory loads (8 per 16 FMAs
// and thread): M2L of 1,048,576 particles, FP32, depth 6 13.2 -> 3.8 ms (0.8 of the rate); 32,768
// particles, FP64, depth 4 0.57 -> 0.16 ms.
#include "solver.cuh"

namespace bbfmm {

namespace r32 {

constexpr int R = 32, WARPS = 8, THREADS = WARPS * 32, BLOCKS = 2 * WARPS, STAGES = 3;
constexpr int B_DOUBLES = R * R;  // [ks 8][fragment 4][lane 32]

__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

template <typename T> struct Eight;  // 8 consecutive components
template <> struct Eight<double> { double2 v[4]; };
template <> struct Eight<float> { float4 v[2]; };
__device__ __forceinline__ void load8(Eight<double> &e, const double *p, bool ok) {
  const double2 *s = reinterpret_cast<const double2 *>(p);
#pragma unroll
  for (int i = 0; i < 4; ++i) e.v[i] = ok ? s[i] : make_double2(0.0, 0.0);
}
__device__ __forceinline__ void load8(Eight<float> &e, const float *p, bool ok) {
  const float4 *s = reinterpret_cast<const float4 *>(p);
#pragma unroll
  for (int i = 0; i < 2; ++i) e.v[i] = ok ? s[i] : make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ double get8(const Eight<double> &e, int k) { return k & 1 ? e.v[k >> 1].y : e.v[k >> 1].x; }
__device__ __forceinline__ double get8(const Eight<float> &e, int k) {
  const float4 q = e.v[k >> 2];
  return (double)((k & 3) == 0 ? q.x : (k & 3) == 1 ? q.y : (k & 3) == 2 ? q.z : q.w);
}

// Grid: x = 8 classes x tiles of 16 blocks (class fastest: the resident CTAs share one source
// region), y = groups of the 189 offsets, each with its own slice of Lout (TO: double with several
// groups, whatever T is, else T).
template <typename T, typename TO>
__global__ void __launch_bounds__(THREADS, 2)
    m2l_r32_kernel(const T *__restrict__ M, const double *__restrict__ Bpack, TO *__restrict__ Lout, int level,
                   const int4 *__restrict__ offs, const int4 *__restrict__ boxes, int nblocks, int nsets) {
  __shared__ __align__(16) double Bs[STAGES][B_DOUBLES];
  const int P = 1 << (level - 1), P3 = P * P * P;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c = blockIdx.x % 8, tile = blockIdx.x / 8;
  const int cb[3] = {(c >> 2) & 1, (c >> 1) & 1, c & 1};
  // block b: listed, or the b-th 2 x 2 x 2 block of the stacked class grids, 4 x 4 x 4 boxes of
  // eight blocks one after the other
  int x0[2], y0[2], z0[2], sb[2];
  bool live[2];
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const int b = tile * BLOCKS + warp * 2 + m;
    live[m] = b < nblocks;
    int4 o = make_int4(0, 0, 0, 0);
    if (live[m]) {
      if (boxes) {
        o = boxes[b];
      } else if (P == 2) {
        o.x = b;
      } else {
        const int nb = P / 4, per = nb * nb * nb, box = b >> 3, w = box % per;
        o = make_int4(box / per, (w % nb) * 4 + 2 * (b & 1), ((w / nb) % nb) * 4 + (b & 2),
                      (w / (nb * nb)) * 4 + ((b & 4) >> 1));
      }
    }
    const int row = lane >> 2;
    x0[m] = o.y + (row & 1);
    y0[m] = o.z + ((row >> 1) & 1);
    z0[m] = o.w + (row >> 2);
    sb[m] = o.x * 8 * P3;
  }
  const int o0 = (189 * blockIdx.y) / gridDim.y, o1 = (189 * (blockIdx.y + 1)) / gridDim.y;
  Lout += (int64_t)blockIdx.y * 8 * nsets * P3 * R;

  auto load_b = [&](int o) {
    if (o < o1) {
      const double *src = Bpack + (int64_t)__ldg(&offs[c * 189 + o].x) * B_DOUBLES;
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(Bs[(o - o0) % STAGES]);
#pragma unroll
      for (int i = 0; i < B_DOUBLES / 2 / THREADS; ++i) {
        const int e = tid + THREADS * i;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * e), "l"(src + 2 * e) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto fetch = [&](int o, Eight<T> *a) {
    const int4 ov = __ldg(offs + c * 189 + o);
    const int gx = cb[0] + ov.y, gy = cb[1] + ov.z, gz = cb[2] + ov.w;
    const int sx = gx & 1, sy = gy & 1, sz = gz & 1;
    const int hx = (gx - sx) / 2, hy = (gy - sy) / 2, hz = (gz - sz) / 2;
    const int sc = ((sx << 2) | (sy << 1) | sz) * P3;
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int px = x0[m] + hx, py = y0[m] + hy, pz = z0[m] + hz;
      const bool ok = live[m] && (unsigned)px < (unsigned)P && (unsigned)py < (unsigned)P && (unsigned)pz < (unsigned)P;
      load8(a[m], M + (ok ? (int64_t)(sb[m] + sc + (pz * P + py) * P + px) * R + 8 * (lane & 3) : 0), ok);
    }
  };
  double acc[2][4][2];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int f = 0; f < 4; ++f) acc[m][f][0] = acc[m][f][1] = 0.0;
  Eight<T> nxt[2];
  fetch(o0, nxt);
  load_b(o0);
  load_b(o0 + 1);
  for (int o = o0; o < o1; ++o) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();  // stage o has landed, and every warp is done with stage o - 1
    load_b(o + 2);
    Eight<T> cur[2] = {nxt[0], nxt[1]};
    if (o + 1 < o1) fetch(o + 1, nxt);
    if (live[0]) {  // the same for the whole warp; block 1 of a live block 0 may hold zeros
      const double *B = Bs[(o - o0) % STAGES] + lane;
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        const double a0 = get8(cur[0], ks), a1 = get8(cur[1], ks);
#pragma unroll
        for (int f = 0; f < 4; ++f) {
          const double b = B[(ks * 4 + f) * 32];
          dmma(acc[0][f][0], acc[0][f][1], a0, b);
          dmma(acc[1][f][0], acc[1][f][1], a1, b);
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    if (!live[m]) continue;
    TO *dst = Lout + (int64_t)(sb[m] + c * P3 + (z0[m] * P + y0[m]) * P + x0[m]) * R + 2 * (lane & 3);
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      dst[8 * f] = (TO)acc[m][f][0];
      dst[8 * f + 1] = (TO)acc[m][f][1];
    }
  }
}

// Bpack[k][ks][f][lane] = E_k(i, j), i = 8 f + (lane >> 2), j = 8 (lane & 3) + ks; E_k(i, j) at
// i + j R of the column-major blocks.
template <typename T>
__global__ void pack32_kernel(const T *__restrict__ Ecol, double *__restrict__ Bpack) {
  const int64_t b = (int64_t)blockIdx.x * B_DOUBLES;
  for (int e = threadIdx.x; e < B_DOUBLES; e += blockDim.x) {
    const int lane = e & 31, f = (e >> 5) & 3, ks = e >> 7;
    Bpack[b + e] = (double)Ecol[b + 8 * f + (lane >> 2) + (8 * (lane & 3) + ks) * R];
  }
}

// ---------------------------------------------------------------- projections
// C[out(m)][n] = scale cs[n] sum_k A[in(m)][k] B(k, n) for m < rows, rows remapped between Morton and
// class-major order: up K = 64, N = 32 (S rows -> M, B = Kweights o U), down K = 32, N = 64 (L rows -> F,
// B = U^T, cs = Kweights). Replaces the 128-row tiles of the general GEMM, which left a level of 64 or
// 512 rows to one or four CTAs walking K in shared-memory steps. A warp takes 16 rows whole: lane u
// of a row's four lanes loads the K / 4 components from K u / 4 on (k-slot u of step ks is component
// K u / 4 + ks) and every product of the row follows from registers; the operator (16 KB in fragment
// order) comes from L1 / L2.
template <typename T, int K, int N, bool OUT_CPG>
__global__ void __launch_bounds__(64) proj32_kernel(int64_t rows, const T *__restrict__ A, const double *__restrict__ Bfrag,
                                                    const T *__restrict__ cs, T scale, T *__restrict__ C, int level,
                                                    int64_t row0, const int64_t *__restrict__ rowlist) {
  constexpr int PER = K / 4, NF = N / 8;
  const int lane = threadIdx.x & 31, u = lane & 3, tr = lane >> 2;
  const int64_t m0 = ((int64_t)blockIdx.x * 2 + (threadIdx.x >> 5)) * 16;
  if (m0 >= rows) return;
  Eight<T> a[2][PER / 8];
  int64_t out[2];
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const int64_t t = m0 + 8 * m + tr;
    const bool ok = t < rows;
    const int64_t cpg = ok ? morton_to_cpg_row(pass_cell(rowlist, row0, t), level) : 0;
    out[m] = ok ? (OUT_CPG ? cpg : t) : -1;
    const T *src = A + (OUT_CPG ? (ok ? t : 0) : cpg) * K + PER * u;
#pragma unroll
    for (int i = 0; i < PER / 8; ++i) load8(a[m][i], src + 8 * i, ok);
  }
  double acc[2][NF][2];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int f = 0; f < NF; ++f) acc[m][f][0] = acc[m][f][1] = 0.0;
#pragma unroll
  for (int ks = 0; ks < PER; ++ks) {
    const double a0 = get8(a[0][ks / 8], ks % 8), a1 = get8(a[1][ks / 8], ks % 8);
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      const double b = __ldg(Bfrag + (ks * NF + f) * 32 + lane);
      dmma(acc[0][f][0], acc[0][f][1], a0, b);
      dmma(acc[1][f][0], acc[1][f][1], a1, b);
    }
  }
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    if (out[m] < 0) continue;
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      const int n = 8 * f + 2 * u;
      const double s0 = cs ? (double)(scale * cs[n]) : (double)scale, s1 = cs ? (double)(scale * cs[n + 1]) : (double)scale;
      T *dst = C + out[m] * N + n;
      dst[0] = (T)(s0 * acc[m][f][0]);
      dst[1] = (T)(s1 * acc[m][f][1]);
    }
  }
}

// Bfrag[ks][f][lane] = B(K / 4 (lane & 3) + ks, 8 f + (lane >> 2)) of a row-major K x N operator.
template <typename T>
__global__ void pack_proj32_kernel(int K, int N, const T *__restrict__ B, double *__restrict__ Bfrag) {
  const int NF = N / 8;
  for (int e = threadIdx.x; e < K * N; e += blockDim.x) {
    const int lane = e & 31, f = (e >> 5) % NF, ks = (e >> 5) / NF;
    Bfrag[e] = (double)B[(K / 4 * (lane & 3) + ks) * N + 8 * f + (lane >> 2)];
  }
}

}  // namespace r32

// Fragment-order copies of Bup (64 x 32) and Bdn (32 x 64), back to back.
template <typename T>
int r32_pack_proj(const T *Bup, const T *Bdn, double *frag, cudaStream_t s) {
  r32::pack_proj32_kernel<T><<<1, 256, 0, s>>>(64, 32, Bup, frag);
  r32::pack_proj32_kernel<T><<<1, 256, 0, s>>>(32, 64, Bdn, frag + 64 * 32);
  return bbfmm_set_cuda_error(cudaGetLastError(), "r32_pack_proj", __FILE__, __LINE__);
}

template <typename T>
int launch_proj_r32(bool up, int64_t rows, const T *A, const double *frag, const T *cs, T scale, T *C, int level, int64_t row0,
                    const int64_t *rowlist, cudaStream_t s) {
  if (rows <= 0) return BBFMM_OK;
  const unsigned grid = (unsigned)((rows + 31) / 32);
  if (up) r32::proj32_kernel<T, 64, 32, true><<<grid, 64, 0, s>>>(rows, A, frag, cs, scale, C, level, row0, rowlist);
  else r32::proj32_kernel<T, 32, 64, false><<<grid, 64, 0, s>>>(rows, A, frag + 64 * 32, cs, scale, C, level, row0, rowlist);
  return bbfmm_set_cuda_error(cudaGetLastError(), "proj_r32", __FILE__, __LINE__);
}

size_t r32_pack_doubles() { return (size_t)BBFMM_NUM_OFFSETS * r32::B_DOUBLES; }

template <typename T>
int r32_pack(const T *Ecol, double *Bpack, cudaStream_t s) {
  r32::pack32_kernel<T><<<BBFMM_NUM_OFFSETS, 256, 0, s>>>(Ecol, Bpack);
  return bbfmm_set_cuda_error(cudaGetLastError(), "r32_pack", __FILE__, __LINE__);
}

static int64_t r32_blocks(int level, int nsets) { return (int64_t)nsets * pow8i(level - 2); }

// Offset groups per target tile: the two CTAs that an SM holds filled with the fewest partial sums
// (each group writes and reads the level once more: about 3 of the 189 offsets' time).
int r32_default_groups(int level, int nsets) {
  const int64_t tiles = 8 * ((r32_blocks(level, nsets) + r32::BLOCKS - 1) / r32::BLOCKS);
  int best = 1;
  double cost = 1e300;
  for (int g = 1; g <= DMMA_PARTS; ++g) {
    const double c = (double)((tiles * g + 295) / 296) * (double)((189 + g - 1) / g + 3);
    if (c < cost * 0.98) {
      cost = c;
      best = g;
    }
  }
  return best;
}

// Writes Lout for every cell of the level (assign), or with a list of 2 x 2 x 2 blocks of parent
// cells (set, x0, y0, z0) for their cells only, in one group.
template <typename T>
int launch_m2l_r32(const double *Bpack, const T *M, T *Lout, int level, const int4 *offs, double *part, int64_t part_elems,
                   cudaStream_t s, int nsets, int ngroups, const int4 *boxes, int nboxes) {
  const int64_t all = r32_blocks(level, nsets), count = all * 64 * r32::R;
  if (boxes && (nboxes < 0 || nboxes > all)) return bbfmm_set_error(BBFMM_ERR_ARG, "box list longer than the level");
  if (boxes && nboxes == 0) return BBFMM_OK;
  int ng = ngroups > 0 ? ngroups : r32_default_groups(level, nsets);
  if (ng > DMMA_PARTS) ng = DMMA_PARTS;
  if (!part || boxes) ng = 1;
  else if (ng > 1 && (int64_t)ng * count > part_elems) ng = (int)(part_elems / count);
  if (ng < 1) ng = 1;
  const int64_t nb = boxes ? nboxes : all;
  const int64_t tiles = 8 * ((nb + r32::BLOCKS - 1) / r32::BLOCKS);
  const dim3 grid((unsigned)tiles, ng);
  if (ng > 1)
    r32::m2l_r32_kernel<T, double><<<grid, r32::THREADS, 0, s>>>(M, Bpack, part, level, offs, boxes, (int)nb, nsets);
  else
    r32::m2l_r32_kernel<T, T><<<grid, r32::THREADS, 0, s>>>(M, Bpack, Lout, level, offs, boxes, (int)nb, nsets);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || ng == 1) return bbfmm_set_cuda_error(e, "m2l_r32", __FILE__, __LINE__);
  return launch_sum_parts<T>(count, ng, part, Lout, s);
}

#define R32_INST(T)                                                                                                  \
  template int r32_pack<T>(const T *, double *, cudaStream_t);                                                       \
  template int r32_pack_proj<T>(const T *, const T *, double *, cudaStream_t);                                       \
  template int launch_proj_r32<T>(bool, int64_t, const T *, const double *, const T *, T, T *, int, int64_t,         \
                                  const int64_t *, cudaStream_t);                                                    \
  template int launch_m2l_r32<T>(const double *, const T *, T *, int, const int4 *, double *, int64_t, cudaStream_t, int, int, \
                                 const int4 *, int);
R32_INST(double)
R32_INST(float)

}  // namespace bbfmm
