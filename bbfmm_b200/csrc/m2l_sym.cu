// M2L folded over the mirror images of an offset (r = 256, FP64 arithmetic on the FP64 tensor
// path; FP64 or FP32 multipoles).
//
// The kernel matrices of two offsets that are mirror images in a coordinate plane differ by the
// reflection of the Chebyshev nodes. When the span of the basis U is invariant under the three
// reflections (it is, unless the rank cuts through a set of equal singular values), U can be
// rotated (sym_prepare) so that every component has a parity in x, y and z: eight classes p of
// about r / 8 components. In that basis E_{s v} = S_s E_v S_s, S_s = diag(+-1 by the parities in
// the axes that s flips), so with a = |v|
//   L_p = sum_a sum_q E_a(p, q) Y_{p^q},   Y_u(j) = sum_s chi_s(u) M_{s a}(j)   (j in class q)
// where s runs over the sign choices of the axes that occur (both signs of 1 and 2, one of 3)
// and chi_s(u) = -1 per flipped axis in which u is odd. The eight sources of an orbit give the
// eight Y_u by additions alone (three butterflies), and one product with E_a replaces eight. In
// an axis where a = 0, E_a(p, q) vanishes unless p and q agree there, which halves the work again.
// The 189 products r x r per target become 39.5.
//
// Tile: 64 targets of one sibling class (eight 2 x 2 x 2 blocks: a 4 x 4 x 4 box, listed blocks, or
// eight stacked sets at level 2) x all outputs. A step is (orbit a, classes q_nz of the nonzero
// axes, 12 components): eight A tiles of 64 x 12 -- Y_u for every u of the nonzero axes and every
// class of the zero ones -- of which the outputs of class p take tile p ^ q_nz. Twelve warps: each
// thread forms two elements of the A tiles, loading the sources' components one step ahead into
// registers, and each warp owns three 8-column output fragments for all 64 targets. The A rows of
// 12 doubles and the B fragments (the operators in step order, 27 KB a step, by cp.async) are both
// read without bank conflicts, and double-buffered with one barrier a step.
//
// Bound by the FP64 tensor path (37 TFLOP/s measured) and the latency of a step with three warps per
// scheduler: the path is busy 50% of the time at level 5 (512 tiles, two groups, 10.9 ms). Offsets and
// validity come from small shared tables, because finding eight sources by integer arithmetic was the
// larger part of a step's instructions. M2L of 262,144 particles, depth 5: unfolded FP64 57.6 ms, folded
// 16.1 ms, with the tables 12.8 ms. Warps that multiply first and form tiles afterwards (13.8 ms) and
// twice the warps with half the targets each (15.8 ms) were slower.
#include <cmath>
#include <limits>
#include <vector>

#include "solver.cuh"

namespace bbfmm {

namespace sy {

constexpr int R = 256, BK = 12, KS = BK / 4, NCH = 3;  // 36 components of a class at most
constexpr int NF = 36, WARPS = 12, THREADS = WARPS * 32, FW = NF / WARPS;
constexpr int NT = 64, A_DOUBLES = 8 * NT * BK, B_DOUBLES = KS * NF * 32;
constexpr int SMEM_BYTES = 2 * (A_DOUBLES + B_DOUBLES) * 8;

constexpr int NORB = 56;  // orbits: |v| in [0, 3]^3 outside [0, 1]^3

// One step: word = ax | ay << 2 | az << 4 (the orbit |v|) | q_nz << 6 | chunk << 9 | orbit index << 16;
// per source i of the orbit (bit pattern of i: the sign, or the class bit in an axis where a = 0)
// the first component and the class as a bit.
struct __align__(16) Step {
  unsigned short comp[8];
  unsigned char cbit[8];
  int word, pad;
};
static_assert(sizeof(Step) == 32, "a step is two 16-byte loads");

struct Classes {
  int cstart[9];             // components of class p: [cstart[p], cstart[p + 1])
  unsigned char fcls[NF];    // output fragment f: its class (NF fragments, unused ones past the end
  unsigned char fcol[NF];    // have fcol = 255) and first column within the class
};

// D (8 x 8) += A (8 x 4) B (4 x 8): A row lane >> 2, column lane & 3; B row lane & 3, column
// lane >> 2; D row lane >> 2, columns 2 (lane & 3) + {0, 1}.
__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// TO: double where several step groups write their sums to slices, whatever T is, else T.
template <typename T, typename TO>
__global__ void __launch_bounds__(THREADS, 1)
    m2l_sym_kernel(const T *__restrict__ M, const double *__restrict__ Bsteps, const Step *__restrict__ steps, int nsteps,
                   const int *__restrict__ orbits, TO *__restrict__ Lout, int level, const __grid_constant__ Classes cl,
                   const int4 *__restrict__ boxes, int nboxes, int nsets) {
  extern __shared__ __align__(16) double smem[];
  double *const Bs = smem + 2 * A_DOUBLES;  // A tiles of two steps, then B tiles of two
  __shared__ int4 s_org[8];  // block k of the tile: (set, or -1 - set when not written; x0, y0, z0)
  // source i of an orbit, for targets of this class: its cell's distance from the target's class-0
  // cell, and the bits that a target's mask must have for the source to exist (shift -1, 0, 1 in x,
  // y, z: bits 0-8; bit 31: no such source)
  __shared__ __align__(16) int s_off[NORB][8], s_sel[NORB][8];
  __shared__ int s_nk[NCH][8];  // k-steps of chunk kk that hold components of class q
  const int P = 1 << (level - 1), P3 = P * P * P;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cls = blockIdx.x % 8;  // sibling class fastest: the resident CTAs share one source region
  const int tile = blockIdx.x / 8;
  if (tid < 8) {
    int4 b;
    if (boxes) {
      const int bi = tile * 8 + tid;
      b = boxes[bi < nboxes ? bi : nboxes - 1];
      if (bi >= nboxes) b.x = -1 - b.x;
    } else if (P == 2) {  // the whole class grid of eight stacked sets
      const int set = tile * 8 + tid;
      b = make_int4(set < nsets ? set : -nsets, 0, 0, 0);  // -nsets = -1 - (nsets - 1)
    } else {
      const int nb = P / 4, per = nb * nb * nb, tb = tile % per;
      b = make_int4(tile / per, (tb % nb) * 4 + 2 * (tid & 1), ((tb / nb) % nb) * 4 + (tid & 2),
                    (tb / (nb * nb)) * 4 + 2 * (tid >> 2));
    }
    s_org[tid] = b;
  }
  const int bit[3] = {(cls >> 2) & 1, (cls >> 1) & 1, cls & 1};
  for (int e = tid; e < NORB * 8; e += THREADS) {
    const int w = orbits[e >> 3];
    int off = 0, sel = 0;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      const int a = (w >> (2 * x)) & 3, s = (e >> (2 - x)) & 1;
      // a = 3: the one sign that occurs, -3 for odd cells; a = 0: the bit picks the class instead
      const bool neg = a == 3 ? bit[x] != 0 : s != 0;
      const int g = bit[x] + (neg ? -a : a), sh = (g - (g & 1)) / 2;
      off += (g & 1) * (4 >> x) * P3 + sh * (x == 0 ? 1 : (x == 1 ? P : P * P));
      sel |= a == 3 && s ? (int)0x80000000 : 1 << (3 * x + sh + 1);
    }
    s_off[e >> 3][e & 7] = off;
    s_sel[e >> 3][e & 7] = sel;
  }
  if (tid < NCH * 8) {
    const int left = cl.cstart[(tid & 7) + 1] - cl.cstart[tid & 7] - (tid >> 3) * BK;
    s_nk[tid >> 3][tid & 7] = left <= 0 ? 0 : (left >= BK ? KS : (left + 3) / 4);
  }
  __syncthreads();
  const int og = blockIdx.y, ng = gridDim.y;
  const int s0 = (int)((int64_t)nsteps * og / ng), s1 = (int)((int64_t)nsteps * (og + 1) / ng);
  Lout += (int64_t)og * 8 * nsets * P3 * R;

  // the two elements of the A tiles this thread forms: component tid % 12 of targets tid / 12 and
  // 32 + tid / 12 (a warp's loads are runs of 12 consecutive components); target t is cell t & 7 of
  // block t >> 3
  const int jt = tid % BK;
  const T *const Mj = M + jt;
  int tb0[2], vm[2];  // class-0 row of the target's cell (levels hold at most 2^30 cells); its mask
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int t = 32 * e + tid / BK;
    const int4 o = s_org[t >> 3];
    const int c[3] = {o.y + (t & 1), o.z + ((t >> 1) & 1), o.w + ((t >> 2) & 1)};
    tb0[e] = (o.x >= 0 ? o.x : -1 - o.x) * 8 * P3 + (c[2] * P + c[1]) * P + c[0];
    vm[e] = 0;
#pragma unroll
    for (int x = 0; x < 3; ++x)
#pragma unroll
      for (int sh = -1; sh <= 1; ++sh)
        if ((unsigned)(c[x] + sh) < (unsigned)P) vm[e] |= 1 << (3 * x + sh + 1);
  }
  int cm = 0;  // bit 8 kk + q: component jt of chunk kk exists in class q
#pragma unroll
  for (int kk = 0; kk < NCH; ++kk)
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (jt + kk * BK < cl.cstart[q + 1] - cl.cstart[q]) cm |= 1 << (8 * kk + q);

  T raw[2][8];
  auto fetch = [&](int st) {
    const uint4 rc = __ldg(reinterpret_cast<const uint4 *>(steps + st));
    const uint4 rb = __ldg(reinterpret_cast<const uint4 *>(steps + st) + 1);
    const int w = (int)rb.z, orb = w >> 16, kk = (w >> 9) & 3;
    const int4 o0 = *reinterpret_cast<const int4 *>(&s_off[orb][0]), o1 = *reinterpret_cast<const int4 *>(&s_off[orb][4]);
    const int4 l0 = *reinterpret_cast<const int4 *>(&s_sel[orb][0]), l1 = *reinterpret_cast<const int4 *>(&s_sel[orb][4]);
    const int off[8] = {o0.x, o0.y, o0.z, o0.w, o1.x, o1.y, o1.z, o1.w};
    const int sel[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
    const unsigned cp[4] = {rc.x, rc.y, rc.z, rc.w}, cb[2] = {rb.x, rb.y};
    const int cmk = ((cm >> (8 * kk)) & 255) << 9;
    const int m[2] = {vm[0] | cmk, vm[1] | cmk};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int need = sel[i] | (int)((cb[i >> 2] >> (8 * (i & 3))) & 255u) << 9;
      const int comp = (int)((cp[i >> 1] >> (16 * (i & 1))) & 0xffffu);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const bool ok = (m[e] & need) == need;
        raw[e][i] = ok ? Mj[(int64_t)(tb0[e] + off[i]) * R + comp] : (T)0;
      }
    }
  };
  // raw of step st -> its eight A tiles
  auto form = [&](int st, double *A) {
    const int w = __ldg(&steps[st].word);
    double v[2][8];
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int i = 0; i < 8; ++i) v[e][i] = (double)raw[e][i];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      const int m = 4 >> x, a = (w >> (2 * x)) & 3;
      if (a == 1 || a == 2) {  // both signs: sum and difference
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (!(i & m)) {
              const double p = v[e][i], n = v[e][i | m];
              v[e][i] = p + n;
              v[e][i | m] = p - n;
            }
      } else if (a == 3) {  // one sign: the same value, negated for odd outputs where the sign is -
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (!(i & m)) v[e][i | m] = bit[x] ? -v[e][i] : v[e][i];
      }
    }
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int i = 0; i < 8; ++i) A[(i * NT + 32 * e) * BK + tid] = v[e][i];
  };
  auto load_b = [&](int st, double *B) {
    const double *src = Bsteps + (int64_t)st * B_DOUBLES;
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(B);
    for (int i = tid; i < B_DOUBLES / 2; i += THREADS)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * i), "l"(src + 2 * i) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  // this warp's output fragments: the class of each (fragments of one class are adjacent)
  int fc[FW];
#pragma unroll
  for (int f = 0; f < FW; ++f) fc[f] = cl.fcls[warp * FW + f];
  const bool same1 = fc[1] == fc[0], same2 = fc[2] == fc[1];
  double acc[8][FW][2];
#pragma unroll
  for (int m = 0; m < 8; ++m)
#pragma unroll
    for (int f = 0; f < FW; ++f) acc[m][f][0] = acc[m][f][1] = 0.0;

  if (s0 < s1) {
    fetch(s0);
    load_b(s0, Bs);
    form(s0, smem);
    if (s0 + 1 < s1) fetch(s0 + 1);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
  }
  for (int st = s0; st < s1; ++st) {
    const int buf = (st - s0) & 1;
    if (st + 1 < s1) load_b(st + 1, Bs + (buf ^ 1) * B_DOUBLES);
    const int w = __ldg(&steps[st].word);
    const int qnz = (w >> 6) & 7, kk = (w >> 9) & 3;
    const int zm = ((w & 3) == 0 ? 4 : 0) | ((w & 12) == 0 ? 2 : 0) | ((w & 48) == 0 ? 1 : 0);
    const int A0 = buf * A_DOUBLES + (lane >> 2) * BK + (lane & 3);
    const int B0 = 2 * A_DOUBLES + buf * B_DOUBLES + (warp * FW) * 32 + lane;
    int nk = 0;  // k-steps of each fragment, four bits each
#pragma unroll
    for (int f = 0; f < FW; ++f) nk |= s_nk[kk][(fc[f] & zm) | qnz] << (4 * f);
    if (st + 1 < s1) {
      form(st + 1, smem + (buf ^ 1) * A_DOUBLES);
      if (st + 2 < s1) fetch(st + 2);
    }
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      double af[8];
#pragma unroll
      for (int f = 0; f < FW; ++f) {
        if (f == 0 || (f == 1 ? !same1 : !same2)) {
#pragma unroll
          for (int m = 0; m < 8; ++m) af[m] = smem[A0 + (fc[f] ^ qnz) * NT * BK + 4 * ks + m * 8 * BK];
        }
        if (ks < ((nk >> (4 * f)) & 15)) {
          const double bf = smem[B0 + (ks * NF + f) * 32];
#pragma unroll
          for (int m = 0; m < 8; ++m) dmma(acc[m][f][0], acc[m][f][1], af[m], bf);
        }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
  }
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    const int4 o = s_org[m];
    if (o.x < 0) continue;
    const int row = lane >> 2;
    const int64_t cell = (int64_t)(o.x * 8 + cls) * P3 +
                         ((int64_t)(o.w + (row >> 2)) * P + o.z + ((row >> 1) & 1)) * P + o.y + (row & 1);
#pragma unroll
    for (int f = 0; f < FW; ++f) {
      const int c0 = cl.cstart[fc[f]], n = cl.cstart[fc[f] + 1] - c0;
      const int col = cl.fcol[warp * FW + f] + 2 * (lane & 3);
      TO *dst = Lout + cell * R + c0 + col;
      if (col < n) dst[0] = (TO)acc[m][f][0];
      if (col + 1 < n) dst[1] = (TO)acc[m][f][1];
    }
  }
}

// Lout[e] = sum_g part[g][e], in a fixed order, for the 64 cells (8 classes x 2 x 2 x 2) of each listed block of parent cells.
template <typename T>
__global__ void __launch_bounds__(256) sym_sum_boxes_kernel(int64_t count, int ng, int P, const int4 *__restrict__ boxes,
                                                            const double *__restrict__ part, T *__restrict__ Lout) {
  const int4 b = boxes[blockIdx.x];
  const int64_t P3 = (int64_t)P * P * P;
  for (int e = threadIdx.x; e < 64 * R; e += blockDim.x) {
    const int t = e / R;
    const int64_t cell = (int64_t)(b.x * 8 + (t >> 3)) * P3 +
                         ((int64_t)(b.w + ((t >> 2) & 1)) * P + b.z + ((t >> 1) & 1)) * P + b.y + (t & 1);
    const int64_t at = cell * R + e % R;
    double v = 0.0;
    for (int g = 0; g < ng; ++g) v += part[(int64_t)g * count + at];
    Lout[at] = (T)v;
  }
}

// ---------------------------------------------------------------- set-up
// C(m, n) = sum_k A(m, k) B(k, n) for a batch (blockIdx.z), element (i, j) of a matrix at
// i * rs + j * cs; sums in FP64. 64 x 64 tiles, 4 x 4 values per thread; dimensions multiples of 64.
// alist (optional): matrix alist[z] of A for product z.
template <typename TA, typename TB, typename TC>
__global__ void __launch_bounds__(256) gemm_kernel(int K, const TA *__restrict__ A, int64_t ars, int64_t acs, int64_t ab,
                                                   const TB *__restrict__ B, int64_t brs, int64_t bcs, int64_t bb,
                                                   TC *__restrict__ C, int64_t crs, int64_t ccs, int64_t cb,
                                                   const int *__restrict__ alist = nullptr) {
  __shared__ double sa[16][65], sb[16][65];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.x * 64, n0 = blockIdx.y * 64;
  A += (alist ? alist[blockIdx.z] : (int)blockIdx.z) * ab;
  B += blockIdx.z * bb;
  C += blockIdx.z * cb;
  double acc[4][4] = {};
  for (int k0 = 0; k0 < K; k0 += 16) {
    __syncthreads();
    for (int e = tid; e < 16 * 64; e += 256) {
      const int ka = acs == 1 ? e & 15 : e >> 6, ma = acs == 1 ? e >> 4 : e & 63;
      sa[ka][ma] = (double)A[(m0 + ma) * ars + (k0 + ka) * acs];
      const int kb = brs == 1 ? e & 15 : e >> 6, nb = brs == 1 ? e >> 4 : e & 63;
      sb[kb][nb] = (double)B[(k0 + kb) * brs + (n0 + nb) * bcs];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      double a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[i] = sa[k][ty + 16 * i];
        b[i] = sb[k][tx + 16 * i];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += a[i] * b[j];
    }
  }
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 4; ++j) C[(m0 + ty + 16 * i) * crs + (n0 + tx + 16 * j) * ccs] = (TC)acc[i][j];
}

__device__ __forceinline__ int class_of(const Classes &cl, int i) {
  int p = 0;
  while (i >= cl.cstart[p + 1]) ++p;
  return p;
}

// One thread per component pair e = i r + j. Eavg[o] (row-major) = mean over the eight sign choices s
// of S_s E'_{s a} S_s for each orbit o (words ax | ay << 2 | az << 4), E' row-major, the matrix of an
// offset at slot[its cell of the 7 x 7 x 7 grid]; off[e] = the pair's largest distance of an image from
// the mean (NaN is kept), mx the largest |E'|, over the orbits of every launch.
__global__ void __launch_bounds__(256) average_kernel(const double *__restrict__ Ep, const int *__restrict__ slot,
                                                      const int *__restrict__ orbits, int norb, Classes cl,
                                                      double *__restrict__ Eavg, double *__restrict__ off, double *mx) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const int u = class_of(cl, e / R) ^ class_of(cl, e % R);
  double most = 0.0, far = off[e];
  for (int o = 0; o < norb; ++o) {
    const int w = orbits[o], a[3] = {w & 3, (w >> 2) & 3, (w >> 4) & 3};
    double v[8], sum = 0.0;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const int x = s & 4 ? -a[0] : a[0], y = s & 2 ? -a[1] : a[1], z = s & 1 ? -a[2] : a[2];
      const double t = Ep[(int64_t)slot[49 * (x + 3) + 7 * (y + 3) + z + 3] * R * R + e];
      v[s] = __popc(s & u) & 1 ? -t : t;
      sum += v[s];
      most = fmax(most, fabs(t));
    }
    sum *= 0.125;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const double d = fabs(v[s] - sum);
      if (d > far || d != d) far = d;
    }
    Eavg[(int64_t)o * R * R + e] = sum;
  }
  off[e] = far;
  __shared__ double s_most[256];
  s_most[threadIdx.x] = most;
  __syncthreads();
  for (int h = 128; h > 0; h >>= 1) {
    if (threadIdx.x < h) s_most[threadIdx.x] = fmax(s_most[threadIdx.x], s_most[threadIdx.x + h]);
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicMax((unsigned long long *)mx, (unsigned long long)__double_as_longlong(s_most[0]));
}

// sq[i r + j] = the largest E_k(i, j)^2 of the 316 offsets (E_k(i, j) at i + j r).
template <typename T>
__global__ void __launch_bounds__(256) largest_kernel(const T *__restrict__ Ecol, double *__restrict__ sq) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  double most = 0.0;
  for (int k = 0; k < BBFMM_NUM_OFFSETS; ++k) {
    const double v = (double)Ecol[(int64_t)k * R * R + e];
    most = fmax(most, v * v);
  }
  sq[(e % R) * R + e / R] = most;
}

// out = (Q o Q)^T in, or in (Q o Q): the squares that rotation from the left or the right adds up.
__global__ void __launch_bounds__(256) rotate_squares_kernel(const double *__restrict__ Q, const double *__restrict__ in,
                                                             int left, double *__restrict__ out) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x, i = e / R, j = e % R;
  double sum = 0.0;
  for (int k = 0; k < R; ++k) {
    const double q = left ? Q[k * R + i] : Q[k * R + j];
    sum += q * q * (left ? in[k * R + j] : in[i * R + k]);
  }
  out[e] = sum;
}

// *bad = 1 where a pair's images differ by more than rel of its rotated root-sum-square entry and base
// of the largest of all, or are not finite.
__global__ void __launch_bounds__(256) symmetric_kernel(const double *__restrict__ sq, const double *__restrict__ off,
                                                        const double *__restrict__ mx, double rel, double base, int *bad) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (__syncthreads_or(!(off[e] <= rel * sqrt(sq[e]) + base * *mx)) && threadIdx.x == 0) *bad = 1;
}

// Bsteps[step][ks][f][lane] = E_a(i, j) for component j = 12 chunk + 4 ks + (lane & 3) of class
// q = (p & zero axes) | q_nz and output i = column fcol + (lane >> 2) of the fragment's class p.
__global__ void pack_steps_kernel(const double *__restrict__ Eavg, const Step *__restrict__ steps, Classes cl,
                                  double *__restrict__ Bsteps) {
  const int w = steps[blockIdx.x].word;
  const int qnz = (w >> 6) & 7, kk = (w >> 9) & 3;
  const int zm = ((w & 3) == 0 ? 4 : 0) | ((w & 12) == 0 ? 2 : 0) | ((w & 48) == 0 ? 1 : 0);
  const double *E = Eavg + (int64_t)(w >> 16) * R * R;
  for (int e = threadIdx.x; e < B_DOUBLES; e += blockDim.x) {
    const int lane = e & 31, f = (e >> 5) % NF, ks = (e >> 5) / NF;
    const int p = cl.fcls[f], q = (p & zm) | qnz;
    const int i = cl.cstart[p] + cl.fcol[f] + (lane >> 2), j = cl.cstart[q] + kk * BK + 4 * ks + (lane & 3);
    const bool in = cl.fcol[f] != 255 && i < cl.cstart[p + 1] && j < cl.cstart[q + 1];
    Bsteps[(int64_t)blockIdx.x * B_DOUBLES + e] = in ? E[i * R + j] : 0.0;
  }
}

}  // namespace sy

struct SymOps {
  sy::Classes cl;
  int nsteps = 0;
  double *Q = nullptr;       // r x r row-major: columns are the rotated basis in the given one
  double *Bsteps = nullptr;  // operators in step order
  sy::Step *steps = nullptr;
  int *orbits = nullptr;
};

void sym_free(void *p) {
  SymOps *o = (SymOps *)p;
  if (!o) return;
  for (void *d : {(void *)o->Q, (void *)o->Bsteps, (void *)o->steps, (void *)o->orbits})
    if (d) cudaFree(d);
  delete o;
}

// q minus its parts along the orthonormal cols[from .. to).
static void take_out(std::vector<double> &q, const std::vector<std::vector<double>> &cols, size_t from, size_t to) {
  const int r = (int)q.size();
  for (size_t e = from; e < to; ++e) {
    const std::vector<double> &c = cols[e];
    double t4[4] = {};
    for (int i = 0; i < r; i += 4)
      for (int k4 = 0; k4 < 4; ++k4) t4[k4] += c[i + k4] * q[i + k4];
    const double t = (t4[0] + t4[1]) + (t4[2] + t4[3]);
    if (t != 0.0)
      for (int i = 0; i < r; ++i) q[i] -= t * c[i];
  }
}

// Orthogonal Q (r x r) whose columns have a parity in each axis, class by class in the order of
// the given components (the largest singular values first): for class p the rows of U folded over
// the eight mirror images of a node with the class's signs span the class's part of U, and the
// columns of its Gram matrix, taken in order with a pivot of at least half the largest that
// remains, are orthonormalised. A component of a parity of its own is then a column with one entry,
// and only components of equal singular values mix; the entries that the rounding of U leaves
// elsewhere are cleared (below 32 roundings), because each would carry the largest operator entries
// into the smallest: in FP32 it left 3e-9 of the largest entry in pairs of 1e-10 of it. False when the
// classes do not add up to r (the span of U is not invariant) or a class is larger than the kernel's
// tiles.
template <typename T>
static bool sym_basis(int n, int r, const T *U, std::vector<double> &Q, int *cstart) {
  const int n3 = n * n * n, h = n / 2, hh = h * h * h;
  std::vector<std::vector<double>> cols;
  std::vector<double> V((size_t)hh * r), d(r), q(r);
  for (int p = 0; p < 8; ++p) {
    cstart[p] = (int)cols.size();
    for (int k = 0; k < r; ++k)
      for (int x = 0; x < h; ++x)
        for (int y = 0; y < h; ++y)
          for (int z = 0; z < h; ++z) {
            double v = 0.0;
            for (int s = 0; s < 8; ++s) {
              const int X = s & 4 ? n - 1 - x : x, Y = s & 2 ? n - 1 - y : y, Z = s & 1 ? n - 1 - z : z;
              const double t = (double)U[(size_t)k * n3 + (X * n + Y) * n + Z];
              v += __builtin_popcount(s & p) & 1 ? -t : t;
            }
            V[(size_t)((x * h + y) * h + z) * r + k] = v * 0.35355339059327376220;  // 1 / sqrt(8)
          }
    for (int k = 0; k < r; ++k) {  // the diagonal of the Gram matrix; its columns are formed as they are taken
      d[k] = 0.0;
      for (int a = 0; a < hh; ++a) d[k] += V[(size_t)a * r + k] * V[(size_t)a * r + k];
    }
    for (;;) {
      double m = 0.0;
      for (int k = 0; k < r; ++k) {
        if (!std::isfinite(d[k])) return false;
        m = std::max(m, d[k]);
      }
      if (m < 1e-4) break;
      if (cols.size() == (size_t)r) return false;
      int k = 0;
      while (d[k] < 0.5 * m) ++k;
      std::fill(q.begin(), q.end(), 0.0);
      for (int a = 0; a < hh; ++a) {
        const double *v = V.data() + (size_t)a * r;
        for (int i = 0; i < r; ++i) q[i] += v[k] * v[i];
      }
      // against the class's earlier columns, then against every earlier one (the classes are
      // orthogonal to about 1e-13 as they are; after that to rounding)
      take_out(q, cols, cstart[p], cols.size());
      take_out(q, cols, 0, cols.size());
      double nn = 0.0;
      for (int i = 0; i < r; ++i) nn += q[i] * q[i];
      nn = 1.0 / std::sqrt(nn);
      for (int i = 0; i < r; ++i) q[i] *= nn;
      for (int i = 0; i < r; ++i) d[i] -= q[i] * q[i];
      cols.push_back(q);
    }
    if ((int)cols.size() - cstart[p] > sy::NCH * sy::BK) return false;
  }
  cstart[8] = (int)cols.size();
  if (cstart[8] != r) return false;
  const double none = 16.0 * std::numeric_limits<T>::epsilon();
  for (size_t j = 0; j < cols.size(); ++j) {  // cleared, then orthonormal again
    std::vector<double> &c = cols[j];
    for (int i = 0; i < r; ++i)
      if (std::fabs(c[i]) < none) c[i] = 0.0;
    take_out(c, cols, 0, j);  // once: what was cleared is below 32 roundings
    double nn = 0.0;
    for (int i = 0; i < r; ++i) nn += c[i] * c[i];
    nn = 1.0 / std::sqrt(nn);
    for (int i = 0; i < r; ++i) c[i] *= nn;
  }
  Q.resize((size_t)r * r);
  for (int j = 0; j < r; ++j)
    for (int i = 0; i < r; ++i) Q[(size_t)i * r + j] = cols[j][i];
  return true;
}

// The folded M2L's operators from U (host, column-major n^3 x r) and E (device, [316][r][r]
// column-major), and the projections' U operators in the rotated basis: Bup (n^3 x r) and Bdn
// (r x n^3) from the given ones (all on the device). *out stays null when the operators do not
// have the mirror symmetry: a basis that does not split into parity classes, or a component pair with
// an image further from the mean of its orbit than the rounding of its entries carries there: 8
// roundings of the given operators' entries, each at the largest of its pair and rotated as errors add
// up (root of the sum of squares), and 64 FP64 roundings of the largest entry of all for the arithmetic
// that made them. Measured beyond the first term: 4 of those in FP32 and FP64, 30 in FP64 for a random
// basis of the same span; entries changed by two roundings need 4 of the 8. The entries of the high
// components are 1e-10 of the largest, so that a bound by the largest entry alone would let them differ
// by any factor.
template <typename T>
int sym_prepare(int n, int r, const T *U, const T *Ecol, const T *Bup, const T *Bdn, T *Bup_sym, T *Bdn_sym,
                void **out, cudaStream_t s) {
  *out = nullptr;
  if (r != sy::R) return BBFMM_OK;
  const int n3 = n * n * n;
  std::vector<double> Q;
  SymOps *o = new SymOps();
  sy::Classes &cl = o->cl;
  if (!sym_basis(n, r, U, Q, cl.cstart)) {
    delete o;
    return BBFMM_OK;
  }
  int nf = 0;
  for (int p = 0; p < 8; ++p)
    for (int c = 0; c < cl.cstart[p + 1] - cl.cstart[p]; c += 8, ++nf)
      if (nf < sy::NF) {
        cl.fcls[nf] = (unsigned char)p;
        cl.fcol[nf] = (unsigned char)c;
      }
  if (nf > sy::NF) {
    delete o;
    return BBFMM_OK;
  }
  for (; nf < sy::NF; ++nf) {
    cl.fcls[nf] = 7;
    cl.fcol[nf] = 255;
  }
  std::vector<int> kt(343, -1), orbits;
  std::vector<sy::Step> steps;
  int k = 0;
  for (int c = 0; c < 343; ++c) {
    const int x = c / 49 - 3, y = (c / 7) % 7 - 3, z = c % 7 - 3;
    if (x < -1 || x > 1 || y < -1 || y > 1 || z < -1 || z > 1) kt[c] = k++;
  }
  // the operators are rotated and averaged a few orbits at a time (chunks of at most 32 offsets): slot
  // of each offset in its chunk, the offsets chunk by chunk, and where chunks begin among both
  constexpr int CHUNK = 32;
  std::vector<int> slot(343, 0), list, ofirst{0}, kfirst{0};
  for (int w = 0; w < 64; ++w) {
    const int a[3] = {w & 3, (w >> 2) & 3, (w >> 4) & 3};
    if (a[0] <= 1 && a[1] <= 1 && a[2] <= 1) continue;
    const int nz = (a[0] ? 4 : 0) | (a[1] ? 2 : 0) | (a[2] ? 1 : 0);
    for (int q = 0; q < 8; ++q)
      if ((q & ~nz) == 0)
        for (int c = 0; c < sy::NCH; ++c) {
          sy::Step st{};
          st.word = w | q << 6 | c << 9 | (int)orbits.size() << 16;
          for (int i = 0; i < 8; ++i) {
            const int qi = q | (i & ~nz & 7);
            st.comp[i] = (unsigned short)(cl.cstart[qi] + c * sy::BK);
            st.cbit[i] = (unsigned char)(1 << qi);
          }
          steps.push_back(st);
        }
    if ((int)list.size() - kfirst.back() + (1 << __builtin_popcount(nz)) > CHUNK) {
      ofirst.push_back((int)orbits.size());
      kfirst.push_back((int)list.size());
    }
    for (int s = 0; s < 8; ++s)
      if ((s & ~nz) == 0) {
        const int x = s & 4 ? -a[0] : a[0], y = s & 2 ? -a[1] : a[1], z = s & 1 ? -a[2] : a[2];
        const int c = 49 * (x + 3) + 7 * (y + 3) + z + 3;
        slot[c] = (int)list.size() - kfirst.back();
        list.push_back(kt[c]);
      }
    orbits.push_back(w);
  }
  ofirst.push_back((int)orbits.size());
  kfirst.push_back((int)list.size());
  o->nsteps = (int)steps.size();
  double *tmp = nullptr, *Ep = nullptr, *Eavg = nullptr, *chk = nullptr;  // chk: largest entry, flag, off, squares
  int *listd = nullptr;  // the offsets, then the slots
  auto cleanup = [&](int rc) {
    for (void *p : {(void *)tmp, (void *)Ep, (void *)Eavg, (void *)chk, (void *)listd})
      if (p) cudaFree(p);
    if (rc != BBFMM_OK || !*out) sym_free(o);
    return rc;
  };
  const size_t rr = (size_t)r * r;
#define SYM_OK(x)                                                                                       \
  do {                                                                                                  \
    cudaError_t e__ = (x);                                                                              \
    if (e__ != cudaSuccess) return cleanup(bbfmm_set_cuda_error(e__, #x, __FILE__, __LINE__));          \
  } while (0)
  SYM_OK(cudaMalloc(&tmp, CHUNK * rr * 8));
  SYM_OK(cudaMalloc(&Ep, CHUNK * rr * 8));
  SYM_OK(cudaMalloc(&Eavg, orbits.size() * rr * 8));
  SYM_OK(cudaMalloc(&chk, (2 + 3 * rr) * 8));
  list.insert(list.end(), slot.begin(), slot.end());
  SYM_OK(cudaMalloc(&listd, list.size() * 4));
  SYM_OK(cudaMalloc(&o->Q, rr * 8));
  SYM_OK(cudaMalloc(&o->orbits, orbits.size() * 4));
  SYM_OK(cudaMalloc(&o->steps, steps.size() * sizeof(sy::Step)));
  SYM_OK(cudaMalloc(&o->Bsteps, steps.size() * sy::B_DOUBLES * 8));
  SYM_OK(cudaMemcpyAsync(o->Q, Q.data(), rr * 8, cudaMemcpyHostToDevice, s));
  SYM_OK(cudaMemcpyAsync(listd, list.data(), list.size() * 4, cudaMemcpyHostToDevice, s));
  SYM_OK(cudaMemcpyAsync(o->orbits, orbits.data(), orbits.size() * 4, cudaMemcpyHostToDevice, s));
  SYM_OK(cudaMemcpyAsync(o->steps, steps.data(), steps.size() * sizeof(sy::Step), cudaMemcpyHostToDevice, s));
  SYM_OK(cudaMemsetAsync(chk, 0, (2 + rr) * 8, s));
  const unsigned grr = (unsigned)(rr / 256);
  double *off = chk + 2, *sq = off + rr, *sq2 = sq + rr;
  for (size_t c = 0; c + 1 < ofirst.size(); ++c) {
    const int k0 = kfirst[c], nk = kfirst[c + 1] - k0, o0 = ofirst[c], no = ofirst[c + 1] - o0;
    const dim3 g(r / 64, r / 64, nk);
    // E'_k = Q^T (E_k Q), row-major; E_k(i, j) at i + j r
    sy::gemm_kernel<T, double, double><<<g, 256, 0, s>>>(r, Ecol, 1, r, (int64_t)rr, o->Q, r, 1, 0, tmp, r, 1, (int64_t)rr,
                                                         listd + k0);
    sy::gemm_kernel<double, double, double><<<g, 256, 0, s>>>(r, o->Q, 1, r, 0, tmp, r, 1, (int64_t)rr, Ep, r, 1,
                                                              (int64_t)rr);
    sy::average_kernel<<<grr, 256, 0, s>>>(Ep, listd + BBFMM_NUM_OFFSETS, o->orbits + o0, no, cl, Eavg + o0 * rr, off, chk);
  }
  sy::largest_kernel<T><<<grr, 256, 0, s>>>(Ecol, sq);
  sy::rotate_squares_kernel<<<grr, 256, 0, s>>>(o->Q, sq, 1, sq2);
  sy::rotate_squares_kernel<<<grr, 256, 0, s>>>(o->Q, sq2, 0, sq);
  int bad = 0;
  sy::symmetric_kernel<<<grr, 256, 0, s>>>(sq, off, chk, 4.0 * std::numeric_limits<T>::epsilon(), 64.0 * 0x1p-53,
                                           (int *)(chk + 1));
  SYM_OK(cudaGetLastError());
  SYM_OK(cudaMemcpyAsync(&bad, chk + 1, 4, cudaMemcpyDeviceToHost, s));
  SYM_OK(cudaStreamSynchronize(s));
  if (bad) return cleanup(BBFMM_OK);
  sy::pack_steps_kernel<<<o->nsteps, 256, 0, s>>>(Eavg, o->steps, cl, o->Bsteps);
  sy::gemm_kernel<T, double, T><<<dim3(n3 / 64, r / 64, 1), 256, 0, s>>>(r, Bup, r, 1, 0, o->Q, r, 1, 0, Bup_sym, r, 1, 0);
  sy::gemm_kernel<double, T, T><<<dim3(r / 64, n3 / 64, 1), 256, 0, s>>>(r, o->Q, 1, r, 0, Bdn, n3, 1, 0, Bdn_sym, n3, 1,
                                                                       0);
  SYM_OK(cudaGetLastError());
  SYM_OK(cudaStreamSynchronize(s));
#undef SYM_OK
  *out = o;
  return cleanup(BBFMM_OK);
}

// `cells` rows of r (a multiple of 64) from the rotated basis to the given one, dst[c][i] =
// sum_i' Q(i, i') src[c][i'], or the other way, dst[c][i'] = sum_i Q(i, i') src[c][i].
template <typename T>
int sym_rotate(const void *op, bool to_given, int64_t cells, const T *src, T *dst, cudaStream_t s) {
  const SymOps *o = (const SymOps *)op;
  const int r = sy::R;
  sy::gemm_kernel<T, double, T><<<dim3((unsigned)(cells / 64), r / 64, 1), 256, 0, s>>>(
      r, src, r, 1, 0, o->Q, to_given ? 1 : r, to_given ? r : 1, 0, dst, r, 1, 0);
  return bbfmm_set_cuda_error(cudaGetLastError(), "sym_rotate", __FILE__, __LINE__);
}

static int64_t sym_tiles(int level, int nsets) {
  const int P = 1 << (level - 1);
  if (P == 2) return 8 * (int64_t)((nsets + 7) / 8);
  const int64_t nb = P / 4;
  return 8 * nsets * nb * nb * nb;
}

// Step groups (CTAs per target tile): the count that makes the waves of the 148 SMs fullest, each
// group more being charged the traffic of its partial sums (about 1/500 of a tile's time).
static int sym_groups(int64_t tiles) {
  int best = 1;
  double cost = 1e300;
  for (int g = 1; g <= DMMA_PARTS; ++g) {
    const double c = (double)((tiles * g + 147) / 148) / g + (g > 1 ? 0.002 * g * (double)tiles / 148 : 0.0);
    if (c < cost * 0.99) {
      cost = c;
      best = g;
    }
  }
  return best;
}
int sym_default_groups(int level, int nsets) { return sym_groups(sym_tiles(level, nsets)); }

// The same for a list of blocks of a level of `cells` cells, whose slices are the level's: at most
// 65,536 cells of them (16 groups at level 4, 2 at level 5, 134 MB).
int sym_list_groups(int nboxes, int64_t cells) {
  const int64_t most = 65536 / cells;
  const int g = sym_groups(8 * (int64_t)((nboxes + 7) / 8));
  return g < most ? g : (most > 1 ? (int)most : 1);
}

// Writes Lout (assign, rotated basis) for every cell of the level, or with a box list of 2 x 2 x 2
// blocks of parent cells (set, x0, y0, z0) for their cells only, in `ngroups` step groups (fewer where
// the scratch holds fewer).
template <typename T>
int launch_m2l_sym(const void *op, const T *M, T *Lout, int level, double *part, int64_t part_elems, cudaStream_t s, int nsets,
                   int ngroups, const int4 *boxes, int nboxes) {
  const SymOps *o = (const SymOps *)op;
  const int64_t P = (int64_t)1 << (level - 1);
  if (boxes && (nboxes < 0 || nboxes > nsets * P * P * P / 8))
    return bbfmm_set_error(BBFMM_ERR_ARG, "box list longer than the level");
  if (boxes && nboxes == 0) return BBFMM_OK;
  const int64_t count = 8 * (int64_t)nsets * P * P * P * sy::R;
  const int64_t tiles = boxes ? 8 * (int64_t)((nboxes + 7) / 8) : sym_tiles(level, nsets);
  int ng = ngroups < DMMA_PARTS ? ngroups : DMMA_PARTS;
  if (!part) ng = 1;
  else if (ng > 1 && (int64_t)ng * count > part_elems) ng = (int)(part_elems / count);
  if (ng < 1) ng = 1;
  const dim3 grid((unsigned)tiles, ng);
  if (ng > 1) {
    BBFMM_CUDA_OK((smem_opt_in<sy::m2l_sym_kernel<T, double>>(sy::SMEM_BYTES)));
    sy::m2l_sym_kernel<T, double><<<grid, sy::THREADS, sy::SMEM_BYTES, s>>>(M, o->Bsteps, o->steps, o->nsteps, o->orbits, part,
                                                                          level, o->cl, boxes, nboxes, nsets);
  } else {
    BBFMM_CUDA_OK((smem_opt_in<sy::m2l_sym_kernel<T, T>>(sy::SMEM_BYTES)));
    sy::m2l_sym_kernel<T, T><<<grid, sy::THREADS, sy::SMEM_BYTES, s>>>(M, o->Bsteps, o->steps, o->nsteps, o->orbits, Lout,
                                                                     level, o->cl, boxes, nboxes, nsets);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || ng == 1) return bbfmm_set_cuda_error(e, "m2l_sym", __FILE__, __LINE__);
  if (!boxes) return launch_sum_parts<T>(count, ng, part, Lout, s);
  sy::sym_sum_boxes_kernel<T><<<nboxes, 256, 0, s>>>(count, ng, (int)P, boxes, part, Lout);
  return bbfmm_set_cuda_error(cudaGetLastError(), "m2l_sym parts", __FILE__, __LINE__);
}

#define SYM_INST(T)                                                                                                   \
  template int sym_prepare<T>(int, int, const T *, const T *, const T *, const T *, T *, T *, void **, cudaStream_t);    \
  template int sym_rotate<T>(const void *, bool, int64_t, const T *, T *, cudaStream_t);                              \
  template int launch_m2l_sym<T>(const void *, const T *, T *, int, double *, int64_t, cudaStream_t, int, int, const int4 *, int);
SYM_INST(double)
SYM_INST(float)

}  // namespace bbfmm
