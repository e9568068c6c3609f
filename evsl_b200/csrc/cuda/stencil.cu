// Chebyshev filter on the merged stencil of a matrix (stencil.cuh): the FP64
// single-vector filter ChebAv (SRC/chebpoly.c:519-598), bit for bit.
//
//   * k_st_step: one launch per degree.  A thread takes J (1 or 2) rows that
//     lie the stencil's largest offset S apart: the gather of row r + S is the
//     next row's own value, so the planes of a 3-D grid (or the lines of a 2-D
//     one) come from L2 (J + 2) / (3 J) times as often, and the loads of both
//     rows are in flight together (the kernel waits for L2, not for DRAM: the
//     vectors of 10^6 rows stay there).  The result
//     y += mu_k w_k is brought up to date every third degree only: the last
//     three w's of a row are in registers then (w_k is formed, w_k-1 is the
//     row's own value of the gathered vector, w_k-2 the recurrence's third
//     term), and adding them one after another is the same sum in the same
//     order at 16 / 3 instead of 16 bytes of y per row and degree.
//     Against the dictionary kernels before it (sparse.cu, the fastest of the
//     seven timed): 3-D Laplacian of 10^6 rows 7.84 -> 6.32 us a degree, 343
//     thousand rows 4.57 -> 3.18, 10^4 rows 2.95 -> 2.4 (launch latency).
//   * k_st_cluster: every degree in one launch, for operators whose vectors
//     fit the shared memory of one thread-block cluster: 10^4 rows 2.4 -> 0.52.
//   * k_st_cols, k_st_clusters: the same two for several columns, each with
//     its own polynomial; k_st_kpm, k_st_kpm_cluster: the same two with the
//     KPM recurrence's inner products; k_st_spmv: the plain product.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <type_traits>
#include <vector>

#include "stencil.cuh"

using namespace evslcu;

namespace {

// ---------------------------------------------------------------------------
// build
// ---------------------------------------------------------------------------
template <class MT>
__global__ void k_st_mask(int n, const unsigned short *__restrict__ pid, const unsigned *__restrict__ tab, MT *mask) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) mask[r] = (MT)tab[pid[r]];
}

// ---------------------------------------------------------------------------
// one degree per launch
// ---------------------------------------------------------------------------
// Rows of thread-column c: (c / S) * J * S + c % S + j * S, j = 0..J-1.
struct StMarch {
  int S, J, cols;
  unsigned magic;  // floor(2^32 / S)
  int ahead;       // one column: blocks that run at once, and so beside the launch ahead
};

// What a degree does to y: terms pending since y was last written (0: none
// now), their coefficients (c2 w_k-2 + c1 w_k-1 + c0 w_k), and whether y
// starts with the first of them.
template <class VT>
struct StY {
  int terms, init;
  VT c2, c1, c0;
};

// J > 1 needs a stencil whose first and last offsets are -S and +S around a
// diagonal entry in the middle (StArg::center).
// Returns the sum of dotv[r] y[r] over the thread's rows (EPI).  yd: where the
// finished y goes (the last degree), else null.
// each(x, w) is called for every row, with its values of v_k and of the result.
// LONE: one column's launch.  Its first blocks prefetch v_k-1, and with J > 1 a
// row's own v_k is loaded before the masks are looked at.
template <class VT, int D, int J, bool FIRST, bool EPI, bool LONE, class F>
__device__ __forceinline__ double st_rows(const StArg<VT, D> &A, const StMarch &M, const VT *__restrict__ vk,
                                          const VT *vkm1, VT *out, VT *y, double *yd, VT t, VT ncc, const StY<VT> &Y,
                                          const double *__restrict__ zold, double nbeta,
                                          const double *__restrict__ dotv, F &&each) {
  constexpr bool OWN = LONE && J > 1;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  int r0 = c;
  if (J > 1) {
    unsigned q = __umulhi((unsigned)c, M.magic);
    int rem = c - (int)q * M.S;
    if (rem >= M.S) {
      ++q;
      rem -= M.S;
    }
    r0 = c < M.cols ? (int)q * J * M.S + rem : A.n;
  }
  // Only the masks are loaded before the wait: the host has waited for the
  // kernel that wrote them (stencil_build).  v_k-1 was written two launches
  // ago, but it is the wait that makes other launches' writes visible; before it
  // the blocks that start beside the launch ahead may only ask for it to be
  // brought near: 343 thousand rows 3.55 -> 3.18 us a degree, 10^6 6.50 -> 6.32
  // (6.54 when the blocks of later waves ask as well).  What needs no mask is
  // loaded before the masks are looked at, which costs the blocks that start
  // after the wait no second latency: 10^6 rows 6.87 -> 6.50.  The prefetch and
  // the early own row gain in one column's launches and lose where many columns
  // fill the chip.
  unsigned m[J];
  bool live[J];
  bool all = true;
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const int r = r0 + j * M.S;
    live[j] = r < A.n;
    m[j] = live[j] ? (unsigned)__ldg(A.mask + r) : 0u;
    if (LONE && !FIRST && live[j] && (int)blockIdx.x < M.ahead)
      asm volatile("prefetch.global.L1 [%0];" ::"l"(vkm1 + r));
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const VT *xr = vk + r0;
  VT acc[J], x[J], xm1[J], yo[J];
#pragma unroll
  for (int j = 0; j < J; ++j) xm1[j] = (!FIRST && live[j]) ? vkm1[r0 + j * M.S] : (VT)0;
#pragma unroll
  for (int j = 0; j < J; ++j) yo[j] = (Y.terms && !Y.init && live[j]) ? y[r0 + j * M.S] : (VT)0;
  VT own[J];  // OWN
  if (OWN) {
#pragma unroll
    for (int j = 0; j < J; ++j) own[j] = live[j] ? __ldg(xr + j * M.S) : (VT)0;
  }
#pragma unroll
  for (int j = 0; j < J; ++j) all = all && m[j] == A.full;
  all = __all_sync(0xffffffffu, all);
  if constexpr (J == 1) {
    acc[0] = (VT)0;
    x[0] = (VT)0;
    if (all) {
      VT g[D];
#pragma unroll
      for (int e = 0; e < D; ++e) g[e] = __ldg(xr + A.off[e]);
#pragma unroll
      for (int e = 0; e < D; ++e) acc[0] = st_fmadd(A.val[e], g[e], acc[0]);
      x[0] = A.center ? g[D / 2] : __ldg(xr);
    } else {
      // an entry the row does not have adds -0: no change to any sum
      VT g[D];
#pragma unroll
      for (int e = 0; e < D; ++e) g[e] = (m[0] >> e & 1u) ? __ldg(xr + A.off[e]) : st_zero(A.val[e]);
      if (live[0]) x[0] = __ldg(xr);
#pragma unroll
      for (int e = 0; e < D; ++e) acc[0] = st_fmadd(A.val[e], g[e], acc[0]);
    }
  } else {
    // p[j]: the value one S below row j; rows share it with their neighbours
    VT p[J + 2], g[J][D];
    if (all) {
#pragma unroll
      for (int j = 0; j < J + 2; ++j) p[j] = (OWN && j >= 1 && j <= J) ? own[j - 1] : __ldg(xr + (j - 1) * M.S);
#pragma unroll
      for (int j = 0; j < J; ++j)
#pragma unroll
        for (int e = 1; e < D - 1; ++e)
          if (e != D / 2) g[j][e] = __ldg(xr + j * M.S + A.off[e]);
#pragma unroll
      for (int j = 0; j < J; ++j) {
        VT a = (VT)0;
#pragma unroll
        for (int e = 0; e < D; ++e)
          a = st_fmadd(A.val[e], e == 0 ? p[j] : e == D / 2 ? p[j + 1] : e == D - 1 ? p[j + 2] : g[j][e], a);
        acc[j] = a;
      }
    } else {
#pragma unroll
      for (int j = 0; j < J + 2; ++j) {
        const bool have = j == 0 ? (m[0] & 1u) != 0 : j == J + 1 ? (m[J - 1] >> (D - 1) & 1u) != 0 : live[j == 0 ? 0 : j > J ? J - 1 : j - 1];
        p[j] = (OWN && j >= 1 && j <= J) ? own[j - 1] : have ? __ldg(xr + (j - 1) * M.S) : (VT)0;
      }
#pragma unroll
      for (int j = 0; j < J; ++j)
#pragma unroll
        for (int e = 1; e < D - 1; ++e)
          if (e != D / 2) g[j][e] = (m[j] >> e & 1u) ? __ldg(xr + j * M.S + A.off[e]) : (VT)0;
#pragma unroll
      for (int j = 0; j < J; ++j) {
        VT a = (VT)0;
#pragma unroll
        for (int e = 0; e < D; ++e)
          if (m[j] >> e & 1u)
            a = st_fmadd(A.val[e], e == 0 ? p[j] : e == D / 2 ? p[j + 1] : e == D - 1 ? p[j + 2] : g[j][e], a);
        acc[j] = a;
      }
    }
#pragma unroll
    for (int j = 0; j < J; ++j) x[j] = p[j + 1];
  }
  double dsum = 0.0;
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const int r = r0 + j * M.S;
    if (!live[j]) continue;
    // vkp1 = A vk; vkp1 += (-cc) vk; vkp1 *= t; vkp1 += (-1) vkm1
    VT w = st_mul(t, st_add(acc[j], st_mul(ncc, x[j])));
    if (!FIRST) w = st_add(w, -xm1[j]);
    out[r] = w;
    each(x[j], w);
    if (Y.terms) {
      VT yv = yo[j];
      if (Y.terms == 3) yv = Y.init ? st_mul(Y.c2, xm1[j]) : st_fmadd_y(Y.c2, xm1[j], yv);
      if (Y.terms >= 2) yv = (Y.init && Y.terms == 2) ? st_mul(Y.c1, x[j]) : st_fmadd_y(Y.c1, x[j], yv);
      yv = st_fmadd_y(Y.c0, w, yv);
      if (yd) {
        double yo2 = (double)yv;
        if (EPI) {
          if (zold) yo2 = __dadd_rn(yo2, __dmul_rn(nbeta, zold[r]));
          if (dotv) dsum += dotv[r] * yo2;
        }
        yd[r] = yo2;
      } else {
        y[r] = yv;
      }
    }
  }
  return dsum;
}

template <int D, int J, bool FIRST, bool EPI>
__global__ void __launch_bounds__(kThreads, J == 2 ? 5 : D <= 9 ? 6 : 2)
    k_st_step(const __grid_constant__ StArg<double, D> A, StMarch M, const double *__restrict__ vk, const double *vkm1,
              double *out, double *y, double *yd, double t, double ncc, StY<double> Y,
              const double *__restrict__ zold, double nbeta, const double *__restrict__ dotv, double *part,
              unsigned int *ctr, double *dot_out) {
  __shared__ double sh[EPI ? kThreads / 32 : 1];
  const double dsum = st_rows<double, D, J, FIRST, EPI, true>(A, M, vk, vkm1, out, y, yd, t, ncc, Y, zold, nbeta, dotv,
                                                              [](double, double) {});
  if (EPI && dot_out) {
    const double b = block_sum(dsum, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = b;
    if (last_block(ctr)) {
      const double tot = reduce_partials(part, gridDim.x, ctr, sh);
      if (threadIdx.x == 0) *dot_out = tot;
    }
  }
}

// The same degree for several columns of one operator (column in blockIdx.y),
// each with its own polynomial.  Columns stay apart in memory: the operator
// costs a byte per row, so there is nothing to share between them, and the
// vectors of a few columns fit L2 where one interleaved block would not.
constexpr int kStCols = 16;

template <class VT>
struct StStepCol {
  const VT *vk, *vkm1;
  VT *out, *y;
  double *yd;        // last degree: where the finished y goes
  const double *mu;  // device
  VT t, ncc;
  int from, flush;  // flush: y takes the terms from .. k now
};
template <class VT>
struct StStepCols {
  StStepCol<VT> c[kStCols];
};

template <class VT, int D, int J, bool FIRST>
__global__ void __launch_bounds__(kThreads, J == 2 ? 5 : D <= 9 ? 6 : 2)
    k_st_cols(const __grid_constant__ StArg<VT, D> A, StMarch M, const __grid_constant__ StStepCols<VT> C, int k) {
  const StStepCol<VT> &I = C.c[blockIdx.y];
  StY<VT> Y{0, 0, (VT)0, (VT)0, (VT)0};
  if (I.flush) {
    Y.terms = k - I.from + 1;
    Y.init = I.from == 0;
    Y.c0 = (VT)__ldg(I.mu + k);
    Y.c1 = (VT)__ldg(I.mu + k - 1);
    Y.c2 = (VT)__ldg(I.mu + (FIRST ? 0 : k - 2));
  }
  st_rows<VT, D, J, FIRST, false, false>(A, M, I.vk, I.vkm1, I.out, I.y, I.yd, I.t, I.ncc, Y, nullptr, 0.0, nullptr,
                                         [](VT, VT) {});
}

// One KPM step (two moments per product, as k_kpm_dbl in sparse.cu) for the
// probes of a group, probe in blockIdx.y, vectors of n values one after
// another: w_k+1 and the block's sums of w_k+1^2, w_k+1 w_k and, at the first
// step, w_0^2, into part[(sum * probes + probe) * blocks + block].  The blocks,
// and so the order of the sums, follow from n alone.
template <int D, int J, bool FIRST>
__global__ void __launch_bounds__(kThreads, J == 2 ? 5 : D <= 9 ? 6 : 2)
    k_st_kpm(const __grid_constant__ StArg<double, D> A, StMarch M, const double *__restrict__ vk, const double *vkm1,
             double *out, double t, double ncc, double *part) {
  constexpr int NS = FIRST ? 3 : 2, NW = kThreads / 32;
  __shared__ double sh[NS][NW];
  const long long at = (long long)blockIdx.y * A.n;
  double s[3] = {0.0, 0.0, 0.0};
  const StY<double> Y{0, 0, 0.0, 0.0, 0.0};
  st_rows<double, D, J, FIRST, false, false>(A, M, vk + at, FIRST ? nullptr : vkm1 + at, out + at, nullptr, nullptr, t,
                                             ncc, Y, nullptr, 0.0, nullptr, [&](double x, double w) {
                                               s[0] += w * w;
                                               s[1] += w * x;
                                               if (FIRST) s[2] += x * x;
                                             });
  // one barrier for all the sums (block_sum's two each kept the warps of a
  // block waiting a third of the time)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NS; ++q) {
    s[q] = warp_sum(s[q]);
    if (lane == 0) sh[q][warp] = s[q];
  }
  __syncthreads();
  if (threadIdx.x < NS) {
    double b = 0.0;
#pragma unroll
    for (int w = 0; w < NW; ++w) b += sh[threadIdx.x][w];
    part[((long long)threadIdx.x * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = b;
  }
}

// The sums of several steps, step and sum in blockIdx.y, probe of the group in
// blockIdx.x: part's `blocks` entries in fixed order.  raw: [step * 3 + sum]
// [all probes], at this group's first probe.
__global__ void __launch_bounds__(kThreads)
    k_st_kpm_sum(int blocks, const double *__restrict__ part, double *raw, int nvec) {
  __shared__ double sh[kThreads / 32];
  const double *p = part + ((long long)blockIdx.y * gridDim.x + blockIdx.x) * blocks;
  double t = 0.0;
  for (int i = threadIdx.x; i < blocks; i += kThreads) t += p[i];
  t = block_sum(t, sh);
  if (threadIdx.x == 0) raw[(long long)blockIdx.y * nvec + blockIdx.x] = t;
}

// Unit probes: block b of a probe's 64 sums its squares, then every block
// scales its share (two launches; the sums' order follows from n alone).
constexpr int kNormBlocks = 64;
__global__ void __launch_bounds__(kThreads) k_st_sumsq(int n, const double *__restrict__ x, double *part) {
  __shared__ double sh[kThreads / 32];
  const double *xc = x + (long long)blockIdx.y * n;
  double t = 0.0;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) t += xc[r] * xc[r];
  t = block_sum(t, sh);
  if (threadIdx.x == 0) part[blockIdx.y * gridDim.x + blockIdx.x] = t;
}
__global__ void __launch_bounds__(kThreads) k_st_unit(int n, const double *__restrict__ x, const double *part, double *v) {
  __shared__ double inv;
  if (threadIdx.x < 32) {
    double t = part[blockIdx.y * kNormBlocks + threadIdx.x] + part[blockIdx.y * kNormBlocks + 32 + threadIdx.x];
    t = warp_sum(t);
    if (threadIdx.x == 0) inv = 1.0 / sqrt(t);
  }
  __syncthreads();
  const double s = inv;
  const long long at = (long long)blockIdx.y * n;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) v[at + r] = __dmul_rn(s, x[at + r]);
}

__global__ void k_st_float(int n, const double *__restrict__ x, float *out) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) out[r] = (float)x[r];
}

// Two rows per thread: FP64 columns and probes from kStTwoRows rows on; FP32
// columns also, and one column only, where one row per thread would need more
// blocks than run at once (6 on an SM).
// Measured before v_k-1 was prefetched, us a degree of one column, 1 / 2 rows per
// thread: 215 thousand rows 2.73 / 3.41, 343 thousand 3.57 / 3.56, 450 thousand
// 3.81 / 4.17, 592 thousand 4.50 / 4.59, 10^6 (3-D) 6.35 / 6.49, 10^6 (2-D) 5.74 /
// 5.37, 4.1 million 25.3 / 25.3; three rows were 4-8% slower than two at every
// size.  FP32 columns
// of a 5-point operator: 100 thousand rows x 16 9.82 / 7.43 (the packing kernel
// 8.64), x 4 3.76 / 3.14, 40 thousand x 8 3.55 / 3.16; FP64, 9 points: 100
// thousand x 16 10.5 / 10.7, x 4 4.08 / 4.84.
constexpr int kStTwoRows = 150000;
bool st_over_one_wave(long long rows) { return rows > 6LL * kThreads * sm_count(); }

StMarch st_march(int n, int span, bool sym, bool two) {
  StMarch M;
  int J = two ? 2 : 1;
  if (!sym || span < 1 || (long long)span * J > n || n > (1 << 29)) J = 1;
  M.S = J > 1 ? span : std::max(n, 1);
  M.J = J;
  M.ahead = 0;
  const long long groups = ((long long)n + (long long)M.S * J - 1) / ((long long)M.S * J);
  M.cols = (int)(groups * M.S);
  M.magic = (unsigned)((1ull << 32) / (unsigned long long)M.S - (M.S == 1 ? 1 : 0));
  return M;
}

template <int D>
int st_step(const evslcu_mat *A, bool first, const double *vk, const double *vkm1, double *out, double *y, double t,
            double ncc, const StY<double> &Y, bool last, const evslcu_cheb_epi *ep) {
  const StArg<double, D> S = st_arg<double, D>(A);
  StMarch M = st_march(A->n, A->st_span, D <= 9 && S.center && S.off[0] == -S.off[D - 1], st_over_one_wave(A->n));
  M.ahead = sm_count() * (M.J == 2 ? 5 : 6);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((M.cols + kThreads - 1) / kThreads);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = stream();
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const bool epi = ep && (int)cfg.gridDim.x <= kMaxPartials;
  auto pick = [&](auto Jc) {
    constexpr int J = D <= 9 ? decltype(Jc)::value : 1;
    return first ? (epi ? k_st_step<D, J, true, true> : k_st_step<D, J, true, false>)
                 : (epi ? k_st_step<D, J, false, true> : k_st_step<D, J, false, false>);
  };
  auto fn = M.J == 2 ? pick(std::integral_constant<int, 2>()) : pick(std::integral_constant<int, 1>());
  cudaError_t e = cudaLaunchKernelEx(&cfg, fn, S, M, vk, vkm1, out, y, last ? y : nullptr, t, ncc, Y,
                                     epi ? ep->zold : nullptr, epi ? ep->nbeta : 0.0, epi ? ep->dotv : nullptr,
                                     partials(), counters() + CTR_CHEB, epi ? ep->dot_out : nullptr);
  if (e != cudaSuccess) return fail(EVSLCU_ERR_CUDA, "stencil filter launch failed: %s", cudaGetErrorString(e));
  EVSLCU_LAUNCH_CHECK("k_st_step");
  if (ep && !epi) return launch_lan_epi(A->n, ep, y);
  return 0;
}

int st_step_any(const evslcu_mat *A, bool first, const double *vk, const double *vkm1, double *out, double *y, double t,
                double ncc, const StY<double> &Y, bool last, const evslcu_cheb_epi *ep) {
  switch (st_width(A->st_d)) {
    case 5: return st_step<5>(A, first, vk, vkm1, out, y, t, ncc, Y, last, ep);
    case 7: return st_step<7>(A, first, vk, vkm1, out, y, t, ncc, Y, last, ep);
    case 9: return st_step<9>(A, first, vk, vkm1, out, y, t, ncc, Y, last, ep);
    case 16: return st_step<16>(A, first, vk, vkm1, out, y, t, ncc, Y, last, ep);
    default: return st_step<32>(A, first, vk, vkm1, out, y, t, ncc, Y, last, ep);
  }
}

// y = A x, column c in blockIdx.y (leading dimension ld).
template <int D>
__global__ void __launch_bounds__(kThreads)
    k_st_spmv(const __grid_constant__ StArg<double, D> A, const double *__restrict__ X, double *__restrict__ Y,
              long long ld) {
  const double *x = X + (long long)blockIdx.y * ld;
  double *y = Y + (long long)blockIdx.y * ld;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < A.n; r += gridDim.x * blockDim.x) {
    const unsigned m = (unsigned)__ldg(A.mask + r);
    double g[D], acc = 0.0;
#pragma unroll
    for (int e = 0; e < D; ++e) g[e] = (m >> e & 1u) ? __ldg(x + r + A.off[e]) : st_zero(A.val[e]);
#pragma unroll
    for (int e = 0; e < D; ++e) acc = st_fmadd(A.val[e], g[e], acc);
    y[r] = acc;
  }
}

// ---------------------------------------------------------------------------
// every degree in one launch: one thread-block cluster per column
// ---------------------------------------------------------------------------
// Most threads of a block: 64 registers with one row per thread and the
// operator in the kernel's arguments, 80 with several rows, 128 with an
// operator from a table.
constexpr int cl_threads(int cap, bool one) { return cap < 0 ? 512 : one ? 1024 : 768; }
constexpr int kClMaxD = 9;       // widest stencil

// One column: its operator, polynomial, vectors and Lanczos epilogue.  Block c
// of the cluster holds rows c * R .. c * R + R - 1.
struct StCol {
  const void *mask;
  const double *x;
  double *y;
  const double *mu;  // device, deg + 1 (null: the launch's own copy)
  const double *zold, *dotv;
  double *dot_out;
  double nbeta, t1, t2, ncc;
  int n, deg, d, R, halo, y_smem;
  unsigned full;
  int center;
  int off[kClMaxD];
  double val[kClMaxD];
};

template <int CAP>
struct StMu {
  double v[CAP > 0 ? CAP : 1];
};

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// Address of this block's shared variable p in block `rank` of the cluster.
__device__ __forceinline__ unsigned peer_addr(const void *p, unsigned rank) {
  unsigned a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void peer_store(unsigned a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
// Stores v at address a of another block and counts its bytes on that block's
// mbarrier bar.
__device__ __forceinline__ void peer_send(unsigned a, double v, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(a),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void peer_send(unsigned a, float v, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(a),
               "r"(__float_as_uint(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void bar_init(unsigned long long *bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((unsigned)__cvta_generic_to_shared(bar)) : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned long long *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(bar)),
               "r"(bytes)
               : "memory");
}
// Waits for the phase of the given parity; false when the polls run out, or
// after one poll when another wait of the block has.  The first poll returns at
// once, each later one suspends the thread for up to a microsecond, so that the
// default limit is about a second.
constexpr int kClPolls = 1 << 20;
int g_cl_polls = kClPolls;
__device__ __forceinline__ bool bar_wait(unsigned long long *bar, unsigned parity, int polls, const int *dead) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(bar);
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(a), "r"(parity)
      : "memory");
  for (int i = 1; !ok && i < polls && !*(const volatile int *)dead; ++i)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(a), "r"(parity), "r"(1000)
        : "memory");
  return ok != 0;
}
// The end of a block that gave up, after a cluster barrier that the others
// reach (or leave the kernel) without sending again: values already on their
// way to its shared memory need a microsecond or two to arrive; this is about a
// hundred.
__device__ __forceinline__ void linger() {
  const long long t = clock64();
  while (clock64() - t < 200000) __nanosleep(1000);
}

// Shared memory: two vectors of R rows with a halo on both sides, which take
// turns as v_k and as v_k-1 / w, and y (FP64 columns too long for it keep y in
// global memory).  A degree reads only this block's shared memory; w of the
// rows within `halo` of an edge is also sent into the neighbour's halo.
//
// Blocks wait for their two neighbours only, through the data itself: a send
// counts its bytes on the receiver's mbarrier (one per degree parity), and
// the warps whose rows read a halo wait for degree k - 1's bytes before they
// start degree k.  (A cluster barrier per degree with release / acquire
// measured 370-500 cycles, this wait is covered by the other rows' work.)
// The halo of v_k-1 may be overwritten by degree k + 1's sends only: the
// neighbour sends those after it has received this block's degree-k rows of
// that edge, which are exactly the rows that read the halo, each sent after
// its reads.  For the same reason a neighbour is at most one degree ahead, so
// two mbarriers are enough.  The last degree sends nothing, and a block's last
// wait has seen every byte sent to it.  (One bulk copy per side
// after a degree's rows, in place of the stores as they are computed, was 3-10%
// slower at every halo width.)
//
// A wait that runs out of polls sets *err (the host's mapped flag) and `dead`.
// From the next degree on the block announces no bytes, sends none and waits no
// more; it goes through its remaining degrees with whatever is there.  Its
// neighbours run out of polls in turn, at most two degrees later, so at most
// two degrees' bytes reach an mbarrier that does not expect them (its count
// takes 2^20 - 1).  The block's threads agree on `dead` at a barrier after the
// last degree, and a block that gave up stays until every other has left its
// last degree, at one cluster barrier; where the epilogue's sum has a cluster
// barrier for all blocks, it is that one.
//
// MANY: the launch's blocks may have more threads than this column's rows need
// (R is a multiple of a warp, so whole warps sit out).
//
// ONE: at most one row per thread, whose w_k, w_k-1 and y stay in registers.
// The instruction count per row is what bounds a degree (a first version with
// its first / last / y tests inside the row loop took 130-190 instructions per
// 32 rows: 0.97 us a degree on 10^4 rows, 3.8 us on 94,800), so those cases
// are compiled apart.
template <class VT, int D, bool ONE, bool MANY, class MU>
__device__ __forceinline__ void st_cluster_body(const StCol &I, MU mu, int polls, int *err) {
  constexpr int VB = (int)sizeof(VT);
  extern __shared__ __align__(16) unsigned char st_smem[];
  __shared__ double red[64];
  __shared__ __align__(16) unsigned long long bars[2];
  __shared__ int dead;
  VT *const sm = reinterpret_cast<VT *>(st_smem);
  const int tid = threadIdx.x, T = blockDim.x;
  const int cr = (int)cluster_rank(), cl = (int)cluster_size();
  const int R = I.R, H = I.halo, n = I.n, deg = I.deg;
  const int row0 = cr * R;
  const int rows = max(0, min(R, n - row0));
  const bool ysm = I.y_smem != 0;
  double *const yg = I.y + row0;
  using MT = typename StMaskT<D>::T;
  const MT *const mask = (const MT *)I.mask + row0;
  const bool low = cr > 0 && rows > 0, high = cr + 1 < cl && row0 + R < n;
  VT *src = sm + H, *dst = sm + (R + 2 * H) + H;
  VT *const ys = sm + 2 * (R + 2 * H);
  MT *const ms = reinterpret_cast<MT *>(ys + (ysm ? R : 0));
  if (tid == 0) {
    bar_init(bars);
    bar_init(bars + 1);
    dead = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = tid - H; i < R + H; i += T) {
    const int g = row0 + i;
    if (g >= 0 && g < n) src[i] = (VT)I.x[g];
  }
  // R = nit T rows, those past n empty ones; the last T are visited first, so
  // that the rows both neighbours wait for come early.
  const int nit = ONE ? 1 : (R + T - 1) / T;
  // bit `it`: the warp's rows of iteration `it` have every entry / read a halo
  unsigned fast = 0, edge = 0, m1 = 0;
  for (int it = 0, i = tid + (nit - 1) * T; it < nit; ++it, i = it == 1 ? tid : i + T) {
    if (MANY && i >= R) continue;
    m1 = i < rows ? (unsigned)__ldg(mask + i) : 0u;
    if (!ONE) ms[i] = (MT)m1;
    if (__all_sync(0xffffffffu, m1 == I.full)) fast |= 1u << it;
    if (__any_sync(0xffffffffu, i < rows && ((low && i < H) || (high && i >= R - H)))) edge |= 1u << it;
  }
  VT val[D];
  int off[D];
#pragma unroll
  for (int e = 0; e < D; ++e) {
    val[e] = (VT)I.val[e];
    off[e] = I.off[e];
  }
  const bool center = I.center != 0;
  const VT t1 = (VT)I.t1, t2 = (VT)I.t2, ncc = (VT)I.ncc;
  // the neighbours' copies: their rows R + i (below) and i - R (above) for row
  // i here; mapa takes addresses of this block's own variables, the rest is
  // added afterwards
  unsigned sl = low ? peer_addr(src, cr - 1) + R * VB : 0, dl = low ? peer_addr(dst, cr - 1) + R * VB : 0;
  unsigned sh = high ? peer_addr(src, cr + 1) - R * VB : 0, dh = high ? peer_addr(dst, cr + 1) - R * VB : 0;
  const unsigned bl = low ? peer_addr(bars, cr - 1) : 0, bh = high ? peer_addr(bars, cr + 1) : 0;
  const unsigned expect = (low ? (unsigned)(H * VB) : 0u) + (high ? (unsigned)(min(H, n - row0 - R) * VB) : 0u);
  if (cl > 1)
    cluster_sync();  // the mbarriers are set and every block runs before anything is sent
  else
    __syncthreads();
  double dsum = 0.0;
  VT rx = (VT)0, rm = (VT)0, ry = (VT)0;  // ONE: the row's w_k-1, w_k-2, y
  if (ONE && tid < rows) rx = src[tid];
  int from = 0;
  // degree k; FIRST: k = 1, LAST: k = deg, FLUSH: y takes the terms from..k
  auto degree = [&](int k, auto first_c, auto flush_c, auto last_c) {
    constexpr bool FIRST = decltype(first_c)::value, FLUSH = decltype(flush_c)::value, LAST = decltype(last_c)::value;
    const VT t = FIRST ? t1 : t2;
    VT c0 = (VT)0, c1 = (VT)0, c2 = (VT)0;
    const int terms = LAST ? k - from + 1 : 3;
    const bool init = from == 0;
    if (FLUSH) {
      c0 = (VT)mu(k);
      c1 = (VT)mu(k - 1);
      c2 = (VT)mu(FIRST ? 0 : k - 2);
    }
    bool stop = !FIRST && *(volatile int *)&dead;
    if (!LAST && tid == 0 && expect && !stop) bar_expect(bars + (k & 1), expect);
    if (!FIRST && edge && !bar_wait(bars + ((k - 1) & 1), (unsigned)((k - 2) >> 1) & 1u, polls, &dead)) {
      stop = true;
      *(volatile int *)&dead = 1;
      *(volatile int *)err = 1;
    }
    const unsigned bk = (unsigned)((k & 1) * 8);
    unsigned fb = fast, eb = stop ? 0u : edge;  // eb: iterations that send
#pragma unroll 2
    for (int it = 0, i = tid + (nit - 1) * T; it < nit; ++it, i = it == 1 ? tid : i + T, fb >>= 1, eb >>= 1) {
      if (MANY && i >= R) continue;
      const VT *xs = src + i;
      VT acc = (VT)0, x, xm1 = (VT)0;
      if (!FIRST) xm1 = ONE ? rm : dst[i];
      if (fb & 1u) {
        VT g[D];
#pragma unroll
        for (int e = 0; e < D; ++e)
          if (!ONE || e != D / 2) g[e] = xs[off[e]];
        if (ONE) g[D / 2] = center ? rx : xs[off[D / 2]];
        x = ONE ? rx : center ? g[D / 2] : xs[0];
#pragma unroll
        for (int e = 0; e < D; ++e) acc = st_fmadd(val[e], g[e], acc);
      } else {
        // an entry the row does not have adds -0: no change to any sum
        const unsigned m = ONE ? m1 : (unsigned)ms[i];
        VT g[D];
#pragma unroll
        for (int e = 0; e < D; ++e) {
          g[e] = st_zero(val[e]);
          if (m >> e & 1u) g[e] = xs[off[e]];
        }
        x = ONE ? rx : xs[0];
#pragma unroll
        for (int e = 0; e < D; ++e) acc = st_fmadd(val[e], g[e], acc);
      }
      VT w = st_mul(t, st_add(acc, st_mul(ncc, x)));
      if (!FIRST) w = st_add(w, -xm1);
      if (!LAST) {
        if ((eb & 1u) && i < rows) {
          if (low && i < H) peer_send(dl + (unsigned)(i * VB), w, bl + bk);
          if (high && i >= R - H) peer_send(dh + (unsigned)(i * VB), w, bh + bk);
        }
        dst[i] = w;
      }
      if (FLUSH && i < rows) {
        VT yv = (VT)0;
        if (!init) yv = ONE ? ry : ysm ? ys[i] : (VT)yg[i];
        if (!FIRST && terms == 3) yv = init ? st_mul(c2, xm1) : st_fmadd_y(c2, xm1, yv);
        if (terms >= 2) yv = (init && terms == 2) ? st_mul(c1, x) : st_fmadd_y(c1, x, yv);
        yv = st_fmadd_y(c0, w, yv);
        if (!LAST) {
          if (ONE)
            ry = yv;
          else if (ysm)
            ys[i] = yv;
          else
            yg[i] = (double)yv;
        } else {
          double yo = (double)yv;
          if (I.zold) yo = __dadd_rn(yo, __dmul_rn(I.nbeta, I.zold[row0 + i]));
          if (I.dotv) dsum += I.dotv[row0 + i] * yo;
          yg[i] = yo;
        }
      }
      if (ONE) {
        rm = rx;
        rx = w;
      }
    }
    if (FLUSH) from = k + 1;
    if (!LAST) {
      __syncthreads();
      VT *const p = src;
      src = dst;
      dst = p;
      unsigned q = sl;
      sl = dl;
      dl = q;
      q = sh;
      sh = dh;
      dh = q;
    }
  };
  const std::true_type yes{};
  const std::false_type no{};
  if (deg == 1) {
    degree(1, yes, yes, yes);
  } else {
    degree(1, yes, no, no);
    int k = 2;
    for (; k + 2 < deg; k += 3) {
      degree(k, no, yes, no);
      degree(k + 1, no, no, no);
      degree(k + 2, no, no, no);
    }
    if (k < deg) {
      degree(k, no, yes, no);
      ++k;
    }
    if (k < deg) {
      degree(k, no, no, no);
      ++k;
    }
    degree(k, no, yes, yes);
  }
  bool gave_up = false;
  if (cl > 1) {
    __syncthreads();
    gave_up = dead != 0;
  }
  if (I.dot_out) {
    // the blocks' sums in rank order, added by block 0
    const double b = block_sum(dsum, red);
    if (cl > 1) {
      if (tid == 0) peer_store(peer_addr(red + 32 + cr, 0), b);
      cluster_sync();
      if (cr == 0 && tid == 0) {
        double s = 0.0;
        for (int c = 0; c < cl; ++c) s += red[32 + c];
        *I.dot_out = s;
      }
    } else if (tid == 0) {
      *I.dot_out = b;
    }
  } else if (gave_up) {
    cluster_sync();
  }
  if (gave_up) linger();
}

// One cluster filters `one`, whose coefficients (up to CAP) come with the
// launch, or from the device when CAP is 0.
template <class VT, int D, int CAP, bool ONE>
__global__ void __launch_bounds__(cl_threads(CAP, ONE), 1)
    k_st_cluster(const __grid_constant__ StCol one, const __grid_constant__ StMu<CAP> mus, int polls, int *err) {
  if constexpr (CAP > 0) {
    st_cluster_body<VT, D, ONE, false>(one, [&](int k) { return mus.v[k]; }, polls, err);
  } else {
    const double *mup = one.mu;
    st_cluster_body<VT, D, ONE, false>(one, [&](int k) { return __ldg(mup + k); }, polls, err);
  }
}

// Cluster q of the launch filters column q of the table, whatever its
// operator: columns of one matrix, or of as many matrices.
constexpr int kClCols = 32;
struct StTab {
  StCol c[kClCols];
};
template <class VT, int D, bool ONE>
__global__ void __launch_bounds__(cl_threads(-1, ONE), 1)
    k_st_clusters(const __grid_constant__ StTab tab, int polls, int *err) {
  const StCol &I = tab.c[blockIdx.x / cluster_size()];
  const double *mup = I.mu;
  auto mu = [&](int k) { return __ldg(mup + k); };
  // 5- and 7-point operators may be in one launch, each with its own row product
  if (D == 7 && I.d <= 5)
    st_cluster_body<VT, 5, ONE, true>(I, mu, polls, err);
  else
    st_cluster_body<VT, D, ONE, true>(I, mu, polls, err);
}

// The whole KPM recurrence of a probe (k_st_kpm's steps, the probe made a unit
// vector first) on one cluster: cluster q of the launch takes probe q of x.
// Vectors, halos and waits are st_cluster_body's.  Block c of probe q leaves
// its sums of step k in part[((k * 3 + sum) * probes + q) * blocks + c].
template <int D, bool ONE>
__global__ void __launch_bounds__(cl_threads(0, ONE), 1)
    k_st_kpm_cluster(const __grid_constant__ StCol I, double *part, int probes, int polls, int *err) {
  constexpr int VB = (int)sizeof(double);
  extern __shared__ __align__(16) unsigned char st_smem[];
  __shared__ double red[64];
  __shared__ double sums[2][3][32];
  __shared__ __align__(16) unsigned long long bars[2];
  __shared__ int dead;
  double *const sm = reinterpret_cast<double *>(st_smem);
  const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = T >> 5;
  const int cr = (int)cluster_rank(), cl = (int)cluster_size(), probe = (int)(blockIdx.x / cl);
  const int R = I.R, H = I.halo, n = I.n, steps = I.deg;
  const int row0 = cr * R;
  const int rows = max(0, min(R, n - row0));
  using MT = typename StMaskT<D>::T;
  const MT *const mask = (const MT *)I.mask + row0;
  const double *const x0 = I.x + (long long)probe * n;
  const bool low = cr > 0 && rows > 0, high = cr + 1 < cl && row0 + R < n;
  double *src = sm + H, *dst = sm + (R + 2 * H) + H;
  MT *const ms = reinterpret_cast<MT *>(sm + 2 * (R + 2 * H));
  if (tid == 0) {
    bar_init(bars);
    bar_init(bars + 1);
    dead = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  double sq = 0.0;
  for (int i = tid - H; i < R + H; i += T) {
    const int g = row0 + i;
    if (g >= 0 && g < n) {
      const double v = x0[g];
      src[i] = v;
      if (i >= 0 && i < R) sq += v * v;
    }
  }
  const int nit = ONE ? 1 : R / T;
  unsigned fast = 0, edge = 0, m1 = 0;
  for (int it = 0, i = tid + (nit - 1) * T; it < nit; ++it, i = it == 1 ? tid : i + T) {
    m1 = i < rows ? (unsigned)__ldg(mask + i) : 0u;
    if (!ONE) ms[i] = (MT)m1;
    if (__all_sync(0xffffffffu, m1 == I.full)) fast |= 1u << it;
    if (__any_sync(0xffffffffu, i < rows && ((low && i < H) || (high && i >= R - H)))) edge |= 1u << it;
  }
  // the probe's norm: every block's sum in every block, added in rank order
  sq = block_sum(sq, red);
  if (cl > 1) {
    cluster_sync();
    if (tid == 0)
      for (int c = 0; c < cl; ++c) peer_store(peer_addr(red + 32 + cr, c), sq);
    cluster_sync();
  } else {
    if (tid == 0) red[32] = sq;
    __syncthreads();
  }
  double tot = 0.0;
  for (int c = 0; c < cl; ++c) tot += red[32 + c];
  const double inv = 1.0 / sqrt(tot);
  for (int i = tid - H; i < R + H; i += T) {
    const int g = row0 + i;
    if (g >= 0 && g < n) src[i] = __dmul_rn(inv, src[i]);
  }
  __syncthreads();
  unsigned dl = low ? peer_addr(dst, cr - 1) + R * VB : 0, sl = low ? peer_addr(src, cr - 1) + R * VB : 0;
  unsigned dh = high ? peer_addr(dst, cr + 1) - R * VB : 0, sh = high ? peer_addr(src, cr + 1) - R * VB : 0;
  const unsigned bl = low ? peer_addr(bars, cr - 1) : 0, bh = high ? peer_addr(bars, cr + 1) : 0;
  const unsigned expect = (low ? (unsigned)(H * VB) : 0u) + (high ? (unsigned)(min(H, n - row0 - R) * VB) : 0u);
  const bool center = I.center != 0;
  double rx = (ONE && tid < rows) ? src[tid] : 0.0, rm = 0.0;
  // a neighbour's first rows may arrive only after it has read its own probe,
  // and go to the other vector: no barrier is needed before the first step
  auto step = [&](int k, auto first_c) {  // k = 1, 2, ... as a filter's degrees
    constexpr bool FIRST = decltype(first_c)::value;
    const bool last = k == steps;
    const double t = FIRST ? I.t1 : I.t2;
    bool stop = !FIRST && *(volatile int *)&dead;
    if (!last && tid == 0 && expect && !stop) bar_expect(bars + (k & 1), expect);
    if (!FIRST && edge && !bar_wait(bars + ((k - 1) & 1), (unsigned)((k - 2) >> 1) & 1u, polls, &dead)) {
      stop = true;
      *(volatile int *)&dead = 1;
      *(volatile int *)err = 1;
    }
    const unsigned bk = (unsigned)((k & 1) * 8);
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    unsigned fb = fast, eb = stop ? 0u : edge;  // eb: iterations that send
    for (int it = 0, i = tid + (nit - 1) * T; it < nit; ++it, i = it == 1 ? tid : i + T, fb >>= 1, eb >>= 1) {
      const double *xs = src + i;
      double acc = 0.0, x, xm1 = 0.0, g[D];
      if (!FIRST) xm1 = ONE ? rm : dst[i];
      if (fb & 1u) {
#pragma unroll
        for (int e = 0; e < D; ++e)
          if (!ONE || e != D / 2) g[e] = xs[I.off[e]];
        if (ONE) g[D / 2] = center ? rx : xs[I.off[D / 2]];
        x = ONE ? rx : center ? g[D / 2] : xs[0];
      } else {
        const unsigned m = ONE ? m1 : (unsigned)ms[i];
#pragma unroll
        for (int e = 0; e < D; ++e) {
          g[e] = st_zero(I.val[e]);
          if (m >> e & 1u) g[e] = xs[I.off[e]];
        }
        x = ONE ? rx : xs[0];
      }
#pragma unroll
      for (int e = 0; e < D; ++e) acc = st_fmadd(I.val[e], g[e], acc);
      double w = __dmul_rn(t, __dadd_rn(acc, __dmul_rn(I.ncc, x)));
      if (!FIRST) w = __dadd_rn(w, -xm1);
      if (!last) {
        if ((eb & 1u) && i < rows) {
          if (low && i < H) peer_send(dl + (unsigned)(i * VB), w, bl + bk);
          if (high && i >= R - H) peer_send(dh + (unsigned)(i * VB), w, bh + bk);
        }
        dst[i] = w;
      }
      if (i < rows) {
        s0 += w * w;
        s1 += w * x;
        if (FIRST) s2 += x * x;
      }
      if (ONE) {
        rm = rx;
        rx = w;
      }
    }
    // the step's sums: one per warp now, the block's by warp 0 after the barrier
    s0 = warp_sum(s0);
    s1 = warp_sum(s1);
    if (FIRST) s2 = warp_sum(s2);
    if (lane == 0) {
      sums[k & 1][0][warp] = s0;
      sums[k & 1][1][warp] = s1;
      if (FIRST) sums[k & 1][2][warp] = s2;
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
      for (int q = 0; q < (FIRST ? 3 : 2); ++q) {
        const double b = warp_sum(lane < nw ? sums[k & 1][q][lane] : 0.0);
        if (lane == 0) part[((long long)((k - 1) * 3 + q) * probes + probe) * cl + cr] = b;
      }
    }
    double *const pv = src;
    src = dst;
    dst = pv;
    unsigned q = sl;
    sl = dl;
    dl = q;
    q = sh;
    sh = dh;
    dh = q;
  };
  step(1, std::true_type{});
  for (int k = 2; k <= steps; ++k) step(k, std::false_type{});
  if (cl > 1 && dead) {  // as st_cluster_body; the last step ended with a barrier
    cluster_sync();
    linger();
  }
}

// raw[i] = part[i * cl] + part[i * cl + 1] + ...
__global__ void k_st_kpm_cl_sum(int count, int cl, const double *__restrict__ part, double *raw) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  double s = 0.0;
  for (int c = 0; c < cl; ++c) s += part[(long long)i * cl + c];
  raw[i] = s;
}

// Blocks of the cluster, rows and shared memory of one column; cl 0: none fits.
struct ClPlan {
  int cl = 0, R = 0, T = 0, halo = 0, y_smem = 0;
  size_t smem = 0;
};
constexpr size_t kClSmemMax = 224 * 1024;  // of 227 KB, less the static and the reserved part

ClPlan cl_plan(int n, int reach, int d, size_t vb, int cl, int cap) {
  ClPlan P;
  const int halo = cl > 1 ? reach : 0;
  const int want = (std::max((n + cl - 1) / cl, halo) + 31) / 32 * 32;
  // R = nit T with as few empty rows as the block sizes allow
  int T = want, nit = 1;
  if (want > cl_threads(cap, true)) {
    const int most = cl_threads(cap, false);
    T = most;
    nit = (want + most - 1) / most;
    for (int t = most - 32; t >= most / 2; t -= 32) {
      const int k = (want + t - 1) / t;
      if (k * t < nit * T) {
        T = t;
        nit = k;
      }
    }
  }
  const int R = nit * T;
  if (nit > 32) return P;  // a bit per iteration
  const size_t vec = 2 * ((size_t)R + 2 * (size_t)halo), masks = nit > 1 ? (size_t)R * (size_t)st_mask_bytes(d) : 0;
  if ((vec + R) * vb + masks <= kClSmemMax)
    P.y_smem = 1;
  else if (vb != sizeof(double) || vec * vb + masks > kClSmemMax)
    return P;
  P.cl = cl;
  P.R = R;
  P.T = T;
  P.halo = halo;
  P.smem = (vec + (P.y_smem ? R : 0)) * vb + masks;
  return P;
}

int g_cl_force = 0;  // blocks per cluster: 0 the rule below, -1 no cluster

// Most blocks per cluster this device runs (16 is above the portable 8).
int cl_limit(const void *fn, int threads) {
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClSmemMax) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  const bool wide = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
  if (!wide) cudaGetLastError();
  for (int cl = wide ? 16 : 8; cl >= 1; cl /= 2) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cl);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = kClSmemMax;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cl;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int got = 0;
    if (cudaOccupancyMaxActiveClusters(&got, fn, &cfg) == cudaSuccess && got >= 1) return cl;
    cudaGetLastError();
  }
  return -1;
}

int *g_cl_err = nullptr;  // mapped host flag: a wait of the cluster filter ran out

int *cl_err() {
  if (!g_cl_err) {
    void *p = nullptr;
    if (cudaHostAlloc(&p, sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    g_cl_err = (int *)p;
    *g_cl_err = 0;
  }
  return g_cl_err;
}

template <class VT, int D, int CAP, bool ONE>
int cl_max1() {
  static int m = 0, dev = -1;  // limits are set per device
  if (m && dev == lib_device()) return m;
  dev = lib_device();
  if constexpr (CAP < 0)
    m = cl_limit((const void *)k_st_clusters<VT, D, ONE>, cl_threads(CAP, ONE));
  else
    m = cl_limit((const void *)k_st_cluster<VT, D, CAP, ONE>, cl_threads(CAP, ONE));
  return m;
}

template <class VT, int D, int CAP>
int cl_max() {
  return std::min(cl_max1<VT, D, CAP, true>(), cl_max1<VT, D, CAP, false>());
}

template <class VT, int D, int CAP>
int cl_launch(const StCol &one, const double *mu, const ClPlan &P) {
  int *err = cl_err();  // same address on the device (unified addressing)
  if (!err) return fail(EVSLCU_ERR_NOMEM, "cluster filter: out of pinned host memory");
  StMu<CAP> mus;
  if (CAP > 0) memcpy(mus.v, mu, sizeof(double) * (size_t)(one.deg + 1));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(P.cl);
  cfg.blockDim = dim3(P.T);
  cfg.dynamicSmemBytes = P.smem;
  cfg.stream = stream();
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = P.cl;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = P.R == P.T ? cudaLaunchKernelEx(&cfg, k_st_cluster<VT, D, CAP, true>, one, mus, g_cl_polls, err)
                           : cudaLaunchKernelEx(&cfg, k_st_cluster<VT, D, CAP, false>, one, mus, g_cl_polls, err);
  if (e != cudaSuccess) return fail(EVSLCU_ERR_CUDA, "cluster filter launch failed: %s", cudaGetErrorString(e));
  EVSLCU_LAUNCH_CHECK("k_st_cluster");
  return 0;
}

template <class VT, int CAP>
int cl_most(int d) {
  return d <= 5 ? cl_max<VT, 5, CAP>() : d <= 7 ? cl_max<VT, 7, CAP>() : cl_max<VT, 9, CAP>();
}
template <class VT, int CAP>
int cl_launch_d(const StCol &one, const double *mu, const ClPlan &P) {
  return one.d <= 5   ? cl_launch<VT, 5, CAP>(one, mu, P)
         : one.d <= 7 ? cl_launch<VT, 7, CAP>(one, mu, P)
                      : cl_launch<VT, 9, CAP>(one, mu, P);
}

template <class VT, int D>
int cl_launch_many(int ncols, const StTab &tab, int cl, int T, size_t smem, bool one) {
  int *err = cl_err();
  if (!err) return fail(EVSLCU_ERR_NOMEM, "cluster filter: out of pinned host memory");
  if ((one ? cl_max1<VT, D, -1, true>() : cl_max1<VT, D, -1, false>()) < cl)
    return fail(EVSLCU_ERR_CUDA, "clusters of %d blocks are not available", cl);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cl * ncols);
  cfg.blockDim = dim3(T);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream();
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = one ? cudaLaunchKernelEx(&cfg, k_st_clusters<VT, D, true>, tab, g_cl_polls, err)
                      : cudaLaunchKernelEx(&cfg, k_st_clusters<VT, D, false>, tab, g_cl_polls, err);
  if (e != cudaSuccess) return fail(EVSLCU_ERR_CUDA, "cluster filter launch failed: %s", cudaGetErrorString(e));
  EVSLCU_LAUNCH_CHECK("k_st_clusters");
  return 0;
}

void cl_column(StCol &C, const evslcu_mat *A, int deg, double cc, double dd, const double *x, double *y,
               const ClPlan &P, int D) {
  memset(&C, 0, sizeof(C));
  C.mask = A->st_mask;
  C.x = x;
  C.y = y;
  C.t1 = 1.0 / dd;
  C.t2 = 2.0 / dd;
  C.ncc = -cc;
  C.n = A->n;
  C.deg = deg;
  C.d = A->st_d;
  C.R = P.R;
  C.halo = P.halo;
  C.y_smem = P.y_smem;
  C.full = A->st_d == D ? (1u << D) - 1u : 0xffffffffu;
  C.center = A->st_d == D && A->st_off[D / 2] == 0;
  for (int e = 0; e < A->st_d; ++e) {
    C.off[e] = A->st_off[e];
    C.val[e] = A->st_val[e];
  }
}

// Device copy of the coefficients of a filter too long for a kernel argument.
double *g_cl_mu = nullptr;
int g_cl_mu_cap = 0;

constexpr int kClOneBlock = 512, kClMostRows5 = 4096, kClMostRows9 = 2304;

// The whole filter on one cluster; *done stays false when the operator does
// not fit one.
int cl_chebav(const evslcu_mat *A, const double *mu, int deg, double cc, double dd, const double *v, double *y,
              const evslcu_cheb_epi *epi, bool *done) {
  if (A->st_d > kClMaxD || g_cl_force < 0) return 0;
  const int most = deg < 64 ? cl_most<double, 64>(A->st_d) : deg < 512 ? cl_most<double, 512>(A->st_d) : cl_most<double, 0>(A->st_d);
  if (most < 1) return 0;
  // One cluster of all the blocks it may have; a block alone below kClOneBlock
  // rows, where a degree costs less than the exchange of halos.  Measured on
  // 16 blocks, us a degree: 0.48 on 1,480 rows, 0.52 on 10^4 (2-D), 0.60 on 6,840
  // (3-D), 1.28 on 38,000 (2-D), 1.8 on 26,000 (3-D), 2.7 on 94,800 (2-D),
  // 3.1 on 62,000 (3-D); k_st_step takes 2.2-2.6 on all of these.
  ClPlan P;
  for (int cl = g_cl_force ? g_cl_force : A->n <= kClOneBlock ? 1 : most; cl >= 1 && !P.cl; cl /= 2)
    P = cl_plan(A->n, A->st_reach, A->st_d, sizeof(double), std::min(cl, most), 0);
  if (!P.cl || (!g_cl_force && P.R > (A->st_d <= 5 ? kClMostRows5 : kClMostRows9))) return 0;
  StCol C;
  cl_column(C, A, deg, cc, dd, v, y, P, st_width(A->st_d));
  if (epi) {
    C.zold = epi->zold;
    C.nbeta = epi->nbeta;
    C.dotv = epi->dotv;
    C.dot_out = epi->dot_out;
  }
  *done = true;
  if (deg < 64) return cl_launch_d<double, 64>(C, mu, P);
  if (deg < 512) return cl_launch_d<double, 512>(C, mu, P);
  if (deg + 1 > g_cl_mu_cap) {
    evslcu_free(g_cl_mu);
    g_cl_mu_cap = std::max(deg + 1, 4096);
    g_cl_mu = (double *)evslcu_malloc(sizeof(double) * (size_t)g_cl_mu_cap);
    if (!g_cl_mu) {
      g_cl_mu_cap = 0;
      return EVSLCU_ERR_NOMEM;
    }
  }
  const int rc = evslcu_h2d_async(g_cl_mu, mu, sizeof(double) * (size_t)(deg + 1));
  if (rc) return rc;
  C.mu = g_cl_mu;
  return cl_launch_d<double, 0>(C, nullptr, P);
}

// Columns filtered together on clusters: col[i] of operator A[i], degree >= 1,
// coefficients on the device.
struct ClMany {
  const evslcu_mat *A;
  const double *mu;
  int deg;
  double cc, dd;
  const double *x;
  double *y;
};

// Most blocks per cluster of those launches (each kernel's own limit is set
// when it is first launched).
int cl_many_most(size_t vb) {
  return vb == sizeof(float) ? cl_max1<float, 7, -1, false>() : cl_max1<double, 7, -1, false>();
}

// Plan of one column in a launch of cl blocks per column and precision vb.
ClPlan cl_plan_many(const evslcu_mat *A, size_t vb, int cl) {
  if (A->st_d > kClMaxD) return ClPlan();
  return cl_plan(A->n, A->st_reach, A->st_d, vb, cl, -1);
}

// Microseconds of a degree of one column with that plan (as measured: up to
// 512 rows a block has one row per thread).
double cl_degree_us(const evslcu_mat *A, const ClPlan &P) {
  if (P.R <= 512) return A->st_d <= 5 ? 0.53 : 0.62;
  return 0.45 + (A->st_d <= 5 ? 0.7e-3 : 1.15e-3) * P.R;
}

// Clusters of cl blocks that run at once (a block has an SM to itself).
int cl_slots(int cl) {
  static int slots[17] = {}, dev = -1;
  if (dev != lib_device()) std::fill(slots, slots + 17, 0);
  dev = lib_device();
  if (slots[cl]) return slots[cl];
  cl_many_most(sizeof(double));  // sets the kernel's limits
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cl * sm_count());
  cfg.blockDim = dim3(cl_threads(-1, false));
  cfg.dynamicSmemBytes = kClSmemMax;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int got = 0;
  if (cudaOccupancyMaxActiveClusters(&got, (const void *)k_st_clusters<double, 7, false>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    got = 0;
  }
  return slots[cl] = got > 0 ? got : std::max(1, sm_count() / cl / 2);
}

// Filters n columns (each of which has a plan) in launches of up to kClCols
// clusters; a launch's operators have masks of one type.  Larger clusters make
// a column faster and let fewer run at once: of the sizes every column fits,
// the launch takes the one whose columns, each starting where a cluster is
// free first, are done soonest.  (Sixteen operators of 1,000 to 17,000 rows,
// degrees 11 to 338: with 8 blocks all run at once and the longest takes 620
// us; with 16 it takes 400 and the others fit beside it.)
template <class VT>
int cl_many(int n, const ClMany *cols) {
  const int most = cl_many_most(sizeof(VT));
  for (int c0 = 0, nc; c0 < n; c0 += nc) {
    nc = 1;
    const int mb = st_mask_bytes(cols[c0].A->st_d);
    while (nc < kClCols && c0 + nc < n && st_mask_bytes(cols[c0 + nc].A->st_d) == mb) ++nc;
    int cl = 0;
    double best = 0.0;
    for (int t = 1; t <= most; t *= 2) {
      std::vector<double> busy((size_t)std::min(nc, cl_slots(t)), 0.0);
      double end = 0.0;
      bool fits = true;
      for (int i = 0; i < nc && fits; ++i) {
        const ClMany &c = cols[c0 + i];
        const ClPlan P = cl_plan_many(c.A, sizeof(VT), t);
        fits = P.cl > 0;
        auto slot = std::min_element(busy.begin(), busy.end());
        *slot += c.deg * cl_degree_us(c.A, P);
        end = std::max(end, *slot);
      }
      if (fits && (!cl || end < best)) {
        cl = t;
        best = end;
      }
    }
    if (!cl) return fail(EVSLCU_ERR_ARG, "cluster filter: a column does not fit");
    StTab tab;
    int D = 5, T = 0;
    size_t smem = 0;
    bool one = true;
    for (int i = 0; i < nc; ++i) D = std::max(D, st_width(cols[c0 + i].A->st_d));
    for (int i = 0; i < nc; ++i) {
      const ClMany &c = cols[c0 + i];
      const ClPlan P = cl_plan_many(c.A, sizeof(VT), cl);
      cl_column(tab.c[i], c.A, c.deg, c.cc, c.dd, c.x, c.y, P, st_width(c.A->st_d));
      tab.c[i].mu = c.mu;
      T = std::max(T, P.T);
      // (a plan of one row per thread has no room for the masks)
      smem = std::max(smem, P.smem + (P.R == P.T ? (size_t)P.R * mb : 0));
      one = one && P.R == P.T;
    }
    const int rc = D == 5   ? cl_launch_many<VT, 5>(nc, tab, cl, T, smem, one)
                   : D == 7 ? cl_launch_many<VT, 7>(nc, tab, cl, T, smem, one)
                            : cl_launch_many<VT, 9>(nc, tab, cl, T, smem, one);
    if (rc) return rc;
  }
  return 0;
}

// Whether n columns of A go to clusters rather than to one launch per degree,
// by the time of a degree of all of them: cl_degree_us, or for k_st_cols 2.2 us
// a launch plus 6.3 (FP32: 3.6) us per million rows, as measured.
bool cl_columns_pay(const evslcu_mat *A, size_t vb, int n, double *us = nullptr) {
  const double step = 2.2 + (vb == 8 ? 6.3e-6 : 3.6e-6) * (double)A->n * n;
  if (us) *us = step;
  if (A->st_d > kClMaxD || g_cl_force < 0) return false;
  const int most = cl_many_most(vb);
  double cluster = 0.0;
  for (int t = 1; t <= most; t *= 2) {
    const ClPlan P = cl_plan_many(A, vb, t);
    if (!P.cl) continue;
    const double c = std::ceil((double)n / cl_slots(t)) * cl_degree_us(A, P);
    if (cluster == 0.0 || c < cluster) cluster = c;
  }
  if (cluster == 0.0) return false;
  if (us) *us = std::min(step, cluster);
  return g_cl_force > 0 || cluster < step;
}

template <class VT, int D>
int st_cols_launch(const evslcu_mat *A, int na, const StStepCols<VT> &C, int k) {
  const StArg<VT, D> S = st_arg<VT, D>(A);
  const bool two = A->n >= kStTwoRows || (sizeof(VT) == 4 && st_over_one_wave((long long)A->n * na));
  const StMarch M = st_march(A->n, A->st_span, D <= 9 && S.center && S.off[0] == -S.off[D - 1], two);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((M.cols + kThreads - 1) / kThreads, na);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = stream();
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  constexpr int J2 = D <= 9 ? 2 : 1;
  auto fn = M.J == 2 ? (k == 1 ? k_st_cols<VT, D, J2, true> : k_st_cols<VT, D, J2, false>)
                     : (k == 1 ? k_st_cols<VT, D, 1, true> : k_st_cols<VT, D, 1, false>);
  cudaError_t e = cudaLaunchKernelEx(&cfg, fn, S, M, C, k);
  if (e != cudaSuccess) return fail(EVSLCU_ERR_CUDA, "stencil filter launch failed: %s", cudaGetErrorString(e));
  EVSLCU_LAUNCH_CHECK("k_st_cols");
  return 0;
}

// Bytes of recurrence vectors that a group of columns may have at once: they
// stay in L2 from degree to degree.  (8 FP64 columns of 343 thousand rows, 100
// degrees: 2.59 ms in groups of 17 MB, 1.98 of 33, 1.82 of 64, 1.66 in one of 88;
// KPM of 10^6 rows gains up to 64 MB and loses 3% at 100.)
constexpr size_t kStColsBytes = (size_t)90 << 20;

// nc (at most kStCols) columns of A, one launch per degree; work: 4 vectors of
// n VT per column.
template <class VT>
int st_cols_group(const evslcu_mat *A, int nc, const ClMany *cols, VT *work) {
  const size_t n = (size_t)A->n;
  int order[kStCols], from[kStCols] = {};
  for (int i = 0; i < nc; ++i) order[i] = i;
  std::stable_sort(order, order + nc, [&](int p, int q) { return cols[p].deg > cols[q].deg; });
  constexpr bool F32 = sizeof(VT) == 4;
  if constexpr (F32) {
    for (int i = 0; i < nc; ++i) {
      k_st_float<<<grid_for(A->n), kThreads, 0, stream()>>>(A->n, cols[i].x, (float *)work + (size_t)(4 * i + 2) * n);
      EVSLCU_LAUNCH_CHECK("k_st_float");
    }
  }
  int active = nc;
  StStepCols<VT> C;
  memset(&C, 0, sizeof(C));
  for (int k = 1; k <= cols[order[0]].deg; ++k) {
    while (cols[order[active - 1]].deg < k) --active;
    for (int a = 0; a < active; ++a) {
      const int i = order[a];
      const ClMany &c = cols[i];
      VT *W[2] = {work + (size_t)(4 * i) * n, work + (size_t)(4 * i + 1) * n};
      const VT *x0;
      VT *y;
      if constexpr (F32) {
        x0 = work + (size_t)(4 * i + 2) * n;
        y = work + (size_t)(4 * i + 3) * n;
      } else {
        x0 = c.x;
        y = c.y;
      }
      StStepCol<VT> &I = C.c[a];
      I.vk = (k == 1) ? x0 : W[(k - 2) % 2];
      I.vkm1 = (k == 1) ? nullptr : ((k == 2) ? x0 : W[(k - 1) % 2]);
      I.out = W[(k - 1) % 2];
      I.y = y;
      I.yd = k == c.deg ? c.y : nullptr;
      I.mu = c.mu;
      I.t = (VT)((k == 1) ? 1.0 / c.dd : 2.0 / c.dd);
      I.ncc = (VT)(-c.cc);
      I.from = from[i];
      I.flush = k == c.deg || k - from[i] == 2;
      if (I.flush) from[i] = k + 1;
    }
    int rc;
    switch (st_width(A->st_d)) {
      case 5: rc = st_cols_launch<VT, 5>(A, active, C, k); break;
      case 7: rc = st_cols_launch<VT, 7>(A, active, C, k); break;
      case 9: rc = st_cols_launch<VT, 9>(A, active, C, k); break;
      case 16: rc = st_cols_launch<VT, 16>(A, active, C, k); break;
      default: rc = st_cols_launch<VT, 32>(A, active, C, k); break;
    }
    if (rc) return rc;
  }
  return 0;
}

// The KPM recurrence of nvec probes on clusters; *done stays false when the
// operator is too large.  The plan follows from n alone, so that a probe's sums
// do not depend on the others.
template <int D>
int kpm_cluster(const evslcu_mat *A, int steps, int nvec, const double *probes, double ctr, double wid, double *raw,
                bool *done) {
  static int most = 0, dev = -1;  // most blocks per cluster, as cl_max1
  if (!most || dev != lib_device()) {
    const void *fn1 = (const void *)k_st_kpm_cluster<D, true>, *fn2 = (const void *)k_st_kpm_cluster<D, false>;
    most = std::min(cl_limit(fn1, cl_threads(0, true)), cl_limit(fn2, cl_threads(0, false)));
    dev = lib_device();
  }
  ClPlan P;
  for (int cl = 1; cl <= most; cl *= 2) {
    const ClPlan Q = cl_plan(A->n, A->st_reach, A->st_d, sizeof(double), cl, 0);
    if (Q.cl) P = Q;
    if (Q.cl && Q.R == Q.T) break;  // the smallest cluster with one row per thread, else the largest
  }
  if (!P.cl || (g_cl_force == 0 && P.R > (A->st_d <= 5 ? kClMostRows5 : kClMostRows9))) return 0;
  int *err = cl_err();
  if (!err) return fail(EVSLCU_ERR_NOMEM, "KPM: out of pinned host memory");
  StCol C;
  cl_column(C, A, steps, ctr, wid, probes, nullptr, P, st_width(A->st_d));
  const size_t count = (size_t)steps * 3 * nvec;
  double *part = (double *)evslcu_malloc(sizeof(double) * count * P.cl);
  if (!part) return EVSLCU_ERR_NOMEM;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(P.cl * nvec);
  cfg.blockDim = dim3(P.T);
  cfg.dynamicSmemBytes = P.smem;
  cfg.stream = stream();
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = P.cl;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = P.R == P.T ? cudaLaunchKernelEx(&cfg, k_st_kpm_cluster<D, true>, C, part, nvec, g_cl_polls, err)
                             : cudaLaunchKernelEx(&cfg, k_st_kpm_cluster<D, false>, C, part, nvec, g_cl_polls, err);
  int rc = e == cudaSuccess ? 0 : fail(EVSLCU_ERR_CUDA, "KPM cluster launch failed: %s", cudaGetErrorString(e));
  count_launch();
  if (!rc) rc = check_launch("k_st_kpm_cluster");
  if (!rc) {
    // (the third sum exists at the first step only; its other places are not read)
    k_st_kpm_cl_sum<<<grid_for((long long)count), kThreads, 0, stream()>>>((int)count, P.cl, part, raw);
    count_launch();
    rc = check_launch("k_st_kpm_cl_sum");
  }
  evslcu_free(part);
  *done = true;
  return rc;
}

template <int D>
int kpm_steps(const evslcu_mat *A, int steps, int nvec, const double *probes, double ctr, double wid, double *raw) {
  const StArg<double, D> S = st_arg<double, D>(A);
  const StMarch M = st_march(A->n, A->st_span, D <= 9 && S.center && S.off[0] == -S.off[D - 1], A->n >= kStTwoRows);
  const size_t n = (size_t)A->n;
  const int grid = (M.cols + kThreads - 1) / kThreads;
  const int group = (int)std::max<size_t>(1, std::min<size_t>((size_t)nvec, kStColsBytes / (16 * n)));
  const int ng = (nvec + group - 1) / group, G = (nvec + ng - 1) / ng;
  const int chunk = std::min(steps, 16);  // steps whose sums are added up together
  const size_t n_part = std::max((size_t)chunk * 3 * G * grid, (size_t)G * kNormBlocks);
  double *w = (double *)evslcu_malloc(sizeof(double) * (2 * n * G + n_part));
  if (!w) return EVSLCU_ERR_NOMEM;
  double *part = w + 2 * n * G;
  constexpr int J2 = D <= 9 ? 2 : 1;
  int rc = 0;
  for (int p0 = 0; p0 < nvec && !rc; p0 += G) {
    const int nb = std::min(G, nvec - p0);
    // V[0] starts as the unit probes; w_k+1 takes the place of w_k-1
    double *V[2] = {w, w + n * nb};
    const double *x = probes + (size_t)p0 * n;
    k_st_sumsq<<<dim3(kNormBlocks, nb), kThreads, 0, stream()>>>(A->n, x, part);
    k_st_unit<<<dim3(std::min(grid_for(A->n), 1024), nb), kThreads, 0, stream()>>>(A->n, x, part, V[0]);
    count_launch(2);
    rc = check_launch("k_st_unit");
    for (int k = 0; k < steps && !rc; ++k) {
      const double t = (k == 0 ? 1.0 : 2.0) / wid;
      double *const pk = part + (size_t)(k % chunk) * 3 * nb * grid;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(grid, nb);
      cfg.blockDim = dim3(kThreads);
      cfg.stream = stream();
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      // the first step after the scaling, or after sums that still read the
      // buffer, waits for the whole launch before it
      attr[0].val.programmaticStreamSerializationAllowed = k % chunk != 0;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      auto fn = M.J == 2 ? (k == 0 ? k_st_kpm<D, J2, true> : k_st_kpm<D, J2, false>)
                         : (k == 0 ? k_st_kpm<D, 1, true> : k_st_kpm<D, 1, false>);
      cudaError_t e = cudaLaunchKernelEx(&cfg, fn, S, M, (const double *)V[k % 2], (const double *)V[(k + 1) % 2],
                                         V[(k + 1) % 2], t, -ctr, pk);
      rc = e == cudaSuccess ? 0 : fail(EVSLCU_ERR_CUDA, "KPM launch failed: %s", cudaGetErrorString(e));
      count_launch();
      if (!rc) rc = check_launch("k_st_kpm");
      if (!rc && (k % chunk == chunk - 1 || k == steps - 1)) {
        const int k0 = k - k % chunk, cnt = k % chunk + 1;
        // (the third sum exists at the first step only; its other places are
        // not read afterwards)
        k_st_kpm_sum<<<dim3(nb, 3 * cnt), kThreads, 0, stream()>>>(grid, part, raw + (size_t)k0 * 3 * nvec + p0, nvec);
        count_launch();
        rc = check_launch("k_st_kpm_sum");
      }
    }
  }
  evslcu_free(w);
  return rc;
}

template <int D>
int kpm_d(const evslcu_mat *A, int steps, int nvec, const double *probes, double ctr, double wid, double *raw) {
  if constexpr (D <= kClMaxD) {
    bool done = false;
    if (g_cl_force >= 0) {
      const int rc = kpm_cluster<D>(A, steps, nvec, probes, ctr, wid, raw, &done);
      if (rc || done) return rc;
    }
  }
  return kpm_steps<D>(A, steps, nvec, probes, ctr, wid, raw);
}

}  // namespace

namespace evslcu {

// Merges the dictionary's patterns into one list of (offset, value) entries;
// leaves M->st_d at 0 when a pattern's offsets do not increase, a value is not
// finite or the list has more than kStMax entries.
int stencil_build(evslcu_mat *M) {
  if (!M->pat_id || M->npat <= 0) return 0;
  const size_t hb = pat_hdr_bytes(M->npat);
  std::vector<int2> hdr(M->npat);
  std::vector<double2> ent(std::max(M->pat_entries, 1));
  int rc = evslcu_d2h(hdr.data(), M->pat_table, sizeof(int2) * M->npat);
  if (!rc && M->pat_entries > 0)
    rc = evslcu_d2h(ent.data(), (const char *)M->pat_table + hb, sizeof(double2) * M->pat_entries);
  if (rc) return rc;
  struct Key {
    int off;
    unsigned long long bits;
    bool operator<(const Key &o) const { return off != o.off ? off < o.off : bits < o.bits; }
  };
  std::map<Key, int> list;
  auto key_of = [&](int i) {
    Key k;
    long long ob;
    memcpy(&ob, &ent[i].y, sizeof(ob));
    memcpy(&k.bits, &ent[i].x, sizeof(k.bits));
    k.off = (int)ob;
    return k;
  };
  for (const int2 &h : hdr)
    for (int j = 0; j < h.y; ++j) {
      const Key k = key_of(h.x + j);
      if (!std::isfinite(ent[h.x + j].x)) return 0;  // 0 * inf would reach rows without the entry
      if (j > 0 && k.off <= key_of(h.x + j - 1).off) return 0;
      list.emplace(k, 0);
      if ((int)list.size() > kStMax) return 0;
    }
  if (list.empty()) return 0;
  int d = 0, reach = 0, span = 0, f32 = 1;
  for (auto &e : list) {
    e.second = d;
    M->st_off[d] = e.first.off;
    memcpy(&M->st_val[d], &e.first.bits, sizeof(double));
    if (!std::isfinite((float)M->st_val[d])) f32 = 0;
    reach = std::max(reach, std::abs(e.first.off));
    span = std::max(span, e.first.off);
    ++d;
  }
  std::vector<unsigned> mask(M->npat, 0u);
  for (int p = 0; p < M->npat; ++p)
    for (int j = 0; j < hdr[p].y; ++j) mask[p] |= 1u << list[key_of(hdr[p].x + j)];
  unsigned *tab = (unsigned *)evslcu_malloc(sizeof(unsigned) * M->npat);
  void *dm = evslcu_malloc((size_t)st_mask_bytes(d) * (size_t)M->n);
  rc = (tab && dm) ? evslcu_h2d(tab, mask.data(), sizeof(unsigned) * M->npat) : EVSLCU_ERR_NOMEM;
  if (!rc) {
    const int g = grid_for(M->n);
    switch (st_mask_bytes(d)) {
      case 1: k_st_mask<<<g, kThreads, 0, stream()>>>(M->n, M->pat_id, tab, (uint8_t *)dm); break;
      case 2: k_st_mask<<<g, kThreads, 0, stream()>>>(M->n, M->pat_id, tab, (uint16_t *)dm); break;
      default: k_st_mask<<<g, kThreads, 0, stream()>>>(M->n, M->pat_id, tab, (uint32_t *)dm); break;
    }
    count_launch();
    rc = check_launch("k_st_mask");
    // the filter kernels read the masks before they wait for the launch ahead
    if (!rc) rc = evslcu_sync();
  }
  evslcu_free(tab);
  if (rc) {
    evslcu_free(dm);
    return rc == EVSLCU_ERR_NOMEM ? 0 : rc;  // the stencil form is optional
  }
  M->st_mask = dm;
  M->st_reach = reach;
  M->st_span = span;
  M->st_f32 = f32;
  M->st_plain = (d == 5 || d == 7 || d == 9) && M->pat_maxlen == d;
  M->st_d = d;
  return 0;
}

void stencil_free(evslcu_mat *M) {
  evslcu_free(M->st_mask);
  M->st_mask = nullptr;
  M->st_d = M->st_plain = 0;
}

// Y(:, c) = A X(:, c) for m columns (1 <= m <= 65535) of a matrix that
// stencil_spmv_ok takes.
int stencil_spmv(const evslcu_mat *A, const double *X, double *Y, int m) {
  const dim3 g(grid_for(A->n), m);
  switch (st_width(A->st_d)) {
    case 5: k_st_spmv<5><<<g, kThreads, 0, stream()>>>(st_arg<double, 5>(A), X, Y, A->n); break;
    case 7: k_st_spmv<7><<<g, kThreads, 0, stream()>>>(st_arg<double, 7>(A), X, Y, A->n); break;
    case 9: k_st_spmv<9><<<g, kThreads, 0, stream()>>>(st_arg<double, 9>(A), X, Y, A->n); break;
    default: k_st_spmv<16><<<g, kThreads, 0, stream()>>>(st_arg<double, 16>(A), X, Y, A->n); break;
  }
  EVSLCU_LAUNCH_CHECK("k_st_spmv");
  return 0;
}

int stencil_error() {
  if (!g_cl_err || !*(volatile int *)g_cl_err) return 0;
  *(volatile int *)g_cl_err = 0;
  return fail(EVSLCU_ERR_TIMEOUT, "a wait of the filter kernel did not complete within its bound");
}

void set_cluster_wait_limit(unsigned long long polls) {
  g_cl_polls = (polls == 0 || polls > (unsigned long long)kClPolls) ? kClPolls : (int)polls;
}

bool stencil_ok(const evslcu_mat *M) { return M->st_d > 0 && M->use_pat && M->kernel == 0; }

// Whether filters take the merged stencil untimed: 5, 7 or 9
// entries, all of them in some row.  These widths are compiled, and full rows
// skip their masks; it was the fastest at every size measured (10^4 to 4.1
// million rows, 1 to 16 columns, both precisions).  Where rows take only part
// of a longer list, as with coefficients that vary, or the list is padded to
// the next width, each row does the whole list's loads and multiplications, and
// the stencil is one of the variants that a first filter times.  Us a degree on
// 10^6 rows, fastest dictionary kernel / stencil: 5 points with 2 diagonal
// values 6.80 / 6.76, with 5 6.92 / 8.16, with 6 sets of coefficients (30
// entries) 6.89 / 23.9, 13 points 11.7 / 11.5, 27 points 21.6 / 25.6; on 10^4
// rows 3.64 / 0.86, 2.66 / 0.94, 2.79 / 2.68, 3.61 / 2.68, 5.28 / 2.78.
bool stencil_plain(const evslcu_mat *M) { return stencil_ok(M) && M->st_plain; }

// Whether products take it: a list of 5 to 16 entries that some row has all of
// (us for 16 columns, dictionary / stencil: 10^6 rows, 3 points 82.8 / 89.5, 5
// points 93.6 / 94.7, 9 points 118 / 106, 13 points 165 / 154, 27 points 326 /
// 590, 5 points with 6 sets of coefficients 93 / 540; 10^5 rows, 13 points 35.6
// / 26.2).
bool stencil_spmv_ok(const evslcu_mat *M) {
  return stencil_ok(M) && M->st_d >= 5 && M->st_d <= 16 && M->st_d == M->pat_maxlen;
}

// Whether KPM runs on it: the dictionary's kernel reads the probes interleaved
// and pays for each launch and reduction, so the list may be up to four times
// as wide as a row (16 probes, us a step on 10^6 rows, dictionary / stencil: 30
// entries in rows of 5 228 / 308, 28 in rows of 7 249 / 314, 10 in 5 228 / 167,
// 26 in 13 539 / 322), and any width on small operators (10^5 rows, 30 in 5 32 /
// 33, 10^4 14.3 / 7.3).
bool stencil_kpm_ok(const evslcu_mat *M) {
  return stencil_ok(M) && (M->n <= 65536 || st_width(M->st_d) <= 4 * M->pat_maxlen);
}

// Microseconds per degree of run(), a filter of degree kTimeDeg.
constexpr int kTimeDeg = 24;
template <class F>
static int time_degrees(F &&run, float *us) {
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  float ms = 0.0f;
  int rc = run();
  if (!rc && (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess))
    rc = fail(EVSLCU_ERR_CUDA, "stencil timing: no events");
  if (!rc) cudaEventRecord(e0, stream());
  if (!rc) rc = run();
  if (!rc) cudaEventRecord(e1, stream());
  if (!rc) rc = evslcu_sync();
  if (!rc) cudaEventElapsedTime(&ms, e0, e1);
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  *us = 1e3f * ms / kTimeDeg;
  return rc;
}

// The filter of one vector, timed on zero vectors; *us stays 0 without memory.
int stencil_time(const evslcu_mat *A, float *us) {
  const size_t n = (size_t)A->n;
  *us = 0.0f;
  double *w = (double *)evslcu_malloc(sizeof(double) * 4 * n);
  if (!w) return 0;
  const std::vector<double> mu((size_t)kTimeDeg + 1, 0.0);
  int rc = evslcu_memset(w, 0, sizeof(double) * 4 * n);
  if (!rc)
    rc = time_degrees(
        [&] { return stencil_chebav(A, mu.data(), kTimeDeg, 0.0, 1.0, w, w + n, w + 2 * n, nullptr); }, us);
  evslcu_free(w);
  return rc;
}

// The filter of ncols (at most kStCols) columns, likewise.
int stencil_columns_time(const evslcu_mat *A, int fp32, int ncols, float *us) {
  const size_t n = (size_t)A->n, work = evslcu_filter_columns_work(A->n, fp32, ncols);
  *us = 0.0f;
  double *w = (double *)evslcu_malloc(sizeof(double) * n * (ncols + 1) + work);
  if (!w) return 0;
  const std::vector<double> mu((size_t)kTimeDeg + 1, 0.0);
  std::vector<evslcu_filter_col> cols((size_t)ncols);
  std::vector<size_t> off((size_t)ncols);
  for (int c = 0; c < ncols; ++c) cols[c] = evslcu_filter_col{mu.data(), kTimeDeg, 0.0, 1.0, w, w + n * (c + 1)};
  int rc = evslcu_memset(w, 0, sizeof(double) * n);
  double *dmu = rc ? nullptr : stencil_columns_mu(ncols, cols.data(), off.data(), &rc);
  if (!rc)
    rc = time_degrees(
        [&] { return stencil_columns(A, fp32, ncols, cols.data(), dmu, off.data(), w + n * (ncols + 1)); }, us);
  evslcu_free(dmu);
  evslcu_free(w);
  return rc;
}

int stencil_chebav(const evslcu_mat *A, const double *mu, int deg, double cc, double dd, const double *v, double *y,
                   double *work, const evslcu_cheb_epi *epi) {
  const size_t n = (size_t)A->n;
  const double t1 = 1.0 / dd, t2 = 2.0 / dd, ncc = -cc;
  bool done = false;
  const int crc = cl_chebav(A, mu, deg, cc, dd, v, y, epi, &done);
  if (crc || done) return crc;
  double *W[2] = {work, work + n};
  int from = 0;  // first degree whose term y does not hold yet
  for (int k = 1; k <= deg; ++k) {
    const double *vk = (k == 1) ? v : W[(k - 2) % 2];
    const double *vkm1 = (k == 1) ? nullptr : ((k == 2) ? v : W[(k - 1) % 2]);
    StY<double> Y{0, 0, 0.0, 0.0, 0.0};
    if (k == deg || k - from == 2) {
      Y.terms = k - from + 1;
      Y.init = from == 0;
      Y.c0 = mu[k];
      if (Y.terms >= 2) Y.c1 = mu[k - 1];
      if (Y.terms == 3) Y.c2 = mu[k - 2];
      from = k + 1;
    }
    const int rc = st_step_any(A, k == 1, vk, vkm1, W[(k - 1) % 2], y, (k == 1) ? t1 : t2, ncc, Y, k == deg,
                               k == deg ? epi : nullptr);
    if (rc) return rc;
  }
  return 0;
}

// Raw sums of the KPM recurrence (sparse.cu, kpm_dots_doubling): raw[(k * 3 +
// sum) * nvec + probe], on the device.
int stencil_kpm(const evslcu_mat *A, int steps, int nvec, const double *probes, double ctr, double wid, double *raw) {
  switch (st_width(A->st_d)) {
    case 5: return kpm_d<5>(A, steps, nvec, probes, ctr, wid, raw);
    case 7: return kpm_d<7>(A, steps, nvec, probes, ctr, wid, raw);
    case 9: return kpm_d<9>(A, steps, nvec, probes, ctr, wid, raw);
    case 16: return kpm_d<16>(A, steps, nvec, probes, ctr, wid, raw);
    default: return kpm_d<32>(A, steps, nvec, probes, ctr, wid, raw);
  }
}

// Whether every column's y may be written while other columns' x are read:
// y's share no memory with x's, except that a column may be filtered in place.
// (One FP64 launch per degree reads x at degrees 1 and 2, a row's own value
// last, and writes y from degree 2 on, or at degree 1 when that is all; the
// other kernels copy x first.)
static bool columns_apart(int n, int fp32, int ncols, const evslcu_filter_col *cols) {
  std::vector<std::pair<uintptr_t, int>> y((size_t)ncols);
  for (int c = 0; c < ncols; ++c) y[c] = {(uintptr_t)cols[c].y, c};
  std::sort(y.begin(), y.end());
  const uintptr_t bytes = sizeof(double) * (uintptr_t)n;
  for (int c = 0; c < ncols; ++c) {
    const uintptr_t x = (uintptr_t)cols[c].x;
    auto it = std::upper_bound(y.begin(), y.end(), std::make_pair(x > bytes ? x - bytes : 0, ncols));
    for (; it != y.end() && it->first < x + bytes; ++it)
      if (it->first != x || it->second != c || (!fp32 && cols[c].deg == 1)) return false;
  }
  return true;
}

// Whether filter_columns takes these columns: a merged stencil, every degree
// at least 1, values finite in the columns' precision (0 * inf would reach rows
// without the entry), and (once the vectors are known) no y in another column's
// way.
bool stencil_columns_ok(const evslcu_mat *A, int fp32, int ncols, const evslcu_filter_col *cols, bool vectors) {
  if (!stencil_ok(A) || (fp32 && !A->st_f32)) return false;
  for (int c = 0; c < ncols; ++c)
    if (cols[c].deg < 1) return false;
  return !vectors || columns_apart(A->n, fp32, ncols, cols);
}

// Device copy of the columns' coefficients, one after another (columns that
// share an array share its copy); off: each column's first.
double *stencil_columns_mu(int ncols, const evslcu_filter_col *cols, size_t *off, int *err) {
  size_t total = 0;
  for (int c = 0; c < ncols; ++c) {
    const bool same = c > 0 && cols[c].mu == cols[c - 1].mu && cols[c].deg == cols[c - 1].deg;
    off[c] = same ? off[c - 1] : total;
    if (!same) total += (size_t)cols[c].deg + 1;
  }
  std::vector<double> h(total);
  for (int c = 0; c < ncols; ++c) memcpy(h.data() + off[c], cols[c].mu, sizeof(double) * ((size_t)cols[c].deg + 1));
  double *d = (double *)evslcu_malloc(sizeof(double) * total);
  *err = d ? evslcu_h2d_async(d, h.data(), sizeof(double) * total)
           : fail(EVSLCU_ERR_NOMEM, "filter coefficients: out of device memory");
  if (*err) {
    evslcu_free(d);
    return nullptr;
  }
  return d;
}

// The columns' filters; dmu, off from stencil_columns_mu.  work: 4 vectors of
// n values for min(ncols, 16) columns.
int stencil_columns(const evslcu_mat *A, int fp32, int ncols, const evslcu_filter_col *cols, const double *dmu,
                    const size_t *off, void *work) {
  std::vector<ClMany> many((size_t)ncols);
  for (int c = 0; c < ncols; ++c)
    many[c] = ClMany{A, dmu + off[c], cols[c].deg, cols[c].cc, cols[c].dd, cols[c].x, cols[c].y};
  const size_t vb = fp32 ? sizeof(float) : sizeof(double);
  if (cl_columns_pay(A, vb, ncols)) return fp32 ? cl_many<float>(ncols, many.data()) : cl_many<double>(ncols, many.data());
  const size_t per = 4 * vb * (size_t)A->n;
  const int group = (int)std::max<size_t>(1, std::min<size_t>(kStCols, kStColsBytes / per));
  // groups of nearly equal size
  const int ng = (ncols + group - 1) / group;
  for (int g = 0, c0 = 0; g < ng; ++g) {
    const int nc = (ncols - c0 + (ng - g) - 1) / (ng - g);
    const int rc = fp32 ? st_cols_group<float>(A, nc, many.data() + c0, (float *)work)
                        : st_cols_group<double>(A, nc, many.data() + c0, (double *)work);
    if (rc) return rc;
    c0 += nc;
  }
  return 0;
}

// Microseconds of a degree of n columns, from those figures.
double stencil_step_us(const evslcu_mat *A, int fp32, int n) {
  double us = 0.0;
  cl_columns_pay(A, fp32 ? sizeof(float) : sizeof(double), n, &us);
  return us;
}

// Takes the columns of an engine's batch that fit a cluster out of it: filters
// them and marks them in done.
int stencil_batch(int ncols, const evslcu_batch_col *cols, unsigned char *done) {
  std::vector<ClMany> many;
  if (g_cl_force >= 0)
    for (int c = 0; c < ncols; ++c) {
      const evslcu_batch_col &b = cols[c];
      if (!stencil_ok(b.A) || b.deg < 1 || !cl_columns_pay(b.A, sizeof(double), 1)) continue;
      many.push_back(ClMany{b.A, b.mu, b.deg, b.cc, b.dd, b.x, b.y});
      done[c] = 1;
    }
  if (many.empty()) return 0;
  // long filters first: a launch of more clusters than run at once ends sooner
  std::stable_sort(many.begin(), many.end(),
                   [](const ClMany &p, const ClMany &q) { return (double)p.deg * p.A->n > (double)q.deg * q.A->n; });
  std::stable_partition(many.begin(), many.end(), [](const ClMany &p) { return st_mask_bytes(p.A->st_d) == 1; });
  return cl_many<double>((int)many.size(), many.data());
}

}  // namespace evslcu

extern "C" {

int evslcu_set_stencil_cluster(int blocks) {
  if (blocks < -1 || blocks > 16 || (blocks > 0 && (blocks & (blocks - 1))))
    return fail(EVSLCU_ERR_ARG, "cluster blocks must be -1, 0 or a power of two up to 16");
  g_cl_force = blocks;
  return 0;
}

void evslcu_stencil_release(void) {
  evslcu_free(g_cl_mu);
  g_cl_mu = nullptr;
  g_cl_mu_cap = 0;
  if (g_cl_err) cudaFreeHost(g_cl_err);
  g_cl_err = nullptr;
}

}  // extern "C"
