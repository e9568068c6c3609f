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
//     seven timed): 3-D Laplacian of 10^6 rows 7.84 -> 6.30 us a degree, 343
//     thousand rows 4.57 -> 3.15, 10^4 rows 2.95 -> 2.4 (launch latency).
//   * k_st_cluster: every degree in one launch, for operators whose vectors
//     fit the shared memory of one thread-block cluster: 10^4 rows 2.4 -> 0.52.
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
};

// What a degree does to y: terms pending since y was last written (0: none
// now), their coefficients (c2 w_k-2 + c1 w_k-1 + c0 w_k), and whether y
// starts with the first of them.
struct StY {
  int terms, init;
  double c2, c1, c0;
};

// J > 1 needs a stencil whose first and last offsets are -S and +S around a
// diagonal entry in the middle (StArg::center).
template <int D, int J, bool FIRST, bool EPI>
__global__ void __launch_bounds__(kThreads, J == 2 ? 5 : D <= 9 ? 6 : 2)
    k_st_step(const __grid_constant__ StArg<double, D> A, StMarch M, const double *__restrict__ vk, const double *vkm1,
              double *out, double *y, double t, double ncc, StY Y, const double *__restrict__ zold, double nbeta,
              const double *__restrict__ dotv, double *part, unsigned int *ctr, double *dot_out) {
  __shared__ double sh[EPI ? kThreads / 32 : 1];
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
  // The masks never change, and v_k-1 was written two launches ago: that one
  // has completed once the previous launch has let this one start (it does so
  // after its own wait).
  unsigned m[J];
  double xm1[J];
  bool live[J];
  bool all = true;
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const int r = r0 + j * M.S;
    live[j] = r < A.n;
    m[j] = live[j] ? (unsigned)__ldg(A.mask + r) : 0u;
    xm1[j] = (!FIRST && live[j]) ? vkm1[r] : 0.0;
  }
#pragma unroll
  for (int j = 0; j < J; ++j) all = all && m[j] == A.full;
  all = __all_sync(0xffffffffu, all);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const double *xr = vk + r0;
  double acc[J], x[J], yo[J];
#pragma unroll
  for (int j = 0; j < J; ++j) yo[j] = (Y.terms && !Y.init && live[j]) ? y[r0 + j * M.S] : 0.0;
  if constexpr (J == 1) {
    acc[0] = 0.0;
    x[0] = 0.0;
    if (all) {
      double g[D];
#pragma unroll
      for (int e = 0; e < D; ++e) g[e] = __ldg(xr + A.off[e]);
#pragma unroll
      for (int e = 0; e < D; ++e) acc[0] = st_fmadd(A.val[e], g[e], acc[0]);
      x[0] = A.center ? g[D / 2] : __ldg(xr);
    } else {
      // an entry the row does not have adds -0: no change to any sum
      double g[D];
#pragma unroll
      for (int e = 0; e < D; ++e) g[e] = (m[0] >> e & 1u) ? __ldg(xr + A.off[e]) : st_zero(A.val[e]);
      if (live[0]) x[0] = __ldg(xr);
#pragma unroll
      for (int e = 0; e < D; ++e) acc[0] = st_fmadd(A.val[e], g[e], acc[0]);
    }
  } else {
    // p[j]: the value one S below row j; rows share it with their neighbours
    double p[J + 2], g[J][D];
    if (all) {
#pragma unroll
      for (int j = 0; j < J + 2; ++j) p[j] = __ldg(xr + (j - 1) * M.S);
#pragma unroll
      for (int j = 0; j < J; ++j)
#pragma unroll
        for (int e = 1; e < D - 1; ++e)
          if (e != D / 2) g[j][e] = __ldg(xr + j * M.S + A.off[e]);
#pragma unroll
      for (int j = 0; j < J; ++j) {
        double a = 0.0;
#pragma unroll
        for (int e = 0; e < D; ++e)
          a = st_fmadd(A.val[e], e == 0 ? p[j] : e == D / 2 ? p[j + 1] : e == D - 1 ? p[j + 2] : g[j][e], a);
        acc[j] = a;
      }
    } else {
#pragma unroll
      for (int j = 0; j < J + 2; ++j) {
        const bool have = j == 0 ? (m[0] & 1u) != 0 : j == J + 1 ? (m[J - 1] >> (D - 1) & 1u) != 0 : live[j == 0 ? 0 : j > J ? J - 1 : j - 1];
        p[j] = have ? __ldg(xr + (j - 1) * M.S) : 0.0;
      }
#pragma unroll
      for (int j = 0; j < J; ++j)
#pragma unroll
        for (int e = 1; e < D - 1; ++e)
          if (e != D / 2) g[j][e] = (m[j] >> e & 1u) ? __ldg(xr + j * M.S + A.off[e]) : 0.0;
#pragma unroll
      for (int j = 0; j < J; ++j) {
        double a = 0.0;
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
    double w = __dmul_rn(t, __dadd_rn(acc[j], __dmul_rn(ncc, x[j])));
    if (!FIRST) w = __dadd_rn(w, -xm1[j]);
    out[r] = w;
    if (Y.terms) {
      double yv = yo[j];
      if (Y.terms == 3) yv = Y.init ? __dmul_rn(Y.c2, xm1[j]) : __dadd_rn(yv, __dmul_rn(Y.c2, xm1[j]));
      if (Y.terms >= 2)
        yv = (Y.init && Y.terms == 2) ? __dmul_rn(Y.c1, x[j]) : __dadd_rn(yv, __dmul_rn(Y.c1, x[j]));
      yv = __dadd_rn(yv, __dmul_rn(Y.c0, w));
      if (EPI) {
        if (zold) yv = __dadd_rn(yv, __dmul_rn(nbeta, zold[r]));
        if (dotv) dsum += dotv[r] * yv;
      }
      y[r] = yv;
    }
  }
  if (EPI && dot_out) {
    const double b = block_sum(dsum, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = b;
    if (last_block(ctr)) {
      const double tot = reduce_partials(part, gridDim.x, ctr, sh);
      if (threadIdx.x == 0) *dot_out = tot;
    }
  }
}

// Two rows per thread where the grid still covers every SM's warps about
// once.  Measured, us a degree, 1 / 2 / 3 rows per thread: 125 thousand rows
// 2.58 / 2.57 / 2.77, 343 thousand 3.21 / 3.15 / 3.47, 10^6 (3-D) 6.51 / 6.30 /
// 6.82, 10^6 (2-D) 5.45 / 5.28 / 5.47, 4.1 million 29.1 / 25.5 / 26.3.
constexpr int kStTwoRows = 150000;

StMarch st_march(int n, int span, bool sym) {
  StMarch M;
  int J = n >= kStTwoRows ? 2 : 1;
  if (!sym || span < 1 || (long long)span * J > n || n > (1 << 29)) J = 1;
  M.S = J > 1 ? span : std::max(n, 1);
  M.J = J;
  const long long groups = ((long long)n + (long long)M.S * J - 1) / ((long long)M.S * J);
  M.cols = (int)(groups * M.S);
  M.magic = (unsigned)((1ull << 32) / (unsigned long long)M.S - (M.S == 1 ? 1 : 0));
  return M;
}

template <int D>
int st_step(const evslcu_mat *A, bool first, const double *vk, const double *vkm1, double *out, double *y, double t,
            double ncc, const StY &Y, const evslcu_cheb_epi *ep) {
  const StArg<double, D> S = st_arg<double, D>(A);
  const StMarch M = st_march(A->n, A->st_span, D <= 9 && S.center && S.off[0] == -S.off[D - 1]);
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
  cudaError_t e = cudaLaunchKernelEx(&cfg, fn, S, M, vk, vkm1, out, y, t, ncc, Y,
                                     epi ? ep->zold : nullptr, epi ? ep->nbeta : 0.0, epi ? ep->dotv : nullptr,
                                     partials(), counters() + CTR_CHEB, epi ? ep->dot_out : nullptr);
  if (e != cudaSuccess) return fail(EVSLCU_ERR_CUDA, "stencil filter launch failed: %s", cudaGetErrorString(e));
  EVSLCU_LAUNCH_CHECK("k_st_step");
  if (ep && !epi) return launch_lan_epi(A->n, ep, y);
  return 0;
}

int st_step_any(const evslcu_mat *A, bool first, const double *vk, const double *vkm1, double *out, double *y, double t,
                double ncc, const StY &Y, const evslcu_cheb_epi *ep) {
  switch (st_width(A->st_d)) {
    case 5: return st_step<5>(A, first, vk, vkm1, out, y, t, ncc, Y, ep);
    case 7: return st_step<7>(A, first, vk, vkm1, out, y, t, ncc, Y, ep);
    case 9: return st_step<9>(A, first, vk, vkm1, out, y, t, ncc, Y, ep);
    case 16: return st_step<16>(A, first, vk, vkm1, out, y, t, ncc, Y, ep);
    default: return st_step<32>(A, first, vk, vkm1, out, y, t, ncc, Y, ep);
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
// Waits for the phase of the given parity; false when the polls run out, or at
// once when another wait of the block has.
constexpr int kClPolls = 1 << 20;
__device__ __forceinline__ bool bar_wait(unsigned long long *bar, unsigned parity, int polls, const int *dead) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(bar);
  for (int i = 0; i < polls; ++i) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
    if (*(const volatile int *)dead) break;
  }
  return false;
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
// A wait that runs out of polls sets *err (the host's mapped flag) and `dead`:
// later waits of the block give up at once, and it stays until the blocks that
// may still send to it are done.
//
// ONE: at most one row per thread, whose w_k, w_k-1 and y stay in registers.
// The instruction count per row is what bounds a degree (a first version with
// its first / last / y tests inside the row loop took 130-190 instructions per
// 32 rows: 0.97 us a degree on 10^4 rows, 3.8 us on 94,800), so those cases
// are compiled apart.
template <class VT, int D, bool ONE, class MU>
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
  const int nit = ONE ? 1 : R / T;
  // bit `it`: the warp's rows of iteration `it` have every entry / read a halo
  unsigned fast = 0, edge = 0, m1 = 0;
  for (int it = 0, i = tid + (nit - 1) * T; it < nit; ++it, i = it == 1 ? tid : i + T) {
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
    if (!LAST && tid == 0 && expect && !*(volatile int *)&dead) bar_expect(bars + (k & 1), expect);
    if (!FIRST && edge && !bar_wait(bars + ((k - 1) & 1), (unsigned)((k - 2) >> 1) & 1u, polls, &dead)) {
      *(volatile int *)&dead = 1;
      *(volatile int *)err = 1;
    }
    const unsigned bk = (unsigned)((k & 1) * 8);
    unsigned fb = fast, eb = edge;
#pragma unroll 2
    for (int it = 0, i = tid + (nit - 1) * T; it < nit; ++it, i = it == 1 ? tid : i + T, fb >>= 1, eb >>= 1) {
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
  if (cl > 1 && dead) cluster_sync();  // nobody's memory goes away while others may still send to it
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
  }
}

// CAP >= 0: one cluster filters `one`, whose coefficients (up to CAP) come
// with the launch, or from the device when CAP is 0.  CAP -1: cluster q of
// the launch filters tab[q].
template <class VT, int D, int CAP, bool ONE>
__global__ void __launch_bounds__(cl_threads(CAP, ONE), 1)
    k_st_cluster(const StCol *__restrict__ tab, const __grid_constant__ StCol one,
                 const __grid_constant__ StMu<CAP> mus, int polls, int *err) {
  if constexpr (CAP > 0) {
    st_cluster_body<VT, D, ONE>(one, [&](int k) { return mus.v[k]; }, polls, err);
  } else if constexpr (CAP == 0) {
    const double *mup = one.mu;
    st_cluster_body<VT, D, ONE>(one, [&](int k) { return __ldg(mup + k); }, polls, err);
  } else {
    const StCol &I = tab[blockIdx.x / cluster_size()];
    const double *mup = I.mu;
    st_cluster_body<VT, D, ONE>(I, [&](int k) { return __ldg(mup + k); }, polls, err);
  }
}

// Blocks of the cluster, rows and shared memory of one column; cl 0: none fits.
struct ClPlan {
  int cl = 0, R = 0, T = 0, halo = 0, y_smem = 0;
  size_t smem = 0;
};
constexpr size_t kClSmemMax = 225 * 1024;

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
template <class VT, int D, int CAP, bool ONE>
int cl_max1() {
  static int m = 0;
  if (m) return m;
  const void *fn = (const void *)k_st_cluster<VT, D, CAP, ONE>;
  m = -1;
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClSmemMax) != cudaSuccess) {
    cudaGetLastError();
    return m;
  }
  const bool wide = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
  if (!wide) cudaGetLastError();
  for (int cl = wide ? 16 : 8; cl >= 1; cl /= 2) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cl);
    cfg.blockDim = dim3(cl_threads(CAP, ONE));
    cfg.dynamicSmemBytes = kClSmemMax;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cl;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int got = 0;
    if (cudaOccupancyMaxActiveClusters(&got, fn, &cfg) == cudaSuccess && got >= 1) {
      m = cl;
      break;
    }
    cudaGetLastError();
  }
  return m;
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

template <class VT, int D, int CAP>
int cl_max() {
  return std::min(cl_max1<VT, D, CAP, true>(), cl_max1<VT, D, CAP, false>());
}

template <class VT, int D, int CAP>
int cl_launch(int ncols, const StCol *tab, const StCol &one, const double *mu, const ClPlan &P) {
  int *err = cl_err();  // same address on the device (unified addressing)
  if (!err) return fail(EVSLCU_ERR_NOMEM, "cluster filter: out of pinned host memory");
  StMu<CAP> mus;
  if (CAP > 0) memcpy(mus.v, mu, sizeof(double) * (size_t)(one.deg + 1));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(P.cl * ncols);
  cfg.blockDim = dim3(P.T);
  cfg.dynamicSmemBytes = P.smem;
  cfg.stream = stream();
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = P.cl;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = P.R == P.T ? cudaLaunchKernelEx(&cfg, k_st_cluster<VT, D, CAP, true>, tab, one, mus, kClPolls, err)
                           : cudaLaunchKernelEx(&cfg, k_st_cluster<VT, D, CAP, false>, tab, one, mus, kClPolls, err);
  if (e != cudaSuccess) return fail(EVSLCU_ERR_CUDA, "cluster filter launch failed: %s", cudaGetErrorString(e));
  EVSLCU_LAUNCH_CHECK("k_st_cluster");
  return 0;
}

template <class VT, int CAP>
int cl_most(int d) {
  return d <= 5 ? cl_max<VT, 5, CAP>() : d <= 7 ? cl_max<VT, 7, CAP>() : cl_max<VT, 9, CAP>();
}
// `one`: the column, or for a table its widest stencil.
template <class VT, int CAP>
int cl_launch_d(int ncols, const StCol *tab, const StCol &one, const double *mu, const ClPlan &P) {
  return one.d <= 5   ? cl_launch<VT, 5, CAP>(ncols, tab, one, mu, P)
         : one.d <= 7 ? cl_launch<VT, 7, CAP>(ncols, tab, one, mu, P)
                      : cl_launch<VT, 9, CAP>(ncols, tab, one, mu, P);
}

void cl_column(StCol &C, const evslcu_mat *A, int deg, double cc, double dd, const double *x, double *y,
               const ClPlan &P) {
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
  const int D = st_width(A->st_d);
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
  cl_column(C, A, deg, cc, dd, v, y, P);
  if (epi) {
    C.zold = epi->zold;
    C.nbeta = epi->nbeta;
    C.dotv = epi->dotv;
    C.dot_out = epi->dot_out;
  }
  *done = true;
  if (deg < 64) return cl_launch_d<double, 64>(1, nullptr, C, mu, P);
  if (deg < 512) return cl_launch_d<double, 512>(1, nullptr, C, mu, P);
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
  return cl_launch_d<double, 0>(1, nullptr, C, nullptr, P);
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
  int d = 0, reach = 0, span = 0;
  for (auto &e : list) {
    e.second = d;
    M->st_off[d] = e.first.off;
    memcpy(&M->st_val[d], &e.first.bits, sizeof(double));
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
  }
  evslcu_free(tab);
  if (rc) {
    evslcu_free(dm);
    return rc == EVSLCU_ERR_NOMEM ? 0 : rc;  // the stencil form is optional
  }
  M->st_mask = dm;
  M->st_reach = reach;
  M->st_span = span;
  M->st_d = d;
  return 0;
}

void stencil_free(evslcu_mat *M) {
  evslcu_free(M->st_mask);
  M->st_mask = nullptr;
  M->st_d = 0;
}

// Y(:, c) = A X(:, c) for m columns (1 <= m <= 65535).
int stencil_spmv(const evslcu_mat *A, const double *X, double *Y, int m) {
  const dim3 g(grid_for(A->n), m);
  switch (st_width(A->st_d)) {
    case 5: k_st_spmv<5><<<g, kThreads, 0, stream()>>>(st_arg<double, 5>(A), X, Y, A->n); break;
    case 7: k_st_spmv<7><<<g, kThreads, 0, stream()>>>(st_arg<double, 7>(A), X, Y, A->n); break;
    case 9: k_st_spmv<9><<<g, kThreads, 0, stream()>>>(st_arg<double, 9>(A), X, Y, A->n); break;
    case 16: k_st_spmv<16><<<g, kThreads, 0, stream()>>>(st_arg<double, 16>(A), X, Y, A->n); break;
    default: k_st_spmv<32><<<g, kThreads, 0, stream()>>>(st_arg<double, 32>(A), X, Y, A->n); break;
  }
  EVSLCU_LAUNCH_CHECK("k_st_spmv");
  return 0;
}

int stencil_error() {
  if (!g_cl_err || !*(volatile int *)g_cl_err) return 0;
  *(volatile int *)g_cl_err = 0;
  return fail(EVSLCU_ERR_TIMEOUT, "a wait of the filter kernel did not complete within its bound");
}

bool stencil_ok(const evslcu_mat *M) { return M->st_d > 0 && M->use_pat && M->kernel == 0; }

// One degree step with y written at once (the kernel's timing among the other
// variants).
int stencil_step(const evslcu_mat *A, bool first, const double *vk, const double *vkm1, double *out, double *y,
                 double t, double ncc, double s, double mu0, const evslcu_cheb_epi *epi) {
  StY Y{first ? 2 : 1, first ? 1 : 0, 0.0, mu0, s};
  return st_step_any(A, first, vk, vkm1, out, y, t, ncc, Y, epi);
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
    StY Y{0, 0, 0.0, 0.0, 0.0};
    if (k == deg || k - from == 2) {
      Y.terms = k - from + 1;
      Y.init = from == 0;
      Y.c0 = mu[k];
      if (Y.terms >= 2) Y.c1 = mu[k - 1];
      if (Y.terms == 3) Y.c2 = mu[k - 2];
      from = k + 1;
    }
    const int rc = st_step_any(A, k == 1, vk, vkm1, W[(k - 1) % 2], y, (k == 1) ? t1 : t2, ncc, Y,
                               k == deg ? epi : nullptr);
    if (rc) return rc;
  }
  return 0;
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
}

}  // extern "C"
