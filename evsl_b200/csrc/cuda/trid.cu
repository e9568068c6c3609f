// Eigenvalues of a symmetric tridiagonal matrix on the GPU, for the
// convergence tests of the filtered Lanczos solvers (the trace test of
// ChebLanNr, SRC/cheblanNr.c:241-262, needs every eigenvalue of T_k every
// 20 steps; the reference calls LAPACK dstev there).
//
// Multisection on Sturm counts: one warp per eigenvalue index i; each round
// the warp evaluates the count of eigenvalues below 128 equally spaced
// shifts of its bracket (4 per lane, their recurrences interleaved) and keeps
// the sub-interval where the count passes i, shrinking the bracket 129-fold.
// The bracket [lo, hi] always satisfies count(lo) <= i < count(hi), whatever
// the rounding of the counts, so the result lies within the final bracket
// of the computed spectrum.  Rounds stop at a relative width of 2 eps or
// after kRounds (bounded).  The count uses the LDL^T recurrence
// q_j = (d_j - x) - e_{j-1}^2 / q_{j-1} with tiny pivots replaced by -pivmin.
#include <algorithm>
#include <cfloat>
#include <cstdint>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"

namespace evslcu {
namespace {

constexpr int kPts = 4;                   // shifts per lane
constexpr int kShifts = 32 * kPts;        // shifts per round
constexpr int kSections = kShifts + 1;    // sub-intervals per round
constexpr int kRounds = 12;               // 129^12 > 2e25
constexpr int kTridThreads = 256;

__global__ void __launch_bounds__(kTridThreads)
    k_trid_bisect(int k, int i0, const double *__restrict__ d, const double *__restrict__ e2, double glo,
                  double ghi, double pivmin, double *__restrict__ w) {
  const int lane = threadIdx.x & 31;
  const int i = i0 + (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (i >= k) return;  // uniform over the warp
  double lo = glo, hi = ghi;
  for (int round = 0; round < kRounds; ++round) {
    const double width = hi - lo;
    if (width <= 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)) + pivmin) break;
    double x[kPts], q[kPts];
    int c[kPts];
#pragma unroll
    for (int p = 0; p < kPts; ++p) {
      x[p] = lo + width * (double)(lane * kPts + p + 1) / (double)kSections;
      q[p] = __ldg(d) - x[p];
      if (fabs(q[p]) < pivmin) q[p] = -pivmin;
      c[p] = q[p] < 0.0;
    }
    for (int j = 1; j < k; ++j) {
      const double dj = __ldg(d + j), ej = __ldg(e2 + j - 1);
#pragma unroll
      for (int p = 0; p < kPts; ++p) {
        q[p] = (dj - x[p]) - ej / q[p];
        if (fabs(q[p]) < pivmin) q[p] = -pivmin;
        c[p] += q[p] < 0.0;
      }
    }
    // first shift whose count exceeds i
    int first = kShifts;
#pragma unroll
    for (int p = kPts - 1; p >= 0; --p)
      if (c[p] > i) first = lane * kPts + p;
    first = __reduce_min_sync(0xffffffffu, first);
    const double nlo = (first == 0) ? lo : lo + width * (double)first / (double)kSections;
    const double nhi = (first == kShifts) ? hi : lo + width * (double)(first + 1) / (double)kSections;
    lo = nlo;
    hi = nhi;
  }
  if (lane == 0) w[i] = 0.5 * (lo + hi);
}

// Inverse iteration for eigenvectors num[0] .. num[m - 1] of T at shift[0] ..
// shift[m - 1], into the columns num[] of Z: one thread per vector, the arithmetic of the host's
// (invit_range, host/tridiag.c) operation for operation, so the vectors are
// the same bit for bit.  A vector is a chain of a few thousand dependent
// divisions and updates that costs the host 60 us at 850 rows; here all of them
// run side by side, and what bounds it is one chain.  Arrays are [row][vector],
// so that a warp's accesses are contiguous; rows are taken eight at a time
// with their loads issued before the chain needs them.
constexpr int kInvitIters = 3;

struct InvitWork {
  double *u0, *u1, *u2, *ml, *x;
  unsigned char *swp;
};

__device__ __forceinline__ double invit_start(uint64_t j, uint64_t i) {
  uint64_t z = (j << 32) + i;
  z += 0x9E3779B97F4A7C15ULL;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  z ^= z >> 31;
  return __dadd_rn(__dmul_rn((double)(z >> 11), 1.0 / 9007199254740992.0), -0.5);
}

__global__ void __launch_bounds__(32)
    k_trid_invit(int n, int m, const int *__restrict__ num, const double *__restrict__ d, const double *__restrict__ e,
                 const double *__restrict__ shift, double tiny, InvitWork W, double *__restrict__ Z, long long ldz) {
  constexpr int U = 8;
  const int c = blockIdx.x * 32 + threadIdx.x;
  if (c >= m) return;
  const size_t M = (size_t)m;
  const int j = num[c];
  const double lam = shift[c];
  double *const u0 = W.u0 + c, *const u1 = W.u1 + c, *const u2 = W.u2 + c, *const ml = W.ml + c, *const x = W.x + c;
  unsigned char *const swp = W.swp + c;
  auto floor_tiny = [&](double v) { return fabs(v) < tiny ? (v < 0.0 ? -tiny : tiny) : v; };
  // LU with partial pivoting of T - lam I: dg, du are rows i's entries so far
  {
    double dg = __dadd_rn(__ldg(d), -lam), du = n > 1 ? __ldg(e) : 0.0;
    for (int i = 0; i < n - 1; ++i) {
      const double sub = __ldg(e + i), dn = __dadd_rn(__ldg(d + i + 1), -lam), un = (i < n - 2) ? __ldg(e + i + 1) : 0.0;
      const size_t at = (size_t)i * M;
      if (fabs(dg) >= fabs(sub)) {
        const double l = (dg != 0.0) ? __ddiv_rn(sub, dg) : 0.0;
        u0[at] = floor_tiny(dg);
        u1[at] = du;
        u2[at] = 0.0;
        ml[at] = l;
        swp[at] = 0;
        dg = __dadd_rn(dn, -__dmul_rn(l, du));
        du = un;
      } else {
        const double l = __ddiv_rn(dg, sub);
        u0[at] = floor_tiny(sub);
        u1[at] = dn;
        u2[at] = un;
        ml[at] = l;
        swp[at] = 1;
        dg = __dadd_rn(du, -__dmul_rn(l, dn));
        du = (i < n - 2) ? __dmul_rn(-l, un) : un;
      }
    }
    u0[(size_t)(n - 1) * M] = floor_tiny(dg);
  }
  for (int i = 0; i < n; ++i) x[(size_t)i * M] = invit_start((uint64_t)j, (uint64_t)i);
  for (int it = 0; it < kInvitIters; ++it) {
    // forward: P L (xi: row i's value so far)
    double xi = x[0];
    for (int b = 0; b < n - 1; b += U) {
      double l[U], xn[U];
      unsigned char sw[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const size_t at = (size_t)min(b + u, n - 2) * M;
        l[u] = ml[at];
        sw[u] = swp[at];
        xn[u] = x[at + M];
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (b + u < n - 1) {
          const double lo = sw[u] ? xn[u] : xi, hi = sw[u] ? xi : xn[u];
          x[(size_t)(b + u) * M] = lo;
          xi = __dadd_rn(hi, -__dmul_rn(l[u], lo));
        }
    }
    // back: U
    double amax = 0.0, x1 = __ddiv_rn(xi, u0[(size_t)(n - 1) * M]), x2 = 0.0;  // x1, x2: rows i + 1, i + 2
    x[(size_t)(n - 1) * M] = x1;
    for (int b = n - 2; b >= 0; b -= U) {
      double p0[U], p1[U], p2[U], xr[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const size_t at = (size_t)max(b - u, 0) * M;
        p0[u] = u0[at];
        p1[u] = u1[at];
        p2[u] = u2[at];
        xr[u] = x[at];
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (b - u >= 0) {
          double t = __dadd_rn(xr[u], -__dmul_rn(p1[u], x1));
          if (b - u < n - 2) t = __dadd_rn(t, -__dmul_rn(p2[u], x2));
          t = __ddiv_rn(t, p0[u]);
          x[(size_t)(b - u) * M] = t;
          x2 = x1;
          x1 = t;
        }
    }
#pragma unroll 8
    for (int i = 0; i < n; ++i) {
      const double v = fabs(x[(size_t)i * M]);
      amax = amax > v ? amax : v;
    }
    if (amax == 0.0) {
      x[(size_t)(j % n) * M] = 1.0;
      amax = 1.0;
    }
    double nrm = 0.0;
#pragma unroll 8
    for (int i = 0; i < n; ++i) {
      const double v = __ddiv_rn(x[(size_t)i * M], amax);
      x[(size_t)i * M] = v;
      nrm = __dadd_rn(nrm, __dmul_rn(v, v));
    }
    nrm = __dsqrt_rn(nrm);
#pragma unroll 8
    for (int i = 0; i < n; ++i) x[(size_t)i * M] = __ddiv_rn(x[(size_t)i * M], nrm);
  }
  // sign convention: largest component (the first of equals) positive
  double big = x[0];
#pragma unroll 8
  for (int i = 1; i < n; ++i) {
    const double v = x[(size_t)i * M];
    if (fabs(v) > fabs(big)) big = v;
  }
  const double sgn = big < 0.0 ? -1.0 : 1.0;
  double *z = Z + (long long)j * ldz;
#pragma unroll 8
  for (int i = 0; i < n; ++i) z[i] = __dmul_rn(sgn, x[(size_t)i * M]);
}

// Scratch of a launch at most; more vectors go in several.
constexpr size_t kInvitBytes = (size_t)512 << 20;

double *g_trid_buf = nullptr;
int g_trid_cap = 0;

// Side-stream form for the convergence tests: inputs staged in pinned host
// memory, the bisection on its own stream, the result copied back
// asynchronously; the solver reads it when it needs it.
cudaStream_t g_side = nullptr;
cudaEvent_t g_main_mark = nullptr, g_side_done = nullptr;
double *g_pin = nullptr;  // pinned: d | e2 | w, g_pin_cap each
int g_pin_cap = 0;
struct {
  bool pending;
  int k, i0;
  double glo;
} g_async = {false, 0, 0, 0.0};

// Gershgorin interval (widened), pivot floor, squared off-diagonals (into
// e2[0..k-1)) and the first index that may reach xmin (see below).
struct TridPrep {
  double glo, ghi, pivmin;
  int i0;
};

TridPrep trid_prep(int k, const double *d, const double *e, double xmin, double *e2) {
  double emax = 0.0, glo = d[0], ghi = d[0];
  for (int j = 0; j < k; ++j) {
    const double ej = (j + 1 < k) ? fabs(e[j]) : 0.0;
    const double ejm = (j > 0) ? fabs(e[j - 1]) : 0.0;
    glo = std::min(glo, d[j] - ej - ejm);
    ghi = std::max(ghi, d[j] + ej + ejm);
    if (j + 1 < k) {
      e2[j] = e[j] * e[j];
      emax = std::max(emax, e2[j]);
    }
  }
  const double pivmin = DBL_MIN * std::max(1.0, emax);
  const double fudge = 2.0 * DBL_EPSILON * std::max(fabs(glo), fabs(ghi)) * k + 2.0 * pivmin;
  glo -= fudge;
  ghi += fudge;
  // Indices below i0 are skipped: their eigenvalues lie below xc, far
  // enough under xmin (1e-8 of the spectral scale, four orders above the
  // counts' rounding) that none of them can reach xmin.  One index of slack
  // on top.  The others are bisected from the same bracket as in the full
  // computation, so they come out bit for bit the same.
  int i0 = 0;
  if (xmin > glo) {
    const double xc = xmin - 1e-8 * std::max(1.0, std::max(fabs(glo), fabs(ghi)));
    double q = d[0] - xc;
    if (fabs(q) < pivmin) q = -pivmin;
    int cnt = q < 0.0;
    for (int j = 1; j < k; ++j) {
      q = (d[j] - xc) - e2[j - 1] / q;
      if (fabs(q) < pivmin) q = -pivmin;
      cnt += q < 0.0;
    }
    i0 = std::max(0, cnt - 1);
  }
  return {glo, ghi, pivmin, i0};
}

int trid_device_buffers(int k) {
  if (k <= g_trid_cap) return 0;
  evslcu_free(g_trid_buf);
  g_trid_cap = std::max(k, 1024);
  g_trid_buf = (double *)evslcu_malloc(sizeof(double) * 3 * (size_t)g_trid_cap);
  if (!g_trid_buf) {
    g_trid_cap = 0;
    return fail(EVSLCU_ERR_NOMEM, "tridiagonal eigenvalues: out of device memory");
  }
  return 0;
}

int trid_launch(int k, const TridPrep &p, cudaStream_t st) {
  if (p.i0 >= k) return 0;
  double *dd = g_trid_buf, *de2 = g_trid_buf + g_trid_cap, *dw = g_trid_buf + 2 * (size_t)g_trid_cap;
  const long long threads = 32LL * (k - p.i0);
  const int grid = (int)((threads + kTridThreads - 1) / kTridThreads);
  k_trid_bisect<<<grid, kTridThreads, 0, st>>>(k, p.i0, dd, de2, p.glo, p.ghi, p.pivmin, dw);
  count_launch();
  return check_launch("k_trid_bisect");
}

}  // namespace
}  // namespace evslcu

using namespace evslcu;

extern "C" {

void evslcu_trid_release(void) {
  if (g_async.pending) {
    cudaEventSynchronize(g_side_done);
    g_async.pending = false;
  }
  evslcu_free(g_trid_buf);
  g_trid_buf = nullptr;
  g_trid_cap = 0;
  if (g_pin) cudaFreeHost(g_pin);
  g_pin = nullptr;
  g_pin_cap = 0;
  if (g_side) {
    cudaStreamDestroy(g_side);
    cudaEventDestroy(g_main_mark);
    cudaEventDestroy(g_side_done);
    g_side = nullptr;
    g_main_mark = g_side_done = nullptr;
  }
}

int evslcu_trid_eigvals_above(int k, const double *d, const double *e, double xmin, double *w) {
  if (k <= 0) return 0;
  if (!d || !w || (k > 1 && !e)) return fail(EVSLCU_ERR_ARG, "evslcu_trid_eigvals: bad arguments");
  // a side-stream test still reading the device buffers goes first
  if (g_async.pending) EVSLCU_CUDA(cudaStreamWaitEvent(stream(), g_side_done, 0));
  int rc = trid_device_buffers(k);
  if (rc) return rc;
  std::vector<double> e2((size_t)std::max(k - 1, 1), 0.0);
  const TridPrep p = trid_prep(k, d, e, xmin, e2.data());
  double *dd = g_trid_buf, *de2 = g_trid_buf + g_trid_cap, *dw = g_trid_buf + 2 * (size_t)g_trid_cap;
  rc = evslcu_h2d_async(dd, d, sizeof(double) * (size_t)k);
  if (!rc && k > 1) rc = evslcu_h2d_async(de2, e2.data(), sizeof(double) * (size_t)(k - 1));
  if (!rc) rc = trid_launch(k, p, stream());
  if (!rc && p.i0 < k) rc = evslcu_d2h(w + p.i0, dw + p.i0, sizeof(double) * (size_t)(k - p.i0));
  if (rc) return rc;
  for (int i = 0; i < p.i0; ++i) w[i] = p.glo;  // below every computed eigenvalue and below xmin
  std::sort(w, w + k);
  return 0;
}

int evslcu_trid_eigvals_async(int k, const double *d, const double *e, double xmin) {
  if (k <= 0 || !d || (k > 1 && !e)) return fail(EVSLCU_ERR_ARG, "evslcu_trid_eigvals_async: bad arguments");
  if (g_async.pending) return fail(EVSLCU_ERR_ARG, "evslcu_trid_eigvals_async: a test is still in flight");
  if (!g_side) {
    EVSLCU_CUDA(cudaStreamCreateWithFlags(&g_side, cudaStreamNonBlocking));
    EVSLCU_CUDA(cudaEventCreateWithFlags(&g_main_mark, cudaEventDisableTiming));
    EVSLCU_CUDA(cudaEventCreateWithFlags(&g_side_done, cudaEventDisableTiming));
  }
  if (k > g_pin_cap) {
    if (g_pin) cudaFreeHost(g_pin);
    g_pin = nullptr;
    const int cap = std::max(k, 2 * g_pin_cap);
    EVSLCU_CUDA(cudaMallocHost(&g_pin, sizeof(double) * 3 * (size_t)cap));
    g_pin_cap = cap;
  }
  int rc = trid_device_buffers(k);
  if (rc) return rc;
  double *pd = g_pin, *pe2 = g_pin + g_pin_cap, *pw = g_pin + 2 * (size_t)g_pin_cap;
  memcpy(pd, d, sizeof(double) * (size_t)k);
  const TridPrep p = trid_prep(k, d, e, xmin, pe2);
  double *dd = g_trid_buf, *de2 = g_trid_buf + g_trid_cap, *dw = g_trid_buf + 2 * (size_t)g_trid_cap;
  // the device buffers come from the library stream's pool: order the side
  // stream after it
  EVSLCU_CUDA(cudaEventRecord(g_main_mark, stream()));
  EVSLCU_CUDA(cudaStreamWaitEvent(g_side, g_main_mark, 0));
  EVSLCU_CUDA(cudaMemcpyAsync(dd, pd, sizeof(double) * (size_t)k, cudaMemcpyHostToDevice, g_side));
  if (k > 1) EVSLCU_CUDA(cudaMemcpyAsync(de2, pe2, sizeof(double) * (size_t)(k - 1), cudaMemcpyHostToDevice, g_side));
  if ((rc = trid_launch(k, p, g_side))) return rc;
  if (p.i0 < k)
    EVSLCU_CUDA(cudaMemcpyAsync(pw + p.i0, dw + p.i0, sizeof(double) * (size_t)(k - p.i0), cudaMemcpyDeviceToHost,
                                g_side));
  EVSLCU_CUDA(cudaEventRecord(g_side_done, g_side));
  g_async = {true, k, p.i0, p.glo};
  return 0;
}

int evslcu_trid_eigvals_async_ready(void) {
  if (!g_async.pending) return 1;
  const cudaError_t e = cudaEventQuery(g_side_done);
  if (e == cudaErrorNotReady) return 0;
  return 1;  // finished, or failed: the wait reports the error
}

int evslcu_trid_eigvals_async_wait(double *w) {
  if (!g_async.pending) return fail(EVSLCU_ERR_ARG, "evslcu_trid_eigvals_async_wait: no test in flight");
  g_async.pending = false;
  EVSLCU_CUDA(cudaEventSynchronize(g_side_done));
  const int k = g_async.k, i0 = g_async.i0;
  const double *pw = g_pin + 2 * (size_t)g_pin_cap;
  if (i0 < k) memcpy(w + i0, pw + i0, sizeof(double) * (size_t)(k - i0));
  for (int i = 0; i < i0; ++i) w[i] = g_async.glo;
  std::sort(w, w + k);
  return 0;
}

int evslcu_trid_invit(int n, const double *d, const double *e, int m, const int *num, const double *shift, double tiny,
                      double *Z, long long ldz) {
  if (n < 2 || m < 1 || !d || !e || !num || !shift || !Z) return fail(EVSLCU_ERR_ARG, "trid_invit: bad arguments");
  const size_t row = 5 * sizeof(double) + 1, in = (size_t)2 * n + 2 * (size_t)m;
  // vectors of a launch: what kInvitBytes hold, fewer when memory is short
  int mc = (int)std::min<size_t>((size_t)m, std::max<size_t>(32, kInvitBytes / (row * (size_t)n)));
  double *buf = nullptr;
  while (!(buf = (double *)evslcu_malloc(sizeof(double) * in + row * (size_t)n * mc))) {
    if (mc <= 32) return EVSLCU_ERR_NOMEM;
    mc = std::max(32, mc / 2);
  }
  double *dd = buf, *de = buf + n, *ds = buf + 2 * (size_t)n, *w = buf + in;
  int *dn = (int *)(ds + m);
  int rc = evslcu_h2d_async(dd, d, sizeof(double) * (size_t)n);
  if (!rc) rc = evslcu_h2d_async(de, e, sizeof(double) * (size_t)(n - 1));
  if (!rc) rc = evslcu_h2d_async(ds, shift, sizeof(double) * (size_t)m);
  if (!rc) rc = evslcu_h2d_async(dn, num, sizeof(int) * (size_t)m);
  const size_t blk = (size_t)n * mc;
  const InvitWork W{w, w + blk, w + 2 * blk, w + 3 * blk, w + 4 * blk, (unsigned char *)(w + 5 * blk)};
  for (int j0 = 0; j0 < m && !rc; j0 += mc) {
    const int c = std::min(mc, m - j0);
    k_trid_invit<<<(c + 31) / 32, 32, 0, stream()>>>(n, c, dn + j0, dd, de, ds + j0, tiny, W, Z, ldz);
    count_launch();
    rc = check_launch("k_trid_invit");
  }
  evslcu_free(buf);
  return rc;
}

int evslcu_trid_eigvals(int k, const double *d, const double *e, double *w) {
  return evslcu_trid_eigvals_above(k, d, e, -HUGE_VAL, w);
}

}  // extern "C"
