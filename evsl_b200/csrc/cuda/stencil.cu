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
#include <algorithm>
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
      double g[D];
#pragma unroll
      for (int e = 0; e < D; ++e) g[e] = (m[0] >> e & 1u) ? __ldg(xr + A.off[e]) : 0.0;
      if (live[0]) x[0] = __ldg(xr);
#pragma unroll
      for (int e = 0; e < D; ++e)
        if (m[0] >> e & 1u) acc[0] = st_fmadd(A.val[e], g[e], acc[0]);
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

}  // namespace

namespace evslcu {

// Merges the dictionary's patterns into one list of (offset, value) entries;
// leaves M->st_d at 0 when a pattern's offsets do not increase or the list
// has more than kStMax entries.
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
