// Merged-stencil form of a matrix with a row-pattern dictionary, and the
// device code that multiplies its rows.
//
// The rows of a structured-grid operator are subsets of ONE short list of
// (column offset, value) entries: a 7-point Laplacian has 27 row patterns but
// 7 entries.  When the dictionary's patterns merge into at most kStMax entries
// in increasing offset order, each row needs only a bit mask (1, 2 or 4
// bytes) saying which entries it has; the list itself is a kernel argument.
// A row product is then, per entry, one load at a register + uniform offset,
// one multiply and one add: no table lookup on the row's dependent chain, no
// value conversion.  The entries of a row are taken in increasing offset
// order, which is its CSR order (the merge requires that), so row sums are
// the CSR row's bit for bit.
#pragma once

#include <stdint.h>

#include "sparse_types.cuh"

namespace evslcu {

constexpr int kStMax = 32;  // entries of a merged stencil

template <int D>
struct StMaskT {
  using T = uint32_t;
};
template <>
struct StMaskT<5> {
  using T = uint8_t;
};
template <>
struct StMaskT<7> {
  using T = uint8_t;
};
template <>
struct StMaskT<9> {
  using T = uint16_t;
};
template <>
struct StMaskT<16> {
  using T = uint16_t;
};

// Bytes of a row's mask and the compiled width for d entries.
inline int st_width(int d) { return d <= 5 ? 5 : d <= 7 ? 7 : d <= 9 ? 9 : d <= 16 ? 16 : 32; }
inline int st_mask_bytes(int d) { return d <= 7 ? 1 : d <= 16 ? 2 : 4; }

// The stencil as a kernel argument.  full: the mask of a row with every
// entry, or 0xffffffff (which no row has) when fewer than D entries are in use; center:
// the entry D / 2 is the diagonal.
template <class VT, int D>
struct StArg {
  int n;
  const typename StMaskT<D>::T *__restrict__ mask;
  unsigned full;
  int center;
  VT val[D];
  int off[D];
};

template <class VT, int D>
inline StArg<VT, D> st_arg(const evslcu_mat *A) {
  StArg<VT, D> S;
  S.n = A->n;
  S.mask = (const typename StMaskT<D>::T *)A->st_mask;
  S.full = (A->st_d == D && D < 32) ? (1u << (D & 31)) - 1u : 0xffffffffu;
  S.center = (A->st_d == D && A->st_off[D / 2] == 0) ? 1 : 0;
  for (int j = 0; j < D; ++j) {
    S.val[j] = (VT)(j < A->st_d ? A->st_val[j] : 0.0);
    S.off[j] = j < A->st_d ? A->st_off[j] : 0;
  }
  return S;
}

// Rounded multiply and add in FP64 (the reference's order), fused in FP32, as
// the other filter kernels.
__device__ __forceinline__ double st_fmadd(double a, double b, double acc) { return __dadd_rn(acc, __dmul_rn(a, b)); }
__device__ __forceinline__ float st_fmadd(float a, float b, float acc) { return fmaf(a, b, acc); }
// The zero whose product with v is -0 (v finite).  Adding -0 leaves every sum
// as it is, signed zeros included, so a row takes an absent entry as v times
// this zero.
__device__ __forceinline__ double st_zero(double v) {
  return __hiloint2double((~__double2hiint(v)) & (int)0x80000000, 0);
}
__device__ __forceinline__ float st_zero(float v) { return __uint_as_float(~__float_as_uint(v) & 0x80000000u); }
// y += c w: rounded multiply and add in both precisions.
__device__ __forceinline__ double st_fmadd_y(double c, double w, double y) { return __dadd_rn(y, __dmul_rn(c, w)); }
__device__ __forceinline__ float st_fmadd_y(float c, float w, float y) { return __fadd_rn(y, __fmul_rn(c, w)); }
__device__ __forceinline__ double st_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float st_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double st_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float st_add(float a, float b) { return __fadd_rn(a, b); }

}  // namespace evslcu
