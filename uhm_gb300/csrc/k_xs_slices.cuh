// Slices of an entry for the sliced tensor-core updates (k_xs.cu), for the kernels
// that write them: the pack kernel and the panel kernels.
#pragma once
#include <cstdint>
#include "k_xs.cuh"

namespace uhm_gpu {

// exponent of a row holding a NaN or an infinity: the update is NaN in that
// whole row and column (an infinity becomes one in the panel's TRSM already:
// the product with the zeros of the diagonal block's inverse)
constexpr int XS_BAD = 1 << 28;
// 64-column chunks per slice of a front's layout in a launch of panel width nb
__device__ __forceinline__ int xs_chunks(int nb, int fs) { return (min(nb, fs) + 63) / 64; }

template <typename T> struct XsType;
template <> struct XsType<double> {
  static constexpr int S = XS_S64;
  static __device__ __forceinline__ int field(double v) { return (__double2hiint(v) >> 20) & 0x7FF; }
  // the field, 1 for a subnormal number, 0 for zero (in integers: an FP64 comparison costs
  // as much as a multiply-add)
  static __device__ __forceinline__ int expo(double v) {
    const int f = field(v);
    return f ? f : (__double2hiint(v) << 1 | __double2loint(v)) != 0;
  }
  static constexpr int FMAX = 0x7FF, EBIAS = 1022;
  // round(v 2^(62 - e)), e = fmax - EBIAS, fmax the largest exponent field of the row (at least 1)
  static __device__ __forceinline__ long long fixed(double v, int fmax) {
    const long long b = __double_as_longlong(v);
    int f = (int)((b >> 52) & 0x7FF);
    long long m = b & 0xFFFFFFFFFFFFFll;
    if (f) m |= 1ll << 52;
    else f = 1;
    const int sh = fmax - f;
    m <<= 9;
    if (sh > 0) m = sh > 62 ? 0 : (m + (1ll << (sh - 1))) >> sh;
    return b < 0 ? -m : m;
  }
};
template <> struct XsType<float> {
  static constexpr int S = XS_S32;
  static __device__ __forceinline__ int field(float v) { return (__float_as_int(v) >> 23) & 0xFF; }
  static __device__ __forceinline__ int expo(float v) {
    const int f = field(v);
    return f ? f : (__float_as_int(v) << 1) != 0;
  }
  static constexpr int FMAX = 0xFF, EBIAS = 126;
  // round(v 2^(30 - e))
  static __device__ __forceinline__ long long fixed(float v, int fmax) {
    const int b = __float_as_int(v);
    int f = (b >> 23) & 0xFF;
    int m = b & 0x7FFFFF;
    if (f) m |= 1 << 23;
    else f = 1;
    const int sh = fmax - f;
    m <<= 6;
    if (sh > 0) m = sh > 31 ? 0 : (m + (1 << (sh - 1))) >> sh;
    return b < 0 ? -m : m;
  }
};

// the digits of one entry, as bits of exact floats (d[p] = slice p)
template <int S>
__device__ __forceinline__ void xs_digits(long long X, uint32_t (&d)[S]) {
  // balanced digits: adding 128 to every place but the top turns each into its
  // byte; float(2^23 + byte) - (2^23 + 128) is the digit
  constexpr long long BIAS = S == 8 ? 0x0080808080808080ll : 0x0000000000808080ll;
  const long long Y = X + BIAS;
#pragma unroll
  for (int p = 0; p < S; ++p) {
    float dg;
    if (p == 0) {
      dg = __int_as_float(0x4B400000 + (int)(Y >> (8 * (S - 1)))) - 12582912.0f;
    } else {
      const uint32_t b = (uint32_t)(Y >> (8 * (S - 1 - p))) & 0xFFu;
      dg = __int_as_float((int)(0x4B000000u | b)) - 8388736.0f;
    }
    d[p] = __float_as_uint(dg);
  }
}

// slices of 16 columns of a row, v, whose row's largest exponent field is fm: row
// `at` of the workspace, and, S = 8, the one `group` rows behind it; t: powers
// of two that the columns are multiplied by (fm with them), null: none
template <typename T>
__device__ __forceinline__ void xs_store16(const XsCtx& x, int64_t at, int64_t group, const T (&v)[16], int fm, bool bad,
                                           const int* t = nullptr) {
  constexpr int S = XsType<T>::S;
  uint8_t* const w0 = reinterpret_cast<uint8_t*>(x.ws) + 128 * at;
  uint32_t d[S][8];
#pragma unroll
  for (int u = 0; u < 16; u += 2) {
    uint32_t d0[S], d1[S];
    xs_digits<S>(bad ? 0 : XsType<T>::fixed(v[u], t ? fm - t[u] : fm), d0);
    xs_digits<S>(bad ? 0 : XsType<T>::fixed(v[u + 1], t ? fm - t[u + 1] : fm), d1);
#pragma unroll
    for (int p = 0; p < S; ++p) d[p][u / 2] = __byte_perm(d0[p], d1[p], 0x7632);
  }
#pragma unroll
  for (int p = 0; p < S; ++p) {
    uint4* w = reinterpret_cast<uint4*>(w0 + 128 * (p >> 2) * group + 32 * (p & 3));
    w[0] = make_uint4(d[p][0], d[p][1], d[p][2], d[p][3]);
    w[1] = make_uint4(d[p][4], d[p][5], d[p][6], d[p][7]);
  }
}

// The slices of a 64-column step's panel rows: 256 threads, thread r + 64 g holds
// columns 16 g .. of row `row` (rows not in the front: in = false).  Every thread
// of the CTA calls it; s_f is free again after the caller's next barrier.
template <typename T>
__device__ __forceinline__ void xs_store_step(const XsCtx& x, int front, int n, int row, bool in, const T (&v)[16],
                                              int (*s_f)[64]) {
  const int r = threadIdx.x % 64, g = threadIdx.x / 64;
  int fm = 1;
#pragma unroll
  for (int u = 0; u < 16; ++u) fm = max(fm, XsType<T>::field(v[u]));
  s_f[g][r] = fm;
  __syncthreads();
#pragma unroll
  for (int e = 0; e < 4; ++e) fm = max(fm, s_f[e][r]);
  if (!in) return;
  const bool bad = fm == XsType<T>::FMAX;
  if (g == 0) x.exps[x.exp0[front] + row] = bad ? XS_BAD : fm - XsType<T>::EBIAS;
  xs_store16<T>(x, x.row0[front] + (int64_t)g * n + row, (int64_t)4 * n, v, fm, bad);
}

}  // namespace uhm_gpu
