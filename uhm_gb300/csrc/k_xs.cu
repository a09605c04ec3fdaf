// Trailing updates C -= A B^T of FP64 and FP32 fronts on the tensor cores, at
// the precision of multiply-adds in the front's own type: the operands are cut
// into 8-bit slices whose BF16 products add up exactly.
//
// Restates the trailing SYRK / GEMM of the front's blocked factorisation
// (LINAL/src/dense/chol.cxx:78-82, lu_piv.cxx:95-105 and the front-level
// updates of UHM/src/matrix/uhm/fla/chol/decompose.cxx:94-95,
// fla/lu_piv/decompose.cxx:148-149).
//
// Slices (the error-free splitting of Ozaki, Ogita, Oishi and Rump, "Error-
// free transformations of matrix multiplication by using fast routines of
// matrix multiplication", 2012, with digits in place of floating parts): every
// row of a panel of W <= 256 columns gets one exponent e, |a| < 2^e, and each
// entry becomes the integer X = round(a 2^(62-e)) (FP64; 2^(30-e) for FP32),
// written in balanced base 256, X = sum_p d_p 256^(S-1-p), -128 <= d_p <=
// 127, |d_0| <= 64, S = 8 (4).  Digits are exact in BF16.  A product a b is
// 2^(ea+eb-124) sum_d 256^(14-d) sum_{p+q=d} d_p d'_q; the sums over k of
// one diagonal d are integers below 2^24 for d <= 4 (W <= 256), so FP32
// accumulation in tensor memory is exact; d = 5..7 stay below 1.75 2^24, where
// a rounding is worth 2^-60 of the row maxima's product.  Diagonals d > 7
// (> 3 for FP32) are left out: about 2^-66 (2^-32) of W times the product of
// the row maxima.  36 (10) of the 64 (16) slice products remain.  The
// diagonals are added up in 64-bit integers, whose last place is 2^-54 (2^-36)
// of the product of the row bounds, and applied to C with one rounding per panel
// instead of one per column.  Measured against 64 bits the solutions are as
// close as the SIMT update's (seven slices without diagonal 7 were 3 to 10
// times further off).
//
// All that is relative to the product of two row maxima, and a multiply-add's error
// to the sum of the products' magnitudes.  Cholesky: both are bounded by
// sqrt(a_ii a_jj), as for a factorisation in the type itself.  LU: the maxima of a
// row of L21 and a column of U12 can lie at different inner k, where l_ik scales as
// 1 / d_k and u_kj as d_k with the unit d_k of an eliminated equation (rows in
// units of 1 and 10^10: solutions of an FP64 front 10^6 to 10^8 times further off).  So
//  - before they are cut, row k of U12 is divided and column k of L21 multiplied by 2^t,
//    t <= 0 how near the row comes to a column's largest entry, at its best column:
//    exact, and the products stay.  Units of equations cancel, every row reaches some
//    column's maximum, and no column's maximum grows, so that the error stays
//    small in proportion to each column, which is what the solution sees.  (Half the
//    difference of the largest exponents of the column and the row balances
//    units as well, but an FP64 convection-diffusion solve of 24^3, coefficients 1 to
//    10^4, had a backward error 140 times larger; so scaled that the largest entry of
//    each column of L21 is near 1, 3 % of the blocks below were left to multiply-adds.)
//  - each row keeps which of the panel's columns come within 2^6 of its maximum, each
//    front which of them some row of the other operand has so near its own.  A row
//    or column of a tile where no column is both (of the front's own part, or of its
//    shared part, whichever the tile is in; columns of region 2, rows of U themselves,
//    are not checked) goes by plain multiply-adds (xs_plain).
// Measured: errors of fronts with units to 2^33 and of rows that no scaling serves are 0.4
// to 2.8 times those of multiply-adds (tests/test_gpu_lu_scaling.py); backward errors
// of 12^3, 16^3 and 24^3 convection-diffusion 4.4e-19, 3.0e-19 and 2.3e-19 (3.8e-19, 2.1e-19
// and 2.1e-19 without scaling).  Less than 0.5 % of the 32 x 32 blocks have such a row or column.
// Cost: factorisations 6^3 p = 3 FP64 LU 6.5 -> 6.65 ms, 12^3 38.0 -> 39.2, 24^3 273 -> 288
// (multiply-adds 8, the check 4.5), FP32 119 -> 129.
//
// Why: GB300 does about 2 FP64 multiply-adds per clock per SM (1.17 TFLOP/s
// measured for the SIMT update), against 1,906 TFLOP/s of BF16 products:
// 36 products per FP64 one still leave 53.  FP32 fronts: 10 products leave
// 190 TFLOP/s against 15 measured for the SIMT update.  Measured on GB300, the
// updates of one factorisation: 16^3 p = 4 FP64 906 -> 33.8 ms (and 2.3 for the
// slices), 13^3 p = 4 FP32 23.0 -> 6.4 (2.0), 12^3 p = 3 FP64 LU 196 -> 10.2 (2.7).
#include <cuda.h>
#include <cudaTypedefs.h>

#include <stdexcept>
#include <type_traits>

#include "k_common.cuh"
#include "k_tc_ptx.cuh"
#include "k_xs.cuh"
#include "k_xs_slices.cuh"

namespace uhm_gpu {

UHM_DEFINE_WAIT_LIMIT(set_wait_limit_xs, 1u << 22)

constexpr int XS_ERR = 7;

// ---------------------------------------------------------------------------
// slices
// ---------------------------------------------------------------------------
// A CTA cuts 256 / NG rows: thread r + (256 / NG) g holds 16 columns 16 g .. of
// row r (a warp's loads of one column are consecutive rows), all its loads in
// flight, and writes its digits as one or two whole rows of the workspace.  NG =
// 4 (64 columns) or 16 (256).  Memory bound: 8 (4) bytes read and 16 (8)
// written per entry; the digits come from integer shifts and byte extraction,
// no FP64.  Measured on GB300 for 256 columns: 29 us with 64 rows per CTA and
// its 64-column chunks in turn (whatever their number), 11 with 16 rows.
template <typename T, int NG>
__global__ void __launch_bounds__(256) k_xs_pack(DevCtx c, XsCtx x, const Item* __restrict__ items, int nb,
                                                  int use) {
  constexpr int S = XsType<T>::S, ROWS = 256 / NG;
  constexpr int NEAR = S == 8 ? XS_NEAR64 : XS_NEAR32;
  __shared__ int s_f[NG][ROWS], s_r[NG][ROWS];
  __shared__ __align__(16) int s_t[16 * NG];
  __shared__ uint32_t s_or[2][8];
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, K0 = it.a, trans = it.c;
  const int W = min(nb, f.fs - K0), nch = xs_chunks(nb, f.fs);
  const bool lu = x.scale != nullptr;
  const int r = threadIdx.x % ROWS, g = threadIdx.x / ROWS;
  const int row = it.b + r;
  const T* __restrict__ G = arena<T>(c) + f.off;
  const int64_t base = trans ? (int64_t)row * n + K0 : row + (int64_t)K0 * n;
  const int64_t step = trans ? 1 : n;
  const bool in = row < n;
  T v[16];
#pragma unroll
  for (int u = 0; u < 16; ++u) v[u] = in && 16 * g + u < W ? G[base + (16 * g + u) * step] : T(0);
  if (lu && threadIdx.x < 16 * NG) {
    int t = 0;
    if ((int)threadIdx.x < W) {
      const int v = x.scale[use * x.scale_n + f.piv_off + K0 + threadIdx.x];
      t = v ? v - XS_SCALE0 : 0;
    }
    s_t[threadIdx.x] = trans ? -t : t;
  }
  const int64_t row0 = (trans ? x.row0b : x.row0)[it.front] + (int64_t)g * n + row;
  if (!lu) {
    int fm = 1;
#pragma unroll
    for (int u = 0; u < 16; ++u) fm = max(fm, XsType<T>::field(v[u]));
    s_f[g][r] = fm;
    __syncthreads();
#pragma unroll
    for (int e = 0; e < NG; ++e) fm = max(fm, s_f[e][r]);
    if (!in || 16 * g >= 64 * nch) return;
    const bool bad = fm == XsType<T>::FMAX;
    if (g == 0) x.exps[x.exp0[it.front] + row] = bad ? XS_BAD : fm - XsType<T>::EBIAS;
    xs_store16<T>(x, row0, (int64_t)4 * nch * n, v, fm, bad);
    return;
  }
  __syncthreads();                             // s_t
  // (a zero counts as the smallest number for the row's exponent and is never near)
  int e[16], fr = 0, fm = -XS_BAD;
#pragma unroll
  for (int u = 0; u < 16; u += 4) {
    const int4 t4 = *reinterpret_cast<const int4*>(s_t + 16 * g + u);
    const int t[4] = {t4.x, t4.y, t4.z, t4.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int fu = XsType<T>::field(v[u + q]);
      fr = max(fr, fu);
      e[u + q] = max(fu, 1) + t[q];
      fm = max(fm, e[u + q]);
    }
  }
  if (fr == XsType<T>::FMAX) fm = XS_BAD;
  s_f[g][r] = fm;
  s_r[g][r] = fr;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NG; ++q) {
    fm = max(fm, s_f[q][r]);
    fr = max(fr, s_r[q][r]);
  }
  const bool bad = fm == XS_BAD, some = fr > 0 && !bad;
  // the columns near the row's maximum; a row without any counts as near in all
  uint32_t mask = 0;
#pragma unroll
  for (int u = 0; u < 16; ++u)
    if (e[u] >= fm - NEAR && XsType<T>::field(v[u])) mask |= 1u << u;
  // their union over the CTA's own and its shared rows (side A of region 2: not checked)
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t all = __reduce_or_sync(0xffffffffu, some && (row >= f.fs) == h ? mask << (16 * (g & 1)) : 0u);
    if ((threadIdx.x & 31) == 0) s_or[h][threadIdx.x >> 5] = all;
  }
  if (in && 16 * g < 64 * nch) {
    const int64_t at = x.exp0[it.front] + (trans ? n : 0) + row;
    reinterpret_cast<uint16_t*>(x.masks)[at * (XS_NBO / 16) + g] = (uint16_t)(some ? mask : 0xFFFFu);
    if (g == 0) x.exps[at] = bad ? XS_BAD : fm - XsType<T>::EBIAS;
    xs_store16<T>(x, row0, (int64_t)4 * nch * n, v, fm, bad, s_t + 16 * g);
  }
  if (use == 2 && !trans) return;
  __syncthreads();
  // (one request per CTA: hundreds meet at one L2 line)
  const int h = threadIdx.x / (NG / 2), w = threadIdx.x % (NG / 2);
  if (h < 2) {
    uint32_t all = 0;
#pragma unroll
    for (int e = 0; e < 16 / NG; ++e) all |= s_or[h][NG == 16 ? w : 4 * w + e];
    if (all) atomicOr(x.near + (4 * use + 2 * trans + h) * x.near_n + x.near0[it.front] + K0 / 32 + w, all);
  }
}

void launch_xs_pack(const DevCtx& c, const XsCtx& x, const Item* items, int n_items, int dtype, int nb, int use,
                    cudaStream_t s) {
  if (!n_items) return;
  if (nb != 64 && nb != XS_NBO) throw std::invalid_argument("slices: panel width must be 64 or 256");
  if (use < 0 || use >= XS_USES) throw std::invalid_argument("slices: the update's region must be 0, 1 or 2");
  if (dtype == F64) {
    if (nb == 64) k_xs_pack<double, 4><<<n_items, 256, 0, s>>>(c, x, items, nb, use);
    else k_xs_pack<double, 16><<<n_items, 256, 0, s>>>(c, x, items, nb, use);
  } else {
    if (nb == 64) k_xs_pack<float, 4><<<n_items, 256, 0, s>>>(c, x, items, nb, use);
    else k_xs_pack<float, 16><<<n_items, 256, 0, s>>>(c, x, items, nb, use);
  }
}

// How near each of an outer panel's rows of U12 comes to a column's largest entry, at
// its best column: a warp takes four columns, whose entries are contiguous.
template <typename T>
__global__ void __launch_bounds__(256) k_xs_scale(DevCtx c, XsCtx x, const Item* __restrict__ items) {
  __shared__ int s_near[XS_NBO];
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, K0 = it.a, W = min(XS_NBO, f.fs - K0), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const T* __restrict__ G = arena<T>(c) + f.off + K0;
  s_near[threadIdx.x] = 0;
  int best[XS_NBO / 32];
#pragma unroll
  for (int i = 0; i < XS_NBO / 32; ++i) best[i] = 0;
  T v[2][XS_NBO / 32];
  auto load = [&](int j, T (&w)[XS_NBO / 32]) {
    const int col = it.b + 4 * warp + j;
#pragma unroll
    for (int i = 0; i < XS_NBO / 32; ++i) w[i] = col < n && lane + 32 * i < W ? G[lane + 32 * i + (int64_t)col * n] : T(0);
  };
  load(0, v[0]);
#pragma unroll
  for (int j = 0; j < XS_SCALE_COLS / 8; ++j) {
    if (j + 1 < XS_SCALE_COLS / 8) load(j + 1, v[(j + 1) & 1]);
    int e[XS_NBO / 32], cm = 0;
#pragma unroll
    for (int i = 0; i < XS_NBO / 32; ++i) {
      e[i] = XsType<T>::expo(v[j & 1][i]);
      cm = max(cm, e[i]);
    }
    cm = __reduce_max_sync(0xffffffffu, cm);
#pragma unroll
    for (int i = 0; i < XS_NBO / 32; ++i)
      if (e[i]) best[i] = max(best[i], XS_SCALE0 + e[i] - cm);
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < XS_NBO / 32; ++i)
    if (best[i]) atomicMax(&s_near[lane + 32 * i], best[i]);
  __syncthreads();
  if (s_near[threadIdx.x]) atomicMax(x.scale + f.piv_off + K0 + threadIdx.x, s_near[threadIdx.x]);
}

void launch_xs_scale(const DevCtx& c, const XsCtx& x, const Item* items, int n_items, int dtype, cudaStream_t s) {
  if (!n_items) return;
  static_assert(XS_NBO == 256 && XS_SCALE_COLS == 32, "a thread per row of the panel, four columns a warp");
  if (dtype == F64) k_xs_scale<double><<<n_items, 256, 0, s>>>(c, x, items);
  else k_xs_scale<float><<<n_items, 256, 0, s>>>(c, x, items);
}

// FP64 Cholesky panel TRSM, X = A Linv^T below a 64-column diagonal block (its
// inverse from k_potrf_inv64), and the slices of X for the panel's own update.
// 16 rows per CTA: thread (i, j) sums columns j, j + 16, j + 32, j + 48 of row
// i, each up to its diagonal (Linv is lower triangular), so every warp issues
// the same 160 of 256 multiply-adds per row.  Bound by those (2 per clock and
// SM); 16 rows instead of 64 spread a panel over every SM: the smallest launch
// took 55 us with 64 rows, 17 with 16, slices included (they were a launch of 12 us
// of their own).  Item: front, a = k0, b = first row, c = 1: slices too.
constexpr int XT_ROWS = XS_TRSM_ROWS;
__global__ void __launch_bounds__(256) k_xs_trsm64(DevCtx c, XsCtx x, const Item* __restrict__ items) {
  constexpr int S = XS_S64;
  __shared__ double Lt[64 * 64];               // Lt[t][j] = Linv[j][t]
  __shared__ double Xs[64][XT_ROWS];           // A, then X
  __shared__ int s_f[XT_ROWS];
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, k0 = it.a, r0 = it.b;
  const int kb = min(64, f.fs - k0);
  double* __restrict__ G = c.a64 + f.off + r0 + (int64_t)k0 * n;
  const double* __restrict__ D = c.dinv64 + f.dinv_off + (int64_t)(k0 / 64) * 4096;
  const int tid = threadIdx.x, i = tid & 15, jg = tid >> 4;
  const bool rv = r0 + i < n;
  {
    double dv[16], xv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int t = jg + 16 * u;
      xv[u] = rv && t < kb ? G[i + (int64_t)t * n] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 16; ++u) dv[u] = D[tid + 256 * u];
#pragma unroll
    for (int u = 0; u < 4; ++u) Xs[jg + 16 * u][i] = xv[u];
#pragma unroll
    for (int u = 0; u < 16; ++u) Lt[tid + 256 * u] = dv[u];
    if (tid < XT_ROWS) s_f[tid] = 1;
  }
  __syncthreads();
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int h = 0; h < 4; ++h) {
#pragma unroll 4
    for (int t = 16 * h; t < 16 * h + 16; ++t) {
      const double xt = Xs[t][i];
#pragma unroll
      for (int u = h; u < 4; ++u) acc[u] += xt * Lt[t * 64 + jg + 16 * u];
    }
  }
  int fm = 1;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int j = jg + 16 * u;
    if (rv && j < kb) G[i + (int64_t)j * n] = acc[u];
    fm = max(fm, XsType<double>::field(acc[u]));
  }
  if (!it.c) return;
  atomicMax(&s_f[i], fm);
  __syncthreads();                             // A has been read
#pragma unroll
  for (int u = 0; u < 4; ++u) Xs[jg + 16 * u][i] = acc[u];
  __syncthreads();
  // thread (row tid / 16, columns 4 (tid % 16) ..): 8 bytes of every slice
  const int r = tid >> 4, c4 = 4 * (tid & 15), row = r0 + r;
  if (row >= n) return;
  fm = s_f[r];
  const bool bad = fm == XsType<double>::FMAX;
  if (c4 == 0) x.exps[x.exp0[it.front] + row] = bad ? XS_BAD : fm - XsType<double>::EBIAS;
  uint32_t d[4][S];
#pragma unroll
  for (int e = 0; e < 4; ++e) xs_digits<S>(bad ? 0 : XsType<double>::fixed(Xs[c4 + e][r], fm), d[e]);
  uint8_t* const w0 =
      reinterpret_cast<uint8_t*>(x.ws) + 128 * (x.row0[it.front] + (int64_t)(c4 >> 4) * n + row) + 2 * (c4 & 15);
#pragma unroll
  for (int p = 0; p < S; ++p)
    *reinterpret_cast<uint2*>(w0 + 128 * (int64_t)((p >> 2) * 4) * n + 32 * (p & 3)) =
        make_uint2(__byte_perm(d[0][p], d[1][p], 0x7632), __byte_perm(d[2][p], d[3][p], 0x7632));
}

void launch_xs_trsm(const DevCtx& c, const XsCtx& x, const Item* items, int n_items, cudaStream_t s) {
  if (!n_items) return;
  k_xs_trsm64<<<n_items, 256, 0, s>>>(c, x, items);
}

// ---------------------------------------------------------------------------
// update
// ---------------------------------------------------------------------------
constexpr int XS_EPI_WARPS = 16;
constexpr int XS_THREADS = 32 * (XS_EPI_WARPS + 2);     // epilogue warps, TMA producer, MMA issuer
constexpr uint32_t XS_BOX = 128 * 128;                  // 128 rows of four slices x 16 columns = 16 KB
constexpr uint32_t XS_SLOT = 2 * XS_BOX;                // four slices of A and of B, 16 columns
constexpr int XS_SLOTS = 7;
constexpr uint32_t XS_SMEM = 1024 + XS_SLOTS * XS_SLOT + 512;
static_assert(8 * (2 * XS_SLOTS + 13) + 8 * XS_EPI_WARPS <= 512, "barriers and the epilogue's words");

#define XS_LD16(taddr, v)                                                                        \
  asm volatile(                                                                                  \
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14," \
      "%15}, [%16];"                                                                              \
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),      \
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),   \
        "=r"(v[14]), "=r"(v[15])                                                                  \
      : "r"(taddr))

#define XS_LD8(taddr, v)                                                                          \
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"          \
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]),          \
                 "=r"(v[6]), "=r"(v[7])                                                           \
               : "r"(taddr))

// One tile takes S = 8 (FP64) in two passes over its columns: diagonals 4 ..
// 7 (26 products of all slices), then diagonals 0 .. 3 (10 products of slices
// 0 .. 3); S = 4 (FP32) only the second pass.  Diagonal d goes to accumulator
// d mod 4, 128 x 128 FP32; the four fill tensor memory.

// a += i 2^SH
template <int SH>
__device__ __forceinline__ void xs_add(long long& a, int i) {
  if constexpr (SH < 31) {
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(a) : "r"(i), "n"(1 << SH));
  } else {
    a += (long long)((unsigned long long)((unsigned)i << (SH - 32)) << 32);
  }
}

// FP32 tiles: conversions to integers run at 16 per clock and SM, additions at 128:
// the sum of an integer below 2^22 and 1.5 2^23 holds it in its low bits, as
// XS_MAGIC + v.  The sums of diagonals 0 .. 3 reach 0.75 2^24 (256 times two products of
// two 8-bit digits and two with a leading one of at most 64); beyond 2^22, a warp's
// vote, they are converted.  (FP64 tiles have no
// registers left for it.)
constexpr uint32_t XS_MAGIC = 0x4B400000u;
__device__ __forceinline__ void xs_ints(uint32_t taddr, uint32_t (&v)[4][8]) {
  uint32_t out = 0;
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[a][j] = __float_as_uint(__uint_as_float(v[a][j]) + 12582912.0f);
      out |= v[a][j] ^ XS_MAGIC;               // bits 23.. are clear within [2^23, 2^24)
    }
  if (__any_sync(0xffffffffu, out >> 23)) {
#pragma unroll
    for (int a = 0; a < 4; ++a) XS_LD8(taddr + a * XS_TILE, v[a]);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int j = 0; j < 8; ++j) v[a][j] = XS_MAGIC + (uint32_t)__float2int_rn(__uint_as_float(v[a][j]));
  }
}

// a 2^E, rounded to nearest (E may leave the exponent range).  FP64 without
// conversions, which run at the FP64 rate: the leading bit by clz, the bits
// below the 53rd rounded to even in integers.
__device__ __forceinline__ double xs_scaled(long long a, int E, double) {
  unsigned long long m = a < 0 ? 0ull - (unsigned long long)a : (unsigned long long)a;
  const int lz = __clzll((long long)m);
  const int e = 1023 + 63 - lz + E;
  if (m == 0) return 0.0;
  if ((unsigned)(e - 1) >= 2044u) {
    const int e1 = max(-2000, min(2000, E)) / 2, e2 = max(-2000, min(2000, E)) - e1;
    return __ll2double_rn(a) * __hiloint2double((1023 + e1) << 20, 0) * __hiloint2double((1023 + e2) << 20, 0);
  }
  m <<= lz;
  const unsigned rem = (unsigned)m & 0x7FFu;
  unsigned long long q = (m >> 11) + ((rem + ((unsigned)(m >> 11) & 1u)) > 0x400u ? 1u : 0u);
  q += (unsigned long long)(e - 1) << 52;      // the leading bit adds the last 1 to the exponent
  if (a < 0) q |= 1ull << 63;
  return __longlong_as_double((long long)q);
}
// |a| < 2^45: a = h 2^23 + l, |h| < 2^22, both exact in FP32 (as above, without a
// conversion), so that their sum rounds once
__device__ __forceinline__ float xs_scaled(long long a, int E, float) {
  const float h = __uint_as_float(XS_MAGIC + (uint32_t)(a >> 23)) - 12582912.0f;
  const float l = __uint_as_float(0x4B000000u | ((uint32_t)a & 0x7FFFFFu)) - 8388608.0f;
  const float x = fmaf(h, 8388608.0f, l);
  const int b = __float_as_int(x), f = (b >> 23) & 0xFF;
  if ((unsigned)(f + E - 1) < 253u && f) return __int_as_float(b + (E << 23));
  const int e1 = max(-240, min(240, E)) / 2, e2 = max(-240, min(240, E)) - e1;
  return x * __int_as_float((127 + e1) << 23) * __int_as_float((127 + e2) << 23);
}

// LU: the rows (bits of left[0]) and columns (left[1]) of this warp's 32 x NC entries
// that the slices do not serve: none of the panel columns near its own maximum is near the maximum of
// any row of the other operand (of the front's own rows, or of its shared ones,
// whichever the entries lie in; a panel that is zero there serves them).
template <int NC>
__device__ __forceinline__ void xs_check(const XsCtx& x, int front, int K0, int n, int fs, int nb, int use, int row,
                                         int rmax, int c0, int cmax, volatile uint32_t* left) {
  const int lane = threadIdx.x & 31, r0 = row - lane;
  const bool rin = row < rmax, cin = lane < NC && c0 + lane < cmax;
  const int64_t e0 = x.exp0[front], w0 = x.near0[front] + K0 / 32;
  const uint2* ma = reinterpret_cast<const uint2*>(x.masks + (e0 + (rin ? row : 0)) * (XS_NBO / 32));
  const uint2* mb = reinterpret_cast<const uint2*>(x.masks + (e0 + n + (cin ? c0 + lane : 0)) * (XS_NBO / 32));
  // (the unions over own rows, then over shared rows)
  const uint2* na = reinterpret_cast<const uint2*>(x.near + 4 * use * x.near_n + w0);
  const uint2* nbv = reinterpret_cast<const uint2*>(x.near + (4 * use + 2) * x.near_n + w0);
  const int64_t own = x.near_n / 2;
  uint32_t hr[2] = {0, 0}, hc[2] = {0, 0}, sa[2] = {0, 0}, sb[2] = {0, 0};
#pragma unroll 2
  for (int w = 0; w < nb / 64; ++w) {          // (every load of a round in flight)
    const uint2 a = ma[w], b = mb[w];
    uint2 pa[2], pb[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      pa[h] = na[w + h * own];
      pb[h] = nbv[w + h * own];
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      hr[h] |= (a.x & pb[h].x) | (a.y & pb[h].y);
      hc[h] |= (b.x & pa[h].x) | (b.y & pa[h].y);
      sa[h] |= pa[h].x | pa[h].y;
      sb[h] |= pb[h].x | pb[h].y;
    }
  }
  bool okr = true, okc = true;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const bool cols = h ? min(c0 + NC, cmax) > fs : c0 < fs, rows = h ? min(r0 + 32, rmax) > fs : r0 < fs;
    okr = okr && (!cols || hr[h] || !sb[h]);
    okc = okc && (!rows || hc[h] || !sa[h] || use == 2);
  }
  const uint32_t wr = __ballot_sync(0xffffffffu, rin && !okr), wc = __ballot_sync(0xffffffffu, cin && !okc);
  if (lane == 0) {
    left[0] = wr;
    left[1] = wc;
  }
  __syncwarp();
}
// the exponent of a row or column left to xs_plain: its slices' sums become zero
__device__ __forceinline__ int xs_exp(int e, bool left) { return left ? -(1 << 29) : e; }

// ... and their entries by multiply-adds in the front's precision, 64 columns of
// the panel at a time: a row's columns along the lanes, then a column's rows.
template <typename T, int NC>
__device__ __noinline__ void xs_plain(T* G, int n, int K0, int W, int row, int rmax, int c0, int cmax,
                                      volatile uint32_t* left) {
  const int lane = threadIdx.x & 31, row0 = row - lane;
  const uint32_t wr = left[0], wc = left[1];
  __syncwarp();                                // C, unchanged in these rows and columns, is stored
  auto entry = [&](int r, int col) {
    T v = __ldcg(G + r + (int64_t)col * n);
    const T* __restrict__ l = G + r + (int64_t)K0 * n;
    const T* __restrict__ u = G + K0 + (int64_t)col * n;
    for (int k0 = 0; k0 < W; k0 += 64) {
      const int k1 = min(k0 + 64, W);
      T s = T(0);
#pragma unroll 16
      for (int k = k0; k < k1; ++k) s += l[(int64_t)k * n] * u[k];
      v -= s;
    }
    G[r + (int64_t)col * n] = v;
  };
  for (uint32_t m = wr; m; m &= m - 1)
    if (lane < NC && c0 + lane < cmax) entry(row0 + __ffs(m) - 1, c0 + lane);
  for (uint32_t m = wc; m; m &= m - 1)
    if (row < rmax && !(wr >> lane & 1)) entry(row, c0 + __ffs(m) - 1);
}

// Persistent: one CTA per SM walks the 128 x 128 tiles.  Warp 16 loads four
// slices of A and B (16 columns, 128-byte swizzle) per ring slot, one thread of
// warp 17 issues the products of a chunk,
// warps 0..15 (a lane quarter and 32 columns each) take the accumulators to
// 64-bit integers in registers while the next pass runs, then update C
// (column by column: a warp's loads and stores are 32 consecutive rows).
// Seven slots of 32 KB.  The four slices share
// 128-byte rows because TMA takes a row at a time: with 32-byte rows a tile of K =
// 256 took 64 us, with 64- and 128-byte ones 42, with the converged issue loop
// (umma_bf16_w) 30, with slice p of A kept in the collector buffer for its products
// (umma_bf16_wa) 27.5; FP32 tiles 13.1, then 11.9.  The tensor pipe alone needs 21 (6):
// a 128 x 128 x 16 product reads 8 KB at 128 B a clock, as long as it takes, and the
// loads (48 slots; 16) write beside it. 
// FP32 tiles load C while their products run and read the four diagonals eight columns
// at a time.  BN = 64: tiles of half the width
// for launches with fewer 128 x 128 tiles than SMs, where a tile's own time
// counts: half the products and half the FP64 additions of the epilogue, whose C
// entries are loaded while the products run.  Bound: shared-memory
// reads of the 128 x 128 products; a tile of a small launch by its epilogue.
// Measured on GB300 for up to 80 tiles
// of K = 64 (256): 29 (60) us with whole tiles, 18 (31) with these.
// Registers: 18 warps are allotted as 20, which leaves 96 a thread; the compiler spills up to 260
// bytes of <double, 128>, 72 of <double, 64> and 88 of the FP32 forms, all of epilogue warps.
template <typename T, int BN, bool LOWER>
__global__ void __launch_bounds__(XS_THREADS, 1)
k_xs_update(DevCtx c, XsCtx x, const __grid_constant__ XsMaps maps, const Item* __restrict__ items, int n_items,
            int nb, int region, int* err) {
  constexpr bool lower = LOWER;
  constexpr int S = XsType<T>::S;
  extern __shared__ __align__(1024) uint8_t xs_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(xs_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + XS_SLOTS * XS_SLOT);
  uint64_t* empty = bars + XS_SLOTS;
  uint64_t* acc_full = empty + XS_SLOTS;
  uint64_t* acc_empty = acc_full + 4;
  uint64_t* drain_bar = acc_empty + 4;
  volatile int* s_abort = reinterpret_cast<volatile int*>(drain_bar + 1);
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(drain_bar + 2);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < XS_SLOTS; ++s) {
      mbar_init(smem_u32(&bars[s]), 1);
      mbar_init(smem_u32(&empty[s]), 1);
    }
    for (int b = 0; b < 4; ++b) {
      mbar_init(smem_u32(&acc_full[b]), 1);
      mbar_init(smem_u32(&acc_empty[b]), XS_EPI_WARPS);
    }
    mbar_init(smem_u32(drain_bar), 1);
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *s_tmem;
  const uint32_t lim = g_wait_limit;

  if (warp == XS_EPI_WARPS) {
    if (lane == 0) {
      // TMA producer
      int s = 0;
      uint32_t ph = 1;               // parity of the empty wait (the first round passes)
      uint32_t issued = 0;
      bool live = true;
      for (int t = blockIdx.x; t < n_items && live; t += gridDim.x) {
        const Item it = items[t];
        const FrontDev f = c.fronts[it.front];
        const int n = f.n, nch = xs_chunks(nb, f.fs);
        const int nk = (min(nb, f.fs - it.c) + 15) / 16;
        const int64_t ya = x.row0[it.front] + it.a;
        const int64_t yb = (lower ? x.row0[it.front] : x.row0b[it.front]) + it.b;
        for (int pass = S == 8 ? 0 : 1; pass < 2 && live; ++pass) {
          const int np = pass == 0 ? 2 : 1;      // groups of four slices
          for (int k = 0; k < nk && live; ++k)
            for (int p = 0; p < np; ++p) {
              if (issued >= XS_SLOTS &&
                  !mbar_wait_lim(smem_u32(&empty[s]), ph, s_abort, err, XS_ERR, lim)) {
                live = false;
                break;
              }
              const uint32_t fb = smem_u32(&bars[s]), st = smem_u32(smem + s * XS_SLOT);
              mbar_expect_tx(fb, XS_BOX + BN * 128);
              const int64_t dr = (int64_t)(p * 4 * nch + k) * n;
              tma_load_2d(st, &maps.m128, 0, (int)(ya + dr), fb);
              tma_load_2d(st + XS_BOX, BN == 128 ? &maps.m128 : &maps.m64, 0, (int)(yb + dr), fb);
              ++issued;
              if (++s == XS_SLOTS) { s = 0; ph ^= 1; }
            }
        }
      }
      // the last loads issued (one per slot at most) land before the CTA exits
      const uint32_t cnt = issued < XS_SLOTS ? issued : XS_SLOTS;
      for (uint32_t q = issued - cnt; q < issued; ++q)
        mbar_drain(smem_u32(&bars[q % XS_SLOTS]), (q / XS_SLOTS) & 1);
    }
  } else if (warp == XS_EPI_WARPS + 1) {
    // MMA issuer: the whole warp, one elected lane issuing
    const uint32_t elected = elect_one();
    const uint32_t idesc = idesc_bf16_f32(XS_TILE, BN);
    const uint32_t ring = smem_u32(smem), bar0 = smem_u32(bars), acc_bar = smem_u32(acc_full);
    int s = 0;
    uint32_t ph = 0;               // parity of the full wait at slot s
    uint32_t used = 0, par = 0;    // bit a: accumulator a has been used / parity of its next reuse
    bool live = true;
    auto wait = [&](uint32_t bar, uint32_t parity) {
      return __all_sync(0xffffffffu, mbar_wait_lim(bar, parity, s_abort, err, XS_ERR, lim)) != 0;
    };
    // the products of diagonal d of one chunk, slices 0..3 in slot s0 and 4..7 in s1
    auto diag = [&](auto dd, uint32_t s0, uint32_t s1, int k, int nk) {
      constexpr int d = decltype(dd)::value, a = d & 3, np = d >= 4 ? S : 4;
      if (k == 0) {
        if ((used >> a) & 1) {
          if (!wait(acc_bar + 8 * (4 + a), (par >> a) & 1)) return false;
          par ^= 1u << a;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        used |= 1u << a;
      }
      const uint32_t acc = tmem + a * XS_TILE;
      uint32_t on = k == 0 ? 0u : 1u;
#pragma unroll
      for (int p = 0; p <= d; ++p) {
        const int q = d - p;
        if (p >= np || q >= np) continue;
        umma_bf16_w(elected, acc, (p < 4 ? s0 : s1) + 2 * (p & 3), (q < 4 ? s0 : s1) + (XS_BOX >> 4) + 2 * (q & 3),
                    SDESC_SW128_HI, idesc, on);
        on = 1u;
      }
      // the last chunk hands each accumulator over as soon as its diagonal is
      // issued, so that the epilogue reads one while the others fill
      if (k == nk - 1) umma_commit_w(elected, acc_bar + 8 * a);
      return true;
    };
    // between the first and the last chunk: the products of diagonals D0 .. D0 + 3
    // slice of A by slice of A, which is read from shared memory once
    auto inner = [&](auto dd, uint32_t s0, uint32_t s1) {
      constexpr int D0 = decltype(dd)::value, np = D0 ? S : 4;
#pragma unroll
      for (int p = 0; p < np; ++p) {
        constexpr int LAST = D0 + 3;
        const int qa = D0 > p ? D0 - p : 0, qb = LAST - p;       // slices of B: qa .. qb
        const uint32_t alo = (p < 4 ? s0 : s1) + 2 * (p & 3);
#pragma unroll
        for (int q = 0; q < np; ++q) {
          if (q < qa || q > qb) continue;
          const uint32_t blo = (q < 4 ? s0 : s1) + (XS_BOX >> 4) + 2 * (q & 3), acc = tmem + ((p + q) & 3) * XS_TILE;
          if (qa == qb) umma_bf16_w(elected, acc, alo, blo, SDESC_SW128_HI, idesc, 1u);
          else if (q == qa) umma_bf16_wa<UMMA_A_FILL>(elected, acc, alo, blo, SDESC_SW128_HI, idesc);
          else if (q == qb) umma_bf16_wa<UMMA_A_LAST>(elected, acc, alo, blo, SDESC_SW128_HI, idesc);
          else umma_bf16_wa<UMMA_A_USE>(elected, acc, alo, blo, SDESC_SW128_HI, idesc);
        }
      }
    };
    auto lo_of = [&](int q) { return sdesc_lo(ring + (uint32_t)q * XS_SLOT); };
    for (int t = blockIdx.x; t < n_items && live; t += gridDim.x) {
      const Item it = items[t];
      const int nk = __shfl_sync(0xffffffffu, (min(nb, c.fronts[it.front].fs - it.c) + 15) / 16, 0);
      if constexpr (S == 8) {
        for (int k = 0; k < nk && live; ++k) {
          const int q = s + 1 == XS_SLOTS ? 0 : s + 1;
          const uint32_t qp = q ? ph : ph ^ 1;
          live = wait(bar0 + 8 * s, ph) && wait(bar0 + 8 * q, qp);
          if (!live) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t s0 = lo_of(s), s1 = lo_of(q);
          if (k > 0 && k < nk - 1) {
            inner(std::integral_constant<int, 4>{}, s0, s1);
          } else {
            live = diag(std::integral_constant<int, 4>{}, s0, s1, k, nk) &&
                   diag(std::integral_constant<int, 5>{}, s0, s1, k, nk) &&
                   diag(std::integral_constant<int, 6>{}, s0, s1, k, nk) &&
                   diag(std::integral_constant<int, 7>{}, s0, s1, k, nk);
          }
          umma_commit_w(elected, bar0 + 8 * (XS_SLOTS + s));
          umma_commit_w(elected, bar0 + 8 * (XS_SLOTS + q));
          s = q + 1 == XS_SLOTS ? 0 : q + 1;
          ph = s ? qp : qp ^ 1;
        }
      }
      for (int k = 0; k < nk && live; ++k) {
        live = wait(bar0 + 8 * s, ph);
        if (!live) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t s0 = lo_of(s);
        if (k > 0 && k < nk - 1) {
          inner(std::integral_constant<int, 0>{}, s0, s0);
        } else {
          live = diag(std::integral_constant<int, 0>{}, s0, s0, k, nk) &&
                 diag(std::integral_constant<int, 1>{}, s0, s0, k, nk) &&
                 diag(std::integral_constant<int, 2>{}, s0, s0, k, nk) &&
                 diag(std::integral_constant<int, 3>{}, s0, s0, k, nk);
        }
        umma_commit_w(elected, bar0 + 8 * (XS_SLOTS + s));
        if (++s == XS_SLOTS) { s = 0; ph ^= 1; }
      }
    }
    // every MMA issued has completed before tensor memory is freed
    umma_commit_w(elected, smem_u32(drain_bar));
    mbar_drain(smem_u32(drain_bar), 0);
  } else {
    // epilogue
    constexpr int NC = BN / 4;       // columns per thread
    const int quarter = warp & 3, cg = warp >> 2;
    const uint32_t tbase = tmem + ((uint32_t)(quarter * 32) << 16) + cg * NC;
    // LU: what of the warp's entries is left to xs_plain (in shared memory: no register is
    // free while the accumulators are read)
    volatile uint32_t* const left = reinterpret_cast<volatile uint32_t*>(drain_bar + 4) + 2 * warp;
    uint32_t par = 0;              // bit a: parity of the next use of accumulator a
    bool live = true;
    for (int t = blockIdx.x; t < n_items && live; t += gridDim.x) {
      const Item it = items[t];
      const FrontDev& f = c.fronts[it.front];
      const int n = f.n, K0 = it.c;
      const int Bnd = region ? min((K0 / XS_NBO) * XS_NBO + XS_NBO, f.fs) : n;
      const int rmax = region == 2 ? Bnd : n, cmax = region == 1 ? Bnd : n;
      const int row = it.a + quarter * 32 + lane, c0 = it.b + cg * NC;
      // columns c0 + j, j < cend, of this thread's row are updated
      const int cend = row < rmax ? min(cmax, lower ? row + 1 : cmax) - c0 : 0;
      T* __restrict__ G = arena<T>(c) + f.off + row + (int64_t)c0 * n;
      if constexpr (S == 4 && BN == 128) {
        // FP32: the products of a tile take less time than eight rounds of C
        // accesses; C is loaded while they run, and the four diagonals are read
        // eight columns at a time
        T cv[NC];
#pragma unroll
        for (int j = 0; j < NC; ++j) cv[j] = j < cend ? __ldcg(G + (int64_t)j * n) : T(0);
        if constexpr (!lower) xs_check<NC>(x, it.front, K0, n, f.fs, nb, region, row, rmax, c0, cmax, left);
        const int* __restrict__ ex = x.exps + x.exp0[it.front];
        const int ea = cend > 0 ? xs_exp(ex[row], !lower && (left[0] >> lane & 1)) - 36 : 0;
        const int ebl = c0 + lane < cmax ? xs_exp(ex[(lower ? 0 : n) + c0 + lane], !lower && (left[1] >> lane & 1)) : 0;  // NC = 32 lanes
#pragma unroll
        for (int a = 0; a < 4; ++a)
          live = live && mbar_wait_lim(smem_u32(&acc_full[a]), par & 1, s_abort, err, XS_ERR, lim);
        live = __all_sync(0xffffffffu, live);
        if (!live) break;
        par ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int h = 0; h < NC / 8; ++h) {
          uint32_t v[4][8];
#pragma unroll
          for (int a = 0; a < 4; ++a) XS_LD8(tbase + a * XS_TILE + 8 * h, v[a]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          xs_ints(tbase + 8 * h, v);
          if (h == NC / 8 - 1) {
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane < 4) mbar_arrive(smem_u32(&acc_empty[lane]));
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            long long s4 = -(long long)XS_MAGIC * 0x1010101ll;
            xs_add<24>(s4, (int)v[0][j]);
            xs_add<16>(s4, (int)v[1][j]);
            xs_add<8>(s4, (int)v[2][j]);
            xs_add<0>(s4, (int)v[3][j]);
            const int E = ea + __shfl_sync(0xffffffffu, ebl, 8 * h + j);
            T d = xs_scaled(s4, E, T(0));
            if (E > XS_BAD / 2) d = T(NAN);
            cv[8 * h + j] -= d;
          }
        }
        if (*s_abort) break;
#pragma unroll
        for (int j = 0; j < NC; ++j)
          if (j < cend) G[(int64_t)j * n] = cv[j];
        if constexpr (!lower)
          if (left[0] | left[1]) xs_plain<T, NC>(arena<T>(c) + f.off, n, K0, min(nb, f.fs - K0), row, rmax, c0, cmax, left);
        continue;
      }
      constexpr bool EARLY = BN == 64;
      T ce[EARLY ? NC : 1];
      if constexpr (EARLY) {
#pragma unroll
        for (int j = 0; j < NC; ++j) ce[j] = j < cend ? __ldcg(G + (int64_t)j * n) : T(0);
      }
      if constexpr (!lower) xs_check<NC>(x, it.front, K0, n, f.fs, nb, region, row, rmax, c0, cmax, left);
      long long acc[NC];
#pragma unroll
      for (int j = 0; j < NC; ++j) acc[j] = 0;
      auto take = [&](auto dd) {
        constexpr int d = decltype(dd)::value, a = d & 3;
        constexpr int SH = d >= 4 ? 8 * (7 - d) : 8 * (3 - d) + (S == 8 ? 18 : 0);
        if (!mbar_wait_lim(smem_u32(&acc_full[a]), (par >> a) & 1, s_abort, err, XS_ERR, lim)) return false;
        par ^= 1u << a;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int h = 0; h < NC / 16; ++h) {
          uint32_t v[16];
          XS_LD16(tbase + a * XS_TILE + 16 * h, v);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (h == NC / 16 - 1) {
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&acc_empty[a]));
          }
#pragma unroll
          for (int j = 0; j < 16; ++j) xs_add<SH>(acc[16 * h + j], __float2int_rn(__uint_as_float(v[j])));
        }
        return true;
      };
      if constexpr (S == 8) {
        // the low diagonals, then rounded to the last place kept
        live = take(std::integral_constant<int, 4>{}) && take(std::integral_constant<int, 5>{}) &&
               take(std::integral_constant<int, 6>{}) && take(std::integral_constant<int, 7>{});
#pragma unroll
        for (int j = 0; j < NC; ++j) acc[j] = (acc[j] + (1 << 13)) >> 14;
      }
      live = live && take(std::integral_constant<int, 0>{}) && take(std::integral_constant<int, 1>{}) &&
             take(std::integral_constant<int, 2>{}) && take(std::integral_constant<int, 3>{});
      if (!live || *s_abort) break;
      // C -= acc 2^(ea + eb - 54) (FP32: - 36); |acc| < 2^62 (2^44)
      if (cend > 0) {
        const int* __restrict__ ex = x.exps + x.exp0[it.front];
        const int* __restrict__ ebp = ex + (lower ? 0 : n) + c0;
        const int ea = xs_exp(ex[row], !lower && (left[0] >> lane & 1)) - (S == 8 ? 54 : 36);
        const uint32_t wc = lower ? 0u : left[1];
#pragma unroll
        for (int j0 = 0; j0 < NC; j0 += 4) {
          T cv[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if constexpr (EARLY) cv[j] = ce[j0 + j];
            else cv[j] = j0 + j < cend ? __ldcg(G + (int64_t)j * n) : T(0);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (j0 + j < cend) {
              const int E = ea + xs_exp(__ldg(ebp + j0 + j), !lower && (wc >> (j0 + j) & 1));
              T d = xs_scaled(acc[j0 + j], E, T(0));
              if (E > XS_BAD / 2) d = T(NAN);
              G[(int64_t)j * n] = cv[j] - d;
            }
          G += 4 * (int64_t)n;
        }
      }
      if constexpr (!lower)
        if (left[0] | left[1]) xs_plain<T, NC>(arena<T>(c) + f.off, n, K0, min(nb, f.fs - K0), row, rmax, c0, cmax, left);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

bool xs_encode(XsMaps* maps, void* base, int64_t rows) {
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  if (!encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn) {
      cudaGetLastError();
      return false;
    }
    encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }
  cuuint64_t dims[2] = {64, (cuuint64_t)rows};
  cuuint64_t strides[1] = {128};
  cuuint32_t estr[2] = {1, 1};
  for (int h = 0; h < 2; ++h) {
    cuuint32_t box[2] = {64, h ? 64u : 128u};
    if (encode(h ? &maps->m64 : &maps->m128, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return false;
  }
  return true;
}

template <typename T, int BN, bool LOWER>
static void xs_update_t(const DevCtx& c, const XsCtx& x, const XsMaps& maps, const Item* items, int n_items,
                        int nb, int region, int cap, int* err, cudaStream_t s) {
  static int n_sm = 0;
  if (!n_sm) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
    if (n_sm <= 0) n_sm = 1;
  }
  cudaFuncSetAttribute(k_xs_update<T, BN, LOWER>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)XS_SMEM);
  const int sms = cap > 0 && cap < n_sm ? cap : n_sm;
  const int grid = n_items < sms ? n_items : sms;
  k_xs_update<T, BN, LOWER><<<grid, XS_THREADS, XS_SMEM, s>>>(c, x, maps, items, n_items, nb, region, err);
}

void launch_xs_update(const DevCtx& c, const XsCtx& x, const XsMaps& maps, const Item* items, int n_items,
                      int dtype, int nb, int region, int lower, int tile_n, int cap, int* err, cudaStream_t s) {
  if (!n_items) return;
  if (nb > XS_NBO) throw std::invalid_argument("sliced update: panel wider than 256");
  if (tile_n != 64 && tile_n != XS_TILE) throw std::invalid_argument("sliced update: tiles are 64 or 128 columns wide");
  if (!lower && !x.near) throw std::invalid_argument("sliced update: LU operands without their check");
  const auto run = [&](auto t, auto low) {
    using T = decltype(t);
    constexpr bool L = decltype(low)::value;
    if (tile_n == 64) xs_update_t<T, 64, L>(c, x, maps, items, n_items, nb, region, cap, err, s);
    else xs_update_t<T, XS_TILE, L>(c, x, maps, items, n_items, nb, region, cap, err, s);
  };
  if (dtype == F64 && lower) run(double(), std::true_type());
  else if (dtype == F64) run(double(), std::false_type());
  else if (lower) run(float(), std::true_type());
  else run(float(), std::false_type());
}

}  // namespace uhm_gpu
