// Front assembly (extend-add) and partial factorisation kernels, SIMT path.
//
// Reference steps restated here:
//   extend-add      Helper_::_merge_A -> Matrix_FLA_::merge (FLA_Axpy of
//                   sub-blocks), UHM/include/uhm/matrix/uhm/helper.hxx:191-222,
//                   UHM/src/matrix/uhm/fla/matrix.cxx:284-303; element scatter
//                   of Mesh_::copy_in, UHM/src/mesh/interf.cxx:108-204
//   Cholesky front  chol_hier, UHM/src/matrix/uhm/fla/chol/decompose.cxx:85-98
//                   (LINAL/src/dense/chol.cxx:46-92, trsm.cxx:221-247, syrk.cxx:58-90)
//   LU fronts       lu_piv_hier / lu_nopiv_hier, fla/lu_piv/decompose.cxx:124-153,
//                   fla/lu_nopiv/decompose.cxx:95-121 (pivot search restricted to
//                   the ATL rows, LINAL/src/dense/lu_piv.cxx:47-111)
//
// The extend-add is a parent-centric gather: every parent entry is written
// exactly once as  0 + sum over sources in source order  (element
// contributions, then children in child order), which is the reference's
// summation order onto a zeroed parent; no atomics, bitwise reproducible.
// The sum is formed in the front's precision: FP64 fronts in FP64, FP32
// fronts in FP32 (FP64 arithmetic runs at a small fraction of the FP32 rate
// on this GPU, and the FP32 front stores the sum in FP32 either way).
#include <cstddef>
#include <cstdio>
#include <stdexcept>
#include <string>
#include "k_common.cuh"
#include "k_potrf.cuh"
#include "k_xs_slices.cuh"

namespace uhm_gpu {

// ---------------------------------------------------------------------------
// assembly
// ---------------------------------------------------------------------------
constexpr int ASM_TJ = 16;
constexpr int ASM_MAXSRC = 64;

// Extend-add of a front below ASM_SCATTER_MIN rows: 16 parent columns per
// CTA, one thread per parent row, the column's sources walked in summation
// order (element first, then the children in child order) through their
// inverse row maps.  Each parent entry is written once; a child's
// lower-stored Schur block is read transposed where the parent row falls
// above its diagonal.  (Forms with several rows per thread, or a warp per
// column with the sources decoded once per pass, issued more instructions
// per entry on these front sizes and measured slower.)
template <typename T>
__global__ void __launch_bounds__(256) k_assemble(DevCtx c, const Item* __restrict__ items,
                                                  int lower) {
  __shared__ SrcDev s_src[ASM_MAXSRC];
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n;
  const int nsrc = f.nsrc;
  for (int s = threadIdx.x; s < nsrc && s < ASM_MAXSRC; s += blockDim.x) s_src[s] = c.srcs[f.src0 + s];
  __syncthreads();
  T* __restrict__ P = arena<T>(c) + f.off;
  const int64_t* __restrict__ cp = c.colptr + f.colptr_off;
  const int32_t* __restrict__ inv = c.inv + f.inv_off;
  const int J0 = it.a;
  const int J1 = min(J0 + ASM_TJ, n);
  for (int J = J0; J < J1; ++J) {
    const int64_t k0 = cp[J], k1 = cp[J + 1];
    const int istart = lower ? J : 0;
    for (int I = istart + threadIdx.x; I < n; I += blockDim.x) {
      T acc = T(0);
      for (int64_t k = k0; k < k1; ++k) {
        const int2 cs = c.colsrc[k];
        const int is = inv[(int64_t)cs.x * n + I];
        if (is >= 0) {
          const SrcDev sd = cs.x < ASM_MAXSRC ? s_src[cs.x] : c.srcs[f.src0 + cs.x];
          int r = is, cc = cs.y;
          if (sd.is_child && c.symmetric && r < cc) { int t = r; r = cc; cc = t; }
          acc += (T)load_src(c, sd, r + (int64_t)cc * sd.ld);
        }
      }
      P[I + (int64_t)J * n] = acc;
    }
  }
}

// Extend-add of a large front, one parent column J per CTA.  The column is
// accumulated in shared memory (in the front's precision): zero, then each source holding
// column J in source order (the element, then the children in child order)
// scatters its column through its row map (an injective map, so a source
// never hits the same entry twice and one barrier between sources keeps the
// order); then the column is written once.  Every entry therefore gets the
// same sum in the same order as in k_assemble (bit-identical), but each
// source entry is read once instead of every parent row looking up every
// source.  NT threads, four rows each per pass.  EARLY: a child's stored
// part of its column (rows at or below its diagonal, every row of an
// unsymmetric child) is read beside the row-map look-up instead of after it
// (only rows stored transposed, and element rows, wait for their parent row
// to be known); it paid on the root's launch (fronts above ASM_EARLY_MIN
// rows, 512 threads) and not on the levels below.
constexpr int ASM_EARLY_MIN = 8192;

template <typename T, int NT, bool EARLY>
__global__ void __launch_bounds__(NT) k_assemble_scatter(DevCtx c, const Item* __restrict__ items, int lower) {
  extern __shared__ __align__(16) unsigned char sc_raw[];
  T* s_col = reinterpret_cast<T*>(sc_raw);
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, J = it.a;
  const int istart = lower ? J : 0;
  for (int I = istart + threadIdx.x; I < n; I += NT) s_col[I] = T(0);
  const int64_t* __restrict__ cp = c.colptr + f.colptr_off;
  const int64_t k0 = cp[J], k1 = cp[J + 1];
  __syncthreads();
  for (int64_t k = k0; k < k1; ++k) {
    const int2 cs = c.colsrc[k];
    const SrcDev sd = c.srcs[f.src0 + cs.x];
    const int32_t* __restrict__ fw = c.fwd + sd.fwd_off;
    const bool sym = sd.is_child && c.symmetric;
    // the source decoded once; per pass every thread issues all its map
    // look-ups, then all its loads, then the shared-memory adds
    const double* __restrict__ b64 = !sd.is_child ? c.emat + sd.off : (sd.dtype == F64 ? c.a64 + sd.off : nullptr);
    const float* __restrict__ b32 = (sd.is_child && sd.dtype != F64) ? c.a32 + sd.off : nullptr;
    const int cc = cs.y;
    // rows r >= rs are stored in column cc and read at once (EARLY)
    const int rs = !EARLY ? sd.m : (sd.is_child ? (sym ? cc : 0) : sd.m);
    for (int r0 = 0; r0 < sd.m; r0 += 4 * NT) {
      int I[4];
      T v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = r0 + threadIdx.x + NT * u;
        I[u] = r < sd.m ? __ldg(fw + r) : -1;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = r0 + threadIdx.x + NT * u;
        v[u] = T(0);
        if (r < sd.m && r >= rs) {
          const int64_t idx = r + (int64_t)cc * sd.ld;
          v[u] = b32 ? (T)b32[idx] : (T)b64[idx];
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = r0 + threadIdx.x + NT * u;
        if (I[u] >= istart) {
          if (r < rs) {
            int rr = r, cl = cc;
            if (sym && rr < cl) { const int t = rr; rr = cl; cl = t; }
            const int64_t idx = rr + (int64_t)cl * sd.ld;
            v[u] = b32 ? (T)b32[idx] : (T)b64[idx];
          }
          s_col[I[u]] += v[u];
        }
      }
    }
    __syncthreads();
  }
  T* __restrict__ P = arena<T>(c) + f.off + (int64_t)J * n;
  for (int I = istart + threadIdx.x; I < n; I += NT) P[I] = s_col[I];
}

template <typename T>
static void assemble_scatter_t(const DevCtx& c, const Item* items, int n_items, int lower, int n_max,
                               cudaStream_t s) {
  const size_t sm = sizeof(T) * (size_t)n_max;
  if (n_max >= ASM_EARLY_MIN) {
    cudaFuncSetAttribute(k_assemble_scatter<T, 512, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_assemble_scatter<T, 512, true><<<n_items, 512, sm, s>>>(c, items, lower);
  } else {
    cudaFuncSetAttribute(k_assemble_scatter<T, 256, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_assemble_scatter<T, 256, false><<<n_items, 256, sm, s>>>(c, items, lower);
  }
}

void launch_assemble_scatter(const DevCtx& c, const Item* items, int n_items, int dtype, int lower,
                             int n_max, cudaStream_t s) {
  if (!n_items) return;
  if (dtype == F64) assemble_scatter_t<double>(c, items, n_items, lower, n_max, s);
  else assemble_scatter_t<float>(c, items, n_items, lower, n_max, s);
}

void launch_assemble(const DevCtx& c, const Item* items, int n_items, int dtype, int lower,
                     cudaStream_t s) {
  if (!n_items) return;
  if (dtype == F64) k_assemble<double><<<n_items, 256, 0, s>>>(c, items, lower);
  else k_assemble<float><<<n_items, 256, 0, s>>>(c, items, lower);
}

// ---------------------------------------------------------------------------
// block-wide argmax |v| (ties -> smaller index), for partial pivoting
// ---------------------------------------------------------------------------
template <typename T, int NT>
__device__ int block_argmax(T best, int bi, T* s_v, int* s_i) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    T ov = __shfl_down_sync(0xffffffffu, best, o);
    int oi = __shfl_down_sync(0xffffffffu, bi, o);
    if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
  }
  if (lane == 0) { s_v[warp] = best; s_i[warp] = bi; }
  __syncthreads();
  if (warp == 0) {
    best = lane < NT / 32 ? s_v[lane] : (T)-1;
    bi = lane < NT / 32 ? s_i[lane] : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      T ov = __shfl_down_sync(0xffffffffu, best, o);
      int oi = __shfl_down_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    if (lane == 0) s_i[0] = bi;
  }
  __syncthreads();
  int r = s_i[0];
  __syncthreads();
  return r;
}

// ---------------------------------------------------------------------------
// whole-front partial factorisation in shared memory (one CTA per front)
// ---------------------------------------------------------------------------
template <typename T, int NT>
__global__ void __launch_bounds__(NT) k_small_factor(DevCtx c, const Item* __restrict__ items,
                                                     int method) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* A = reinterpret_cast<T*>(smem_raw);
  __shared__ T s_v[NT / 32];
  __shared__ int s_i[NT / 32];
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, fs = f.fs;
  T* __restrict__ G = arena<T>(c) + f.off;
  const bool chol = method == M_CHOL;
  const bool pivot = method == M_LU_PIV;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int NW = NT / 32;
  // the front in (its lower triangle for Cholesky): a warp per column, no
  // index division
  for (int j = warp; j < n; j += NW)
    for (int i = (chol ? j : 0) + lane; i < n; i += 32) A[i + (int64_t)j * n] = G[i + (int64_t)j * n];
  __syncthreads();
  for (int k = 0; k < fs; ++k) {
    if (chol) {
      if (threadIdx.x == 0) {
        T d = A[k + (int64_t)k * n];
        if (!(d > (T)0)) { set_status(c, it.front, d != d ? ST_NAN : ST_NOT_SPD); d = (T)1; }
        A[k + (int64_t)k * n] = my_sqrt<T>(d);
      }
      __syncthreads();
      const T dkk = A[k + (int64_t)k * n];
      for (int i = k + 1 + threadIdx.x; i < n; i += NT) A[i + (int64_t)k * n] /= dkk;
      __syncthreads();
      for (int j = k + 1 + warp; j < n; j += NW) {
        const T ajk = A[j + (int64_t)k * n];
        T* __restrict__ col = A + (int64_t)j * n;
        const T* __restrict__ colk = A + (int64_t)k * n;
        for (int i = j + lane; i < n; i += 32) col[i] -= colk[i] * ajk;
      }
      __syncthreads();
    } else {
      if (pivot) {
        T best = (T)-1;
        int bi = k;
        for (int i = k + threadIdx.x; i < fs; i += NT) {
          const T v = my_abs<T>(A[i + (int64_t)k * n]);
          if (v > best) { best = v; bi = i; }
        }
        const int p = block_argmax<T, NT>(best, bi, s_v, s_i);
        if (threadIdx.x == 0) c.piv[f.piv_off + k] = p;
        if (p != k)
          for (int j = threadIdx.x; j < n; j += NT) {
            T t = A[k + (int64_t)j * n];
            A[k + (int64_t)j * n] = A[p + (int64_t)j * n];
            A[p + (int64_t)j * n] = t;
          }
        __syncthreads();
      }
      T akk = A[k + (int64_t)k * n];
      if (akk == (T)0 || akk != akk) {
        if (threadIdx.x == 0) set_status(c, it.front, akk != akk ? ST_NAN : ST_ZERO_PIVOT);
        akk = (T)1;
      }
      for (int i = k + 1 + threadIdx.x; i < n; i += NT) A[i + (int64_t)k * n] /= akk;
      __syncthreads();
      for (int j = k + 1 + warp; j < n; j += NW) {
        const T akj = A[k + (int64_t)j * n];
        T* __restrict__ col = A + (int64_t)j * n;
        const T* __restrict__ colk = A + (int64_t)k * n;
        for (int i = k + 1 + lane; i < n; i += 32) col[i] -= colk[i] * akj;
      }
      __syncthreads();
    }
  }
  for (int j = warp; j < n; j += NW)
    for (int i = (chol ? j : 0) + lane; i < n; i += 32) G[i + (int64_t)j * n] = A[i + (int64_t)j * n];
}

// v / d from r, an approximation of 1 / d (to an ulp or two): the quotient and
// Markstein's correction by its remainder, rounded as a division but for rare
// ties.  (Products with the reciprocal root instead: an error of r is common to its
// whole column of L and, on a uniform mesh, to every element's front; the
// solutions of 12^3 and 16^3 p = 4 Poisson meshes were 1.3 and 1.5 times further
// from the exact ones than with a square root and divisions.)  An infinite
// d (r = 0) is given as 0: the quotients of finite numbers are then zero, as by division.
__device__ __forceinline__ double fp64_div(double v, double d, double r) {
  const double q = v * r;
  return fma(fma(-q, d, v), r, q);
}

// The factor panel of a small FP64 front in shared memory, four columns per
// step: one thread per row factors the 4 x 4 pivot block and substitutes its
// row, then 4 x 2 register tiles of the panel's lower triangle take the rank-4
// update.  Bound by the FP64 multiply-adds (2 per clock and SM: 85 us of them on
// a 125 x 125 front).  Measured on GB300 against an FP64 square root and division
// per column with a barrier on either side: that front 275 -> 242 us.
template <int NT>
__device__ __forceinline__ void small_panel4(const DevCtx& c, int front, double* __restrict__ A, int n, int fs) {
  const int tid = threadIdx.x;
  for (int P = 0; P < fs; P += 4) {
    const int w = min(4, fs - P), r = P + tid;
    double t[4];
    if (r < n) {
      double lb[4][4], rd[4], ld[4];
      bool inf[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        rd[m] = ld[m] = 1.0;
        inf[m] = false;
        if (m >= w) continue;
        double s = A[P + m + (P + m) * n];
#pragma unroll
        for (int l = 0; l < m; ++l) s -= lb[m][l] * lb[m][l];
        if (!(s > 0.0)) {
          if (tid == 0) set_status(c, front, s != s ? ST_NAN : ST_NOT_SPD);
          s = 1.0;
        }
        rd[m] = rsqrt(s);
        {
          const double h = s * rd[m];          // sqrt(s), corrected the same way
          const double e = fma(-h, h, s);
          ld[m] = fabs(e) < s ? fma(0.5 * rd[m], e, h) : h;
          inf[m] = (__double2hiint(s) & 0x7FF00000) == 0x7FF00000;
          if (inf[m]) ld[m] = 0.0;
        }
#pragma unroll
        for (int i = m + 1; i < 4; ++i) {
          double v = i < w ? A[P + i + (P + m) * n] : 0.0;
#pragma unroll
          for (int l = 0; l < m; ++l) v -= lb[i][l] * lb[m][l];
          lb[i][m] = fp64_div(v, ld[m], rd[m]);
        }
      }
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        double v = m < w ? A[r + (P + m) * n] : 0.0;
#pragma unroll
        for (int l = 0; l < m; ++l) v -= lb[m][l] * t[l];
        t[m] = r == P + m ? (inf[m] ? HUGE_VAL : ld[m]) : fp64_div(v, ld[m], rd[m]);
      }
    }
    __syncthreads();                     // the pivot block has been read
    if (r < n) {
#pragma unroll
      for (int m = 0; m < 4; ++m)
        if (m < w && r >= P + m) A[r + (P + m) * n] = t[m];
    }
    __syncthreads();
    // half tiles of the columns b .. fs-1, tile column j with its Rt - j row
    // tiles, counted column by column: unit e -> (j, i)
    const int b = P + 4, Rt = (n - b + 3) / 4, Ct = (fs - b + 3) / 4;
    const int units = Ct > 0 ? Ct * Rt - Ct * (Ct - 1) / 2 : 0;
    for (int e2 = tid; e2 < 2 * units; e2 += NT) {
      const int e = e2 >> 1;
      const float h = (float)Rt + 0.5f;
      int j = (int)(h - sqrtf(fmaxf(h * h - 2.f * (float)e, 0.f)));
      while (j > 0 && j * Rt - j * (j - 1) / 2 > e) --j;
      while ((j + 1) * Rt - (j + 1) * j / 2 <= e) ++j;
      const int r0 = b + 4 * (j + e - (j * Rt - j * (j - 1) / 2)), c0 = b + 4 * j + 2 * (e2 & 1);
      double a[4][2];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 2; ++v)
          a[u][v] = r0 + u < n && c0 + v < fs && r0 + u >= c0 + v ? A[r0 + u + (c0 + v) * n] : 0.0;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const double* __restrict__ col = A + (P + m) * n;
        double x[4], y[2];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = r0 + u < n ? col[r0 + u] : 0.0;
#pragma unroll
        for (int v = 0; v < 2; ++v) y[v] = c0 + v < n ? col[c0 + v] : 0.0;
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int v = 0; v < 2; ++v) a[u][v] -= x[u] * y[v];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 2; ++v)
          if (r0 + u < n && c0 + v < fs && r0 + u >= c0 + v) A[r0 + u + (c0 + v) * n] = a[u][v];
    }
    __syncthreads();
  }
}

// Cholesky fronts in shared memory, one CTA per front: the lower triangle is
// staged with eight loads in flight per thread; the fs factor columns are
// factored column by column as in k_small_factor (FP64: four at a time,
// small_panel4), but each step updates only the panel's later columns; the
// Schur block is then updated once from the
// factor panel in 4 x 4 register tiles, subtracting the fs products in
// column order -- the same operations in the same order as k_small_factor's
// rank-1 steps, with one shared-memory read and write per
// Schur entry instead of one per entry and step.
template <typename T, int NT>
__global__ void __launch_bounds__(NT) k_small_chol(DevCtx c, const Item* __restrict__ items) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* A = reinterpret_cast<T*>(smem_raw);
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, fs = f.fs;
  T* __restrict__ G = arena<T>(c) + f.off;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int NW = NT / 32;
  const int nn = n * n;
  // flat index e = i + j n walked in steps of NT with (i, j) kept by carry
  const int qs = NT / n, rs = NT % n;
  {
    int i0 = threadIdx.x % n, j0 = threadIdx.x / n;
    for (int e0 = 0; e0 < nn; e0 += 8 * NT) {
      T v[8];
      int i = i0, j = j0;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int e = e0 + threadIdx.x + u * NT;
        v[u] = (e < nn && i >= j) ? G[e] : T(0);
        i += rs; j += qs;
        if (i >= n) { i -= n; ++j; }
      }
      i = i0; j = j0;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int e = e0 + threadIdx.x + u * NT;
        if (e < nn && i >= j) A[e] = v[u];
        i += rs; j += qs;
        if (i >= n) { i -= n; ++j; }
      }
      i0 = i; j0 = j;
    }
  }
  __syncthreads();
  if constexpr (sizeof(T) == 8) {
    small_panel4<NT>(c, it.front, A, n, fs);
  } else {
    for (int k = 0; k < fs; ++k) {
      if (threadIdx.x == 0) {
        T d = A[k + k * n];
        if (!(d > (T)0)) { set_status(c, it.front, d != d ? ST_NAN : ST_NOT_SPD); d = (T)1; }
        A[k + k * n] = my_sqrt<T>(d);
      }
      __syncthreads();
      const T dkk = A[k + k * n];
      for (int i = k + 1 + threadIdx.x; i < n; i += NT) A[i + k * n] /= dkk;
      __syncthreads();
      for (int j = k + 1 + warp; j < fs; j += NW) {
        const T ajk = A[j + k * n];
        T* __restrict__ col = A + j * n;
        const T* __restrict__ colk = A + k * n;
        for (int i = j + lane; i < n; i += 32) col[i] -= colk[i] * ajk;
      }
      __syncthreads();
    }
  }
  // Schur block S (rows / columns fs .. n-1): S -= L21 L21^T by 4 x 4 tiles
  // of its lower triangle, tile t -> (ti, tj), ti >= tj
  const int m = n - fs, tm = (m + 3) / 4, ntile = tm * (tm + 1) / 2;
  for (int t = threadIdx.x; t < ntile; t += NT) {
    int ti = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);
    while (ti * (ti + 1) / 2 > t) --ti;
    while ((ti + 1) * (ti + 2) / 2 <= t) ++ti;
    const int tj = t - ti * (ti + 1) / 2;
    const int r0 = fs + 4 * ti, c0 = fs + 4 * tj;
    T acc[4][4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int i = r0 + u, j = c0 + v;
        acc[u][v] = (i < n && j < n && i >= j) ? A[i + j * n] : T(0);
      }
    for (int k = 0; k < fs; ++k) {
      const T* __restrict__ colk = A + k * n;
      T x[4], y[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        x[u] = r0 + u < n ? colk[r0 + u] : T(0);
        y[u] = c0 + u < n ? colk[c0 + u] : T(0);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v] -= x[u] * y[v];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int i = r0 + u, j = c0 + v;
        if (i < n && j < n && i >= j) A[i + j * n] = acc[u][v];
      }
  }
  __syncthreads();
  {
    int i0 = threadIdx.x % n, j0 = threadIdx.x / n;
    for (int e0 = 0; e0 < nn; e0 += 8 * NT) {
      int i = i0, j = j0;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int e = e0 + threadIdx.x + u * NT;
        if (e < nn && i >= j) G[e] = A[e];
        i += rs; j += qs;
        if (i >= n) { i -= n; ++j; }
      }
      i0 = i; j0 = j;
    }
  }
}

void launch_small_factor(const DevCtx& c, const Item* items, int n_items, int dtype, int method,
                         int max_n, cudaStream_t s) {
  if (!n_items) return;
  if (method == M_CHOL) {
    if (dtype == F64) {
      const size_t sm = (size_t)max_n * max_n * sizeof(double);
      cudaFuncSetAttribute(k_small_chol<double, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
      k_small_chol<double, 256><<<n_items, 256, sm, s>>>(c, items);
    } else {
      const size_t sm = (size_t)max_n * max_n * sizeof(float);
      cudaFuncSetAttribute(k_small_chol<float, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
      k_small_chol<float, 256><<<n_items, 256, sm, s>>>(c, items);
    }
    return;
  }
  if (dtype == F64) {
    size_t sm = (size_t)max_n * max_n * sizeof(double);
    cudaFuncSetAttribute(k_small_factor<double, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sm);
    k_small_factor<double, 256><<<n_items, 256, sm, s>>>(c, items, method);
  } else {
    size_t sm = (size_t)max_n * max_n * sizeof(float);
    cudaFuncSetAttribute(k_small_factor<float, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sm);
    k_small_factor<float, 256><<<n_items, 256, sm, s>>>(c, items, method);
  }
}

// ---------------------------------------------------------------------------
// blocked large-front Cholesky: diagonal block, panel TRSM, trailing update
// item: front, a = k0 (step start), b = row block / tile row, c = tile col
// ---------------------------------------------------------------------------
// Cholesky of one diagonal block (kb <= 64) and the inverse of its factor,
// 256 threads = 8 warps (potrf_block, shared by k_potrf_diag and the fused
// k_potrf_trsm).  Warp w owns the column block 8w..8w+7 of the symmetric
// 64 x 64 block and of the inverse X = L^{-1} being formed; lane (ti, h)
// keeps the 4 x 4 tile at rows 4 ti.., columns 8w + 4h.. of both in
// registers.  Right-looking, four columns P..P+3 per phase: the columns, as
// reduced by all earlier phases, were published in shared memory (V[P+j]);
// every thread factors their 4 x 4 pivot block itself, forms the factor
// entries of its 4 rows and 4 columns by a 4-step substitution
//   l_rj = (v_{P+j}[r] - sum_{m<j} l_rm l_{P+j,P+m}) / l_{P+j,P+j},
// and applies the rank-4 update A -= L_r L_c^T to its tile; the owners of
// columns P+4..P+7 then publish them.  In the same phase the owners of rows
// P..P+3 of X finish them with the pivot block's substitution and the other
// rows take the rank-4 update X -= L[:, P:P+4] X[P:P+4, :] (column blocks of
// X are independent, so rows go through shared memory per warp).  One block
// barrier per phase, 16 in all.  A warp does only the factor work that
// reaches its columns and only the inverse work whose rows are nonzero in
// them.  Blocks narrower than 64 are padded with the identity.  Pivots
// use rsqrt (the factor is refined in FP64 by the mixed path; FP64 blocks:
// k_potrf_inv64).  Measured alternatives: one column per phase (64 barriers)
// took 2x as long; a fully unrolled left-looking version (one row per
// thread, ~100 KB of straight-line code) was bound by instruction fetch;
// hand-offs between warps on mbarriers or shared flags instead of the block
// barrier were slower (their wake-up latency).
__global__ void __launch_bounds__(256) k_potrf_diag(DevCtx c, const Item* __restrict__ items, int nb) {
  using T = float;
  __shared__ __align__(16) PotrfShared<T> sh;
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, k0 = it.a;
  const int kb = min(nb, f.fs - k0);
  T* __restrict__ G = arena<T>(c) + f.off + k0 + (int64_t)k0 * n;
  T x[4][4];
  bool bad;
  // L is written over the block in place: only this CTA reads it
  potrf_block<T>(G, n, kb, sh, x, bad, G);
  if (bad && threadIdx.x == 0) set_status(c, it.front, ST_NOT_SPD);
  T* Dinv = c.dinv32;
  if (nb == 64 && Dinv) potrf_store_inverse<T>(kb, x, Dinv + f.dinv_off + (int64_t)(k0 / 64) * 4096);
}

UHM_DEFINE_WAIT_LIMIT(set_wait_limit_factor, 1u << 22)

// 1 / v by Chebyshev's iteration: an FP32 start x of the mantissa, then
// x (1 + r + r^2), r = 1 - v x (the next term, r^3, is below 2^-66); three
// dependent FP64 operations, 0.5000 ulp over 10^8 values of every exponent
__device__ __forceinline__ double fp64_rcp(double v) {
  const int hi = __double2hiint(v), f = (hi >> 20) & 0x7FF;
  if (f < 24 || f > 2022) return 1.0 / v;
  const float m = __int_as_float((127 << 23) | (hi & 0xFFFFF) << 3 | (int)((unsigned)__double2loint(v) >> 29));
  const uint32_t xb = __float_as_uint(1.0f / m);               // (1/2, 1]
  const double x = __hiloint2double((int)((hi & 0x80000000u) | ((xb >> 3) + ((1023 - 127 - (f - 1023)) << 20))),
                                    (int)(xb << 29));
  const double r = fma(-v, x, 1.0);
  return fma(x, fma(r, r, r), x);
}

// The diagonal block of FP64 fronts: only the inverse is formed (the solves and the
// TRSM use nothing else), and no multiply-add is spent on zeros.  GB300 does
// about 2 FP64 multiply-adds per clock per SM, so a warp instruction costs its
// scheduler ~64 clocks whatever its lanes do: the block is bound by their
// count and by the chain of pivots, and is spread over a cluster of two CTAs.
// Rank 0 factors A = U D U^T (U unit lower; a pivot costs its reciprocal, three
// dependent FP64 operations, and a step's vectors no product after their
// substitution); rank 1 forms Z = U^{-1} a step behind it, from the columns of U
// that rank 0 writes into its shared memory, and stores L^{-1} = D^{-1/2} Z.
//
// Both keep 4 x 4 tiles (i, j), i >= j, in registers, half a tile per thread,
// 4 x 4 tiles per warp (ten warps), so that whole warps are done early: step q (pivot
// columns P .. P+3) takes t -= U[tile i, q] W[:, tile j], W the rows' products with
// the pivots (A: j > q) or the solved rows P .. P+3 of Z (j <= q < i).  Two more
// warps solve the step's 64 vectors by a 4-step substitution, one thread each, and,
// rank 0, factor the pivot block (every thread).  Rank 0's solvers run one step
// ahead: their vectors leave the tiles before the update of the step before,
// which the solvers apply themselves, so that pivots and bulk updates overlap; they
// hand over on named barriers.
// Measured on GB300: 294 us per block in the tile-per-thread form
// (k_potrf_diag's), which updates the full squares; one CTA for both 67 with the
// steps in turn, 60 with the solvers ahead, 58 without square roots; 54 so.
constexpr int PD_WARPS = 12, PD_THREADS = 32 * PD_WARPS;
// role of each warp, by rank: tile group 0 .. 9 ((I, J), I >= J, by J), 16 / 17
// solver; a warp's scheduler is its index mod 4 (rank 0: the solvers' take the groups
// that are done first)
__device__ __constant__ signed char pd_role[2][PD_WARPS] = {{16, 17, 4, 6, 0, 2, 5, 7, 1, 3, 9, 8},
                                                            {16, 17, 1, 2, 0, 3, 4, 5, 7, 9, 6, 8}};
__device__ __constant__ signed char pd_group[10][2] = {{0, 0}, {1, 0}, {2, 0}, {3, 0}, {1, 1},
                                                       {2, 1}, {3, 1}, {2, 2}, {3, 2}, {3, 3}};

__device__ __forceinline__ void pd_arrive(int id) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(PD_THREADS) : "memory");
}
__device__ __forceinline__ void pd_sync(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(PD_THREADS) : "memory");
}
__device__ __forceinline__ uint32_t pd_peer(const void* p) {       // the same variable of rank 1
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 1;"
               : "=r"(r) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))));
  return r;
}
__device__ __forceinline__ void pd_put(uint32_t a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

struct PdShared {
  double V[2][4][64];        // vectors handed to the solvers
  double W[2][4][64];        // their results
  double B[16][4][64];       // columns of U: rank 0 the last two steps', rank 1 every step's
  double l[16][4][4];        // U's pivot blocks
  double ds[64];             // D (rank 1: then D^{-1/2})
  double pv[4][4];           // rank 0
  double Z[64][65];          // rank 1
  int sc[64];                // powers of two of a badly scaled block's rows and columns
  unsigned long long bar[16];        // rank 1: step q's column has arrived
};

__global__ void __launch_bounds__(PD_THREADS) k_potrf_inv64(DevCtx c, const Item* __restrict__ items) {
  extern __shared__ __align__(16) unsigned char pd_smem[];
  PdShared& sh = *reinterpret_cast<PdShared*>(pd_smem);
  const Item it = items[blockIdx.x >> 1];
  const int rank = blockIdx.x & 1;
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, k0 = it.a;
  const int kb = min(64, f.fs - k0);
  const int role = pd_role[rank][threadIdx.x >> 5], lane = threadIdx.x & 31;
  if (threadIdx.x < 16)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;"
                 ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(&sh.bar[threadIdx.x]))));
  if (threadIdx.x == 0) asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  // this thread's half tile: rows r0 .. r0+3, columns c0, c0+1
  int i = -1, j = -1;
  if (role >= 0 && role < 16) {
    i = 4 * pd_group[role][0] + ((lane >> 1) & 3);
    j = 4 * pd_group[role][1] + (lane >> 3);
    if (i < j) i = -1;
  }
  const int r0 = 4 * i, c0 = 4 * j + 2 * (lane & 1);
  double a[4][2];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      const int r = r0 + u, cc = c0 + v;
      a[u][v] = rank || i < 0 || r < cc ? 0.0
                : (r < kb && cc < kb)   ? c.a64[f.off + (k0 + r) + (int64_t)(k0 + cc) * n]
                                        : (r == cc ? 1.0 : 0.0);
    }
  // Diagonal entries below 2^-895: reciprocals of their pivots may overflow where the
  // entries of U are ordinary numbers.  The block is then factored with its rows and
  // columns scaled to a diagonal near 1, the inverse's columns scaled back.
  bool small = false;
  if (threadIdx.x < kb) {
    const double v = c.a64[f.off + (int64_t)(k0 + threadIdx.x) * (n + 1)];
    const int e = XsType<double>::expo(v);
    small = v > 0.0 && e < 128;
    sh.sc[threadIdx.x] = v > 0.0 ? (1023 - e) / 2 : 0;
  }
  const bool scaled = __syncthreads_or(small);
  if (scaled && rank == 0 && i >= 0) {
#pragma unroll 1
    for (int e = 0; e < 8; ++e)
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 2; ++v)
          if (e == 2 * u + v && r0 + u < kb && c0 + v < kb) a[u][v] = scalbn(a[u][v], sh.sc[r0 + u] + sh.sc[c0 + v]);
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  auto update = [&](const double (*b)[64], const double (*w)[64]) {
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      double l[4];
      Vec4<double>::ld(&b[m][r0], l);
      const double2 x = *reinterpret_cast<const double2*>(&w[m][c0]);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        a[u][0] -= l[u] * x.x;
        a[u][1] -= l[u] * x.y;
      }
    }
  };
  // barriers: 1 the solvers; 2, 3 vectors of step q (q mod 2) published; 4, 5 results of step q written
  if (rank == 0 && role < 16) {
    auto publish = [&](int q) {              // column q
      if (j == q && i >= q) {
#pragma unroll
        for (int e = 0; e < 2; ++e)
          Vec4<double>::st(&sh.V[q & 1][c0 + e - 4 * q][r0], {a[0][e], a[1][e], a[2][e], a[3][e]});
      }
    };
    publish(0);
    publish(1);
    pd_arrive(2);
#pragma unroll 1
    for (int q = 0; q < 16; ++q) {
      pd_sync(4 + (q & 1));
      if (i >= 0 && j > q + 1) update(sh.B[q & 1], sh.W[q & 1]);
      if (role < 2) {
        // (two groups that are done early) column q of U to rank 1, its pivot block, D
        const int P = 4 * q, cc = 32 * role + lane;
        if (cc >= P + 4) {
#pragma unroll
          for (int m = 0; m < 4; ++m) pd_put(pd_peer(&sh.B[q][m][cc]), sh.B[q & 1][m][cc]);
        }
        if (role == 0 && lane < 16) pd_put(pd_peer(&sh.l[q][0][0] + lane), (&sh.l[q][0][0])[lane]);
        if (role == 1 && lane < 4) pd_put(pd_peer(&sh.ds[P + lane]), sh.ds[P + lane]);
        __syncwarp();
        if (lane == 0)
          asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(pd_peer(&sh.bar[q])) : "memory");
      }
      if (q < 14) {
        publish(q + 2);
        pd_arrive(2 + (q & 1));
      }
    }
  } else if (rank == 0) {
    const int cc = 32 * (role - 16) + lane;
    bool bad = false;
    double w[4];                             // this row's results
#pragma unroll 1
    for (int q = 0; q < 16; ++q) {
      const int P = 4 * q;
      if (q != 1) pd_sync(2 + (q & 1));
      double t[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) t[m] = cc >= P ? sh.V[q & 1][m][cc] : 0.0;
      if (q > 0) {
        // the update of step q - 1
#pragma unroll
        for (int l = 0; l < 4; ++l) {
          double y[4];
          Vec4<double>::ld(&sh.B[(q - 1) & 1][l][P], y);
#pragma unroll
          for (int m = 0; m < 4; ++m) t[m] -= y[m] * w[l];
        }
      }
      if (cc >= P && cc < P + 4) Vec4<double>::st(&sh.pv[cc - P][0], t);       // A(cc, P ..)
      asm volatile("bar.sync 1, 64;" ::: "memory");
      double p[4][4], l[4][4], rd[4], d[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) Vec4<double>::ld(&sh.pv[r][0], p[r]);
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        d[m] = p[m][m];
        if (!(d[m] > 0.0)) { bad = true; d[m] = 1.0; }
        rd[m] = fp64_rcp(d[m]);
#pragma unroll
        for (int r = m + 1; r < 4; ++r) {
          l[r][m] = p[r][m] * rd[m];
#pragma unroll
          for (int e = m + 1; e <= r; ++e) p[r][e] -= l[r][m] * p[e][m];
        }
      }
      // (no row is left for the lower warp once its 32 are done)
      if (__any_sync(0xffffffffu, cc >= P + 4)) {
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          w[m] = t[m];
#pragma unroll
          for (int e = 0; e < m; ++e) w[m] -= l[m][e] * w[e];
          sh.W[q & 1][m][cc] = w[m];
          sh.B[q & 1][m][cc] = w[m] * rd[m];
        }
      }
      if (role == 17 && lane < 4) {          // lane r: row r of the pivot block
#pragma unroll
        for (int r = 0; r < 4; ++r)
          if (lane == r) {
            sh.ds[P + r] = d[r];
#pragma unroll
            for (int e = 0; e < r; ++e) sh.l[q][r][e] = l[r][e];
          }
      }
      asm volatile("bar.sync 1, 64;" ::: "memory");            // B of this step, before either warp's next
      pd_arrive(4 + (q & 1));
    }
    if (cc == 0 && bad) set_status(c, it.front, ST_NOT_SPD);
  } else if (role >= 0 && role < 16) {
#pragma unroll 1
    for (int q = 0; q < 15; ++q) {
      pd_sync(4 + (q & 1));
      if (j <= q && q < i) update(sh.B[q], sh.W[q & 1]);
      if (i == q + 1 && j <= q) {            // row q + 1 of Z
#pragma unroll
        for (int u = 0; u < 4; ++u)
          *reinterpret_cast<double2*>(&sh.V[(q + 1) & 1][u][c0]) = make_double2(a[u][0], a[u][1]);
      }
      pd_arrive(2 + ((q + 1) & 1));
    }
  } else if (role >= 16) {
    const int cc = 32 * (role - 16) + lane;
    const uint32_t lim = g_wait_limit;
    bool live = true;
#pragma unroll 1
    for (int q = 0; q < 16; ++q) {
      const int P = 4 * q;
      if (q > 0) pd_sync(2 + (q & 1));
      for (uint32_t k = 0; live; ++k) {
        uint32_t ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n"
                     " selp.b32 %0, 1, 0, p;\n}\n"
                     : "=r"(ok) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(&sh.bar[q]))) : "memory");
        if (ok) break;
        if (k >= lim) live = false;
      }
      double z[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        double w = cc < P ? sh.V[q & 1][m][cc] : (cc == P + m ? 1.0 : 0.0);
#pragma unroll
        for (int e = 0; e < m; ++e) w -= sh.l[q][m][e] * z[e];
        z[m] = w;
        sh.W[q & 1][m][cc] = w;
        sh.Z[P + m][cc] = w;
      }
      if (q < 15) pd_arrive(4 + (q & 1));
    }
    if (!live) set_status(c, it.front, ST_WAIT);
  }
  __syncthreads();
  if (rank == 1) {
    if (threadIdx.x < 64) sh.ds[threadIdx.x] = rsqrt(sh.ds[threadIdx.x]);
    __syncthreads();
    double* __restrict__ D = c.dinv64 + f.dinv_off + (int64_t)(k0 / 64) * 4096;
    for (int e = threadIdx.x; e < 4096; e += PD_THREADS) {
      const int r = e & 63, cc = e >> 6;     // entry (r, cc)
      D[e] = cc <= r && r < kb ? sh.Z[r][cc] * sh.ds[r] : 0.0;
    }
    if (scaled) {
      __syncthreads();
      for (int e = threadIdx.x; e < 64 * kb; e += PD_THREADS) D[e] = scalbn(D[e], sh.sc[e >> 6]);
    }
  }
  // neither CTA leaves while the other may still write to it
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

static void launch_potrf_inv64(const DevCtx& c, const Item* items, int n_items, cudaStream_t s) {
  cudaFuncSetAttribute(k_potrf_inv64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PdShared));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * n_items);
  cfg.blockDim = dim3(PD_THREADS);
  cfg.dynamicSmemBytes = sizeof(PdShared);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_potrf_inv64, c, items);
  if (e != cudaSuccess) throw std::runtime_error(std::string("FP64 diagonal block launch failed: ") + cudaGetErrorString(e));
}

void launch_potrf_diag(const DevCtx& c, const Item* items, int n_items, int dtype, int nb,
                       cudaStream_t s) {
  if (!n_items) return;
  if (nb > 64) throw std::invalid_argument("potrf_diag: block wider than 64");
  if (dtype == F64)
    launch_potrf_inv64(c, items, n_items, s);
  else
    k_potrf_diag<<<n_items, 256, 0, s>>>(c, items, nb);
}

constexpr int TRSM_RB = 64;   // rows per panel-TRSM block

// X (rows r0..r0+RB of columns k0..k0+kb) <- X * L11^{-T}, as a product with
// the inverse computed by the diagonal-block kernel (stored column-major 64 x
// 64): no sequential sweep.  Both tiles are loaded in one batch of registers.
__global__ void __launch_bounds__(256) k_trsm_panel(DevCtx c, const Item* __restrict__ items, XsCtx x, int slices) {
  __shared__ int s_f[4][64];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, k0 = it.a, r0 = it.b;
  const int kb = min(64, f.fs - k0);
  const int rb = min(TRSM_RB, n - r0);
  float* L = reinterpret_cast<float*>(smem_raw);        // the inverse, rows padded to 68
  float* X = L + 64 * 68;                               // TRSM_RB x 64, ld TRSM_RB
  float* __restrict__ G = c.a32 + f.off;
  const float* __restrict__ Dinv = c.dinv32 + f.dinv_off + (int64_t)(k0 / 64) * 4096;
  float xv[16], dv[16];
#pragma unroll
  for (int u = 0; u < 16; ++u) {
    const int idx = threadIdx.x + 256 * u, i = idx % TRSM_RB, j = idx / TRSM_RB;
    xv[u] = (i < rb && j < kb) ? G[(r0 + i) + (int64_t)(k0 + j) * n] : 0.f;
    dv[u] = Dinv[idx];
  }
#pragma unroll
  for (int u = 0; u < 16; ++u) {
    const int idx = threadIdx.x + 256 * u;
    // Dinv is column-major: Dinv[t * 64 + j] = Linv[j][t]; keep it as
    // rows t of length 64 padded to 68 (16-byte rows), L[t * 68 + j] = Linv[j][t]
    const int t = idx / 64, j = idx % 64;
    X[idx] = xv[u];
    L[t * 68 + j] = (t < kb && j < kb) ? dv[u] : 0.f;
  }
  __syncthreads();
  const int i = threadIdx.x % TRSM_RB, jg = threadIdx.x / TRSM_RB;   // 4 column groups of 16
  float acc[16];
#pragma unroll
  for (int u = 0; u < 16; ++u) acc[u] = 0.f;
  // Linv is lower triangular: columns jg * 16 .. need t <= jg * 16 + 15
  const int te = min(kb, 16 * jg + 16);
  for (int t = 0; t < te; ++t) {
    const float xt = X[i + t * TRSM_RB];
#pragma unroll
    for (int u4 = 0; u4 < 16; u4 += 4) {
      float l4[4];
      Vec4<float>::ld(&L[t * 68 + jg * 16 + u4], l4);
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[u4 + e] += xt * l4[e];
    }
  }
#pragma unroll
  for (int u = 0; u < 16; ++u) {
    const int j = jg * 16 + u;
    if (i < rb && j < kb) G[(r0 + i) + (int64_t)(k0 + j) * n] = acc[u];
  }
  if (slices && k0 + kb < min(k0 / XS_NBO * XS_NBO + XS_NBO, f.fs))
    xs_store_step<float>(x, it.front, n, r0 + i, i < rb, acc, s_f);
}

void launch_trsm_panel(const DevCtx& c, const Item* items, int n_items, int dtype, int nb, const XsCtx& x, int slices,
                       cudaStream_t s) {
  if (!n_items) return;
  if (dtype == F64) throw std::invalid_argument("trsm_panel: FP64 fronts take xs_trsm");
  if (nb != 64) throw std::invalid_argument("trsm_panel: panels are 64 columns wide");
  const size_t sm = (size_t)(64 * 68 + TRSM_RB * 64) * sizeof(float);
  cudaFuncSetAttribute(k_trsm_panel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  k_trsm_panel<<<n_items, 256, sm, s>>>(c, items, x, slices);
}

// Diagonal block and panel TRSM of one 64-column step in one launch.  Every
// CTA factors the diagonal block and forms its inverse itself (potrf_block;
// the SMs would otherwise idle through that latency-bound step), then
// applies X <- X L^{-T} = X (L^{-1})^T to its 64-row block of the panel.  The
// CTA flagged in the item writes the inverse, which is how the factor's
// diagonal block is kept: the flag-driven solves and this TRSM use only the
// inverse, and writing L over the block in place would race with other
// CTAs still reading A's block, so the arena keeps A's diagonal block.  A CTA
// takes several consecutive row blocks, so that a step's launch is one wave.
// Item: front, a = k0, b = first row of the first block (n: none),
// c = writer (bit 0) + 2 * number of row blocks.  slices: the rows' slices for
// the update inside the outer panel too (a launch of their own took 11 us and
// more a step).
constexpr int PT_LD = 68;   // row length of the transposed inverse in shared memory (16-byte rows)

__global__ void __launch_bounds__(256) k_potrf_trsm(DevCtx c, const Item* __restrict__ items, XsCtx xs, int slices) {
  using T = float;
  __shared__ int s_f[4][64];
  extern __shared__ __align__(16) unsigned char pt_smem[];
  PotrfShared<T>& sh = *reinterpret_cast<PotrfShared<T>*>(pt_smem);
  T* Lt = reinterpret_cast<T*>(pt_smem + ((sizeof(PotrfShared<T>) + 15) / 16) * 16);   // 64 x PT_LD
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, k0 = it.a;
  const int kb = min(64, f.fs - k0);
  T* __restrict__ A = arena<T>(c) + f.off;
  T* __restrict__ G = A + k0 + (int64_t)k0 * n;
  const int tid = threadIdx.x;
  T x[4][4];
  bool bad;
  potrf_block<T>(G, n, kb, sh, x, bad, nullptr);
  const bool writer = it.c & 1;
  const int nrb = it.c >> 1;
  if (writer) {
    if (bad && tid == 0) set_status(c, it.front, ST_NOT_SPD);
    potrf_store_inverse<T>(kb, x, c.dinv32 + f.dinv_off + (int64_t)(k0 / 64) * 4096);
  }
  if (it.b >= n || nrb == 0) return;
  // L^{-1} transposed into Lt (Lt[t * PT_LD + j] = Linv[j][t]); the panel
  // blocks into V in turn (its factor values are no longer needed)
  {
    const int ti = tid & 15, tj = tid >> 4;
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int j = 4 * ti + u, t = 4 * tj + v;   // x[u][v] = Linv[j][t]
        Lt[t * PT_LD + j] = (j < kb && t < kb) ? x[u][v] : T(0);
      }
  }
  T* X = &sh.V[0][0];   // 64 x 64, column-major
  const int i = tid % TRSM_RB, jg = tid / TRSM_RB;   // 4 column groups of 16
  for (int blk = 0; blk < nrb; ++blk) {
    const int r0 = it.b + blk * TRSM_RB;
    if (r0 >= n) break;
    const int rb = min(TRSM_RB, n - r0);
    {
      T xv[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int idx = tid + 256 * u, ii = idx % TRSM_RB, j = idx / TRSM_RB;
        xv[u] = (ii < rb && j < kb) ? A[(r0 + ii) + (int64_t)(k0 + j) * n] : (T)0;
      }
      __syncthreads();   // the previous block's reads of X are done
#pragma unroll
      for (int u = 0; u < 16; ++u) X[tid + 256 * u] = xv[u];
    }
    __syncthreads();
    T acc[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) acc[u] = T(0);
    for (int t = 0; t < kb; ++t) {
      const T xt = X[i + t * TRSM_RB];
#pragma unroll
      for (int u4 = 0; u4 < 16; u4 += 4) {
        T l4[4];
        Vec4<T>::ld(&Lt[t * PT_LD + jg * 16 + u4], l4);
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[u4 + e] += xt * l4[e];
      }
    }
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int j = jg * 16 + u;
      if (i < rb && j < kb) A[(r0 + i) + (int64_t)(k0 + j) * n] = acc[u];
    }
    if (slices && k0 + kb < min(k0 / XS_NBO * XS_NBO + XS_NBO, f.fs))
      xs_store_step<T>(xs, it.front, n, r0 + i, i < rb, acc, s_f);
  }
}

void launch_potrf_trsm(const DevCtx& c, const Item* items, int n_items, int dtype, const XsCtx& x, int slices,
                       cudaStream_t s) {
  if (!n_items) return;
  if (dtype == F64) throw std::invalid_argument("potrf_trsm: FP64 fronts take potrf_diag and xs_trsm");
  const size_t sm = ((sizeof(PotrfShared<float>) + 15) / 16) * 16 + sizeof(float) * 64 * PT_LD;
  cudaFuncSetAttribute(k_potrf_trsm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  k_potrf_trsm<<<n_items, 256, sm, s>>>(c, items, x, slices);
}

// FP32 update of one 128 x 64 tile of the front by a panel of kb <= 64 columns:
//   C[rows, cols] -= A[rows, k0:k0+kb] * B,  B = A[cols, k0:k0+kb]^T  (ROWPANEL=false: SYRK)
//                                            B = A[k0:k0+kb, cols]    (ROWPANEL=true: LU GEMM)
// item: front, a = k0, b = tile row, c = tile col (tiles counted from k0+kb).
// With two-level blocking (nbo > 0) B = K0 + min(nbo, fs - K0) is the first
// row / column of the current outer panel's trailing block, and region
// selects what is updated: 0 every entry, 1 columns < B (inside the outer
// panel), 2 rows < B and columns >= B (the outer panel's rows right of it).
//
// Both operands go to shared memory whole, by 4-byte asynchronous copies (a
// column of a front starts at any multiple of 4 bytes) with C's entries loaded
// behind them; a warp takes 128 rows x 8 columns, a lane four rows 32 apart, so
// that C is read and written 32 rows at a time and a step of k is four
// shared-memory words and two broadcast 16-byte ones per 32 multiply-adds.
// Bound by those multiply-adds and, K being 64 at most, by the tile's loads.
// Measured on GB300, the updates inside the panels of 24^3 p = 3 LU (14,911 rows
// down): 14.3 (64 x 64 tiles, four by four entries a thread) -> 10.6 ms.
constexpr int TU_BM = TILE_UPDATE_ROWS, TU_BN = TILE_UPDATE_COLS, TU_K = 64;
constexpr int TU_LDA = TU_BM + 1, TU_LDB = TU_BN + 4;
constexpr size_t TU_SMEM = sizeof(float) * TU_K * (TU_LDA + TU_LDB);

// 4 bytes to shared memory, zero where !ok
__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool ok) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(ok ? 4 : 0) : "memory");
}

template <bool ROWPANEL>
__global__ void __launch_bounds__(256, 2)
k_tile_update(DevCtx c, const Item* __restrict__ items, int nb, int nbo, int region) {
  extern __shared__ __align__(16) float tu_smem[];
  float* Bs = tu_smem;                       // Bs[t][column], 16-byte rows
  float* As = tu_smem + TU_K * TU_LDB;       // As[t][row]
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, k0 = it.a;
  const int kb = min(nb, f.fs - k0);
  const int base = k0 + kb;
  const int R0 = base + it.b * TU_BM, C0 = base + it.c * TU_BN;
  const int Bnd = nbo > 0 ? min((k0 / nbo) * nbo + nbo, f.fs) : n;
  const int rmax = region == 2 ? Bnd : n;
  const int cmin = region == 2 ? Bnd : 0;
  const int cmax = region == 1 ? Bnd : n;
  float* __restrict__ G = c.a32 + f.off;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll 8
  for (int e = 0; e < TU_BM * TU_K / 256; ++e) {
    const int idx = tid + 256 * e, r = idx % TU_BM, t = idx / TU_BM;
    const bool ok = R0 + r < n && t < kb;
    cp_async4(As + t * TU_LDA + r, ok ? G + R0 + r + (int64_t)(k0 + t) * n : G, ok);
  }
#pragma unroll 8
  for (int e = 0; e < TU_BN * TU_K / 256; ++e) {
    const int idx = tid + 256 * e;
    const int r = ROWPANEL ? idx / TU_K : idx % TU_BN, t = ROWPANEL ? idx % TU_K : idx / TU_BN;
    const bool ok = C0 + r < n && t < kb;
    const int64_t at = ROWPANEL ? (k0 + t) + (int64_t)(C0 + r) * n : (C0 + r) + (int64_t)(k0 + t) * n;
    cp_async4(Bs + t * TU_LDB + r, ok ? G + at : G, ok);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  float cv[4][8], acc[4][8];
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int gr = R0 + lane + 32 * i, gc = C0 + 8 * warp + j;
      const bool ok = gr < rmax && gc >= cmin && gc < cmax && (ROWPANEL || gr >= gc);
      cv[i][j] = ok ? G[gr + (int64_t)gc * n] : 0.f;
      acc[i][j] = 0.f;
    }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
#pragma unroll 4
  for (int t = 0; t < TU_K; ++t) {
    float a[4], b[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = As[t * TU_LDA + lane + 32 * i];
    const float4 b0 = *reinterpret_cast<const float4*>(Bs + t * TU_LDB + 8 * warp);
    const float4 b1 = *reinterpret_cast<const float4*>(Bs + t * TU_LDB + 8 * warp + 4);
    b[0] = b0.x; b[1] = b0.y; b[2] = b0.z; b[3] = b0.w;
    b[4] = b1.x; b[5] = b1.y; b[6] = b1.z; b[7] = b1.w;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] += a[i] * b[j];
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int gr = R0 + lane + 32 * i, gc = C0 + 8 * warp + j;
      const bool ok = gr < rmax && gc >= cmin && gc < cmax && (ROWPANEL || gr >= gc);
      if (ok) G[gr + (int64_t)gc * n] = cv[i][j] - acc[i][j];
    }
}

template <bool ROWPANEL>
static void tile_update(const DevCtx& c, const Item* items, int n_items, int dtype, int nb, int nbo, int region,
                        cudaStream_t s) {
  if (!n_items) return;
  if (nb > 64) throw std::invalid_argument("trailing update: panel width above 64");
  if (dtype == F64) throw std::invalid_argument("trailing update: FP64 fronts take the sliced update");
  cudaFuncSetAttribute(k_tile_update<ROWPANEL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TU_SMEM);
  k_tile_update<ROWPANEL><<<n_items, 256, TU_SMEM, s>>>(c, items, nb, nbo, region);
}

void launch_syrk_update(const DevCtx& c, const Item* items, int n_items, int dtype, int nb, int nbo, cudaStream_t s) {
  tile_update<false>(c, items, n_items, dtype, nb, nbo, nbo > 0 ? 1 : 0, s);
}

void launch_gemm_update(const DevCtx& c, const Item* items, int n_items, int dtype, int nb, int nbo, int region,
                        cudaStream_t s) {
  tile_update<true>(c, items, n_items, dtype, nb, nbo, region, s);
}

// ---------------------------------------------------------------------------
// blocked large-front LU: panel (with pivot search restricted to rows < fs),
// row-panel solve U12 = L11^{-1} A12, trailing GEMM (k_tile_update<..., true>)
// ---------------------------------------------------------------------------
template <typename T, int NT>
__global__ void __launch_bounds__(NT) k_getrf_panel(DevCtx c, const Item* __restrict__ items,
                                                    int nb, int pivot) {
  __shared__ T s_v[NT / 32];
  __shared__ int s_i[NT / 32];
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, fs = f.fs, k0 = it.a;
  const int kb = min(nb, fs - k0);
  const int jend = it.b > 0 ? min(it.b, n) : n;   // rows are swapped in columns it.c .. jend - 1
  T* __restrict__ G = arena<T>(c) + f.off;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int NW = NT / 32;
  for (int k = k0; k < k0 + kb; ++k) {
    if (pivot) {
      T best = (T)-1;
      int bi = k;
      for (int i = k + threadIdx.x; i < fs; i += NT) {
        const T v = my_abs<T>(G[i + (int64_t)k * n]);
        if (v > best) { best = v; bi = i; }
      }
      const int p = block_argmax<T, NT>(best, bi, s_v, s_i);
      if (threadIdx.x == 0) c.piv[f.piv_off + k] = p;
      if (p != k)
        for (int j = it.c + threadIdx.x; j < jend; j += NT) {
          T t = G[k + (int64_t)j * n];
          G[k + (int64_t)j * n] = G[p + (int64_t)j * n];
          G[p + (int64_t)j * n] = t;
        }
      __syncthreads();
    }
    T akk = G[k + (int64_t)k * n];
    if (akk == (T)0 || akk != akk) {
      if (threadIdx.x == 0) set_status(c, it.front, akk != akk ? ST_NAN : ST_ZERO_PIVOT);
      akk = (T)1;
    }
    __syncthreads();
    for (int i = k + 1 + threadIdx.x; i < n; i += NT) G[i + (int64_t)k * n] /= akk;
    __syncthreads();
    for (int j = k + 1 + warp; j < k0 + kb; j += NW) {
      const T akj = G[k + (int64_t)j * n];
      for (int i = k + 1 + lane; i < n; i += 32) G[i + (int64_t)j * n] -= G[i + (int64_t)k * n] * akj;
    }
    __syncthreads();
  }
}

void launch_getrf_panel(const DevCtx& c, const Item* items, int n_items, int dtype, int nb,
                        int pivot, cudaStream_t s) {
  if (!n_items) return;
  if (dtype == F64) k_getrf_panel<double, 512><<<n_items, 512, 0, s>>>(c, items, nb, pivot);
  else k_getrf_panel<float, 512><<<n_items, 512, 0, s>>>(c, items, nb, pivot);
}

// ---------------------------------------------------------------------------
// LU panel in shared memory: one CTA, a cluster, or a whole grid per front
// ---------------------------------------------------------------------------
// The panel (rows k0..n-1, columns k0..k0+kb-1) of each item is split into
// chunks of R rows, one per CTA, held in shared memory (row-major: a thread
// updates four columns of its row with 16-byte accesses).  For each column k of the panel, every CTA
//   1. offers its candidate pivot: the largest |a| in column k among its rows
//      in [k0+k, fs) (the reference searches the eliminated rows only), ties
//      to the lowest row, with the row's kb values; the CTA holding row k0+k
//      also hands out that row;
//   2. picks the pivot from all its item's candidates (same rule: the largest
//      value, the lowest row on ties; this is the first maximum of a sequential
//      search; compared as integers, the bits of |a|);
//   3. swaps the two rows in its chunk when it holds them, and applies l_r =
//      a_rk / a_kk, a_rj -= l_r u_j to its rows below the pivot row, column
//      k + 1 first, whose candidates are found on the way.
// The result is the reference's partial pivoting (FLA_LU_piv inside the
// eliminated block) exactly; only the panel's own columns are swapped here,
// the other columns of the front by k_laswp afterwards.
//
// Two ways to hand candidates and rows over:
// CL: the item's CTAs are a cluster (1 .. 16 of them) and write into each
// other's shared memory; one cluster barrier per column orders it (buffers
// alternate by column: nobody writes column k + 2 before everybody has
// passed the barrier of k + 1, that is, has used column k).  Item: front, a = k0.
// !CL (rows beyond a cluster's shared memory, or FP64 fronts whose update
// wants more SMs): 8-byte words in global memory whose upper bits hold the
// column (k + 1) beside the data, polled until they carry it; no counter, flag
// or fence.  The same argument holds for their reuse, since a CTA publishes its
// candidate of k + 1 only when it has read all of column k (also without
// pivoting, where no candidate wins).  The words are cleared before the
// launch; the launch is cooperative, every wait is bounded, and a CTA that
// gives up raises the error word, which ends the others' waits.  Item: front, a
// = k0, b = first CTA, c = number of CTAs.
//
// Bound by the latency of a column: about 3 us in either form (two or three
// block barriers, one exchange, the reductions), then by the update's shared-
// memory traffic (FP32) or multiply-adds (FP64).  Measured on GB300, the panels
// of one factorisation, against a grid barrier on a counter per column: 24^3 p =
// 3 FP32 141 + 2.5 (one-CTA panels in global memory) -> 57.1 ms, 12^3 p = 3
// FP64 55.9 + 4.8 -> 23.3, 6^3 p = 3 4.9 + 2.0 -> 4.3.  The chunk by columns instead
// (one column of a row per access) took 69.0, 25.7 and 4.4: bank conflicts where a
// row is read, and four times the shared-memory instructions.  !CL with each
// candidate in front of its row and its two words polled one after the other: 59.4
// and 24.2 (a panel of 152 CTAs 187 us FP32, 207 FP64, now 166 and 200).
constexpr int GC_ERR = 3;
constexpr int GC_POLL = (GC_MAX_CTAS + 31) / 32;
constexpr int64_t GC_REC = 2 * 64;              // words of a row's record (two per FP64 value)
static_assert(gc_words(1, 1) == 4 + 4 * GC_REC, "record size of the launcher's callers");


template <typename T> struct LuBits;
template <> struct LuBits<double> {
  static constexpr int WORDS = 2;               // exchange words per value
  static constexpr int LD = 66;                 // row of the chunk (16-byte loads of 8 rows hit every bank once)
  static __device__ __forceinline__ uint64_t key(double v) {
    return v == v ? (uint64_t)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull : 0ull;
  }
  static __device__ __forceinline__ uint32_t half(double v, int h) {
    return h ? (uint32_t)__double2loint(v) : (uint32_t)__double2hiint(v);
  }
  static __device__ __forceinline__ double make(uint32_t hi, uint32_t lo) { return __hiloint2double((int)hi, (int)lo); }
};
template <> struct LuBits<float> {
  static constexpr int WORDS = 1;
  static constexpr int LD = 68;
  static __device__ __forceinline__ uint64_t key(float v) {
    return v == v ? (uint64_t)(__float_as_uint(v) & 0x7FFFFFFFu) : 0ull;
  }
  static __device__ __forceinline__ uint32_t half(float v, int) { return __float_as_uint(v); }
  static __device__ __forceinline__ float make(uint32_t hi, uint32_t) { return __uint_as_float(hi); }
};
constexpr int LU_NONE = 0x7fffffff;             // no candidate row

// the warp's best candidate: the largest key, the lowest row on ties (LU_NONE
// where no lane has one)
template <typename T>
__device__ __forceinline__ void lu_best(uint64_t& key, int& r) {
  const uint32_t all = 0xffffffffu;
  if constexpr (sizeof(T) == 4) {
    const uint32_t k = r == LU_NONE ? 0u : (uint32_t)key + 1, mx = __reduce_max_sync(all, k);
    r = (int)__reduce_min_sync(all, k == mx ? (uint32_t)r : (uint32_t)LU_NONE);
    key = mx ? mx - 1 : 0;
  } else {
    const uint32_t h = r == LU_NONE ? 0u : (uint32_t)(key >> 32) + 1, mh = __reduce_max_sync(all, h);
    const uint32_t l = h == mh && mh ? (uint32_t)key : 0u, ml = __reduce_max_sync(all, l);
    r = (int)__reduce_min_sync(all, h == mh && l == ml ? (uint32_t)r : (uint32_t)LU_NONE);
    key = mh ? (uint64_t)(mh - 1) << 32 | ml : 0;
  }
}

__device__ __forceinline__ void gc_put(uint64_t* p, uint64_t v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ uint64_t gc_get(const uint64_t* p) {
  uint64_t v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
// words p[32 e + lane] (e < N, while < cnt), all loads in flight, until every
// one carries the tag; false (and the error word set) when the wait gives up
template <int N>
__device__ __forceinline__ bool gc_poll(const uint64_t* p, int cnt, uint32_t tag, uint64_t (&x)[N], int* err) {
  const int lane = threadIdx.x & 31;
  const uint32_t lim = g_wait_limit;
  uint32_t open = 0;
#pragma unroll
  for (int e = 0; e < N; ++e) open |= (lane + 32 * e < cnt ? 1u : 0u) << e;
  for (uint32_t i = 0; open; ++i) {
    uint64_t y[N];
#pragma unroll
    for (int e = 0; e < N; ++e)
      if ((open >> e) & 1) y[e] = gc_get(p + lane + 32 * e);
#pragma unroll
    for (int e = 0; e < N; ++e)
      if (((open >> e) & 1) && (uint32_t)(y[e] >> 56) == tag) { x[e] = y[e]; open &= ~(1u << e); }
    if (!open) break;
    if (i >= lim) { atomicExch(err, GC_ERR); return false; }
    if ((i & 255) == 255 && *(volatile int*)err) return false;
    if (i > 64) __nanosleep(20);
  }
  return true;
}
// the same for pairs of words: p[2 (32 e + lane)] and the word behind it
template <int N>
__device__ __forceinline__ bool gc_poll2(const uint64_t* p, int cnt, uint32_t tag, uint64_t (&x0)[N], uint64_t (&x1)[N],
                                         int* err) {
  const int lane = threadIdx.x & 31;
  const uint32_t lim = g_wait_limit;
  uint32_t open = 0;
#pragma unroll
  for (int e = 0; e < N; ++e) open |= (lane + 32 * e < cnt ? 1u : 0u) << e;
  for (uint32_t i = 0; open; ++i) {
    uint64_t y0[N], y1[N];
#pragma unroll
    for (int e = 0; e < N; ++e)
      if ((open >> e) & 1)
        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                     : "=l"(y0[e]), "=l"(y1[e]) : "l"(p + 2 * (lane + 32 * e)) : "memory");
#pragma unroll
    for (int e = 0; e < N; ++e)
      if (((open >> e) & 1) && (uint32_t)(y0[e] >> 56) == tag && (uint32_t)(y1[e] >> 56) == tag) {
        x0[e] = y0[e];
        x1[e] = y1[e];
        open &= ~(1u << e);
      }
    if (!open) break;
    if (i >= lim) { atomicExch(err, GC_ERR); return false; }
    if ((i & 255) == 255 && *(volatile int*)err) return false;
    if (i > 64) __nanosleep(20);
  }
  return true;
}
__device__ __forceinline__ uint32_t lu_smem(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint32_t lu_mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void lu_put(uint32_t a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void lu_put(uint32_t a, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void lu_put(uint32_t a, uint64_t v) {
  asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}
__device__ __forceinline__ void lu_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float lu_rcp(float v) { return 1.0f / v; }
__device__ __forceinline__ double lu_rcp(double v) { return fp64_rcp(v); }

// rows received in one column: of every candidate (CL) or of the pivot, then row k0 + k
template <typename T, bool CL>
struct LuRecv {
  T row[CL ? GC_CLUSTER : 1][64];
  T diag[64];
  uint64_t cand[CL ? GC_CLUSTER : 1][2];        // key, row
};

// A subnormal pivot's reciprocal may overflow where the quotients by it are ordinary
// numbers: it and its column are scaled up first.  (Every thread of the CTA; out of
// line, so that the column loop's registers stay as they are.)
template <typename T, int NT>
__device__ __noinline__ T lu_scale_up(T* col, int rows, T* diag, T akk) {
  constexpr T UP = T(sizeof(T) == 8 ? 0x1p128 : 0x1p64);
  __syncthreads();                             // every thread has read the pivot
  for (int r = threadIdx.x; r < rows; r += NT) col[r] *= UP;
  if (threadIdx.x == 0) *diag *= UP;
  __syncthreads();
  return akk * UP;
}

template <typename T, bool CL, int NT>
__global__ void __launch_bounds__(NT) k_getrf_smem(DevCtx c, const Item* __restrict__ items, int n_items, int nb,
                                                   int pivot, int rmax, int csize, uint64_t* __restrict__ xbuf,
                                                   int* err) {
  extern __shared__ __align__(16) unsigned char gc_smem[];
  using LuRecvT = LuRecv<T, CL>;
  constexpr int NW = NT / 32, WORDS = LuBits<T>::WORDS, SR = LuBits<T>::LD;
  __shared__ __align__(16) LuRecv<T, CL> recv[2];
  __shared__ uint64_t s_key[NW];
  __shared__ int s_row[NW];
  __shared__ int s_item, s_p;
  __shared__ T s_rinv;
  T* S = reinterpret_cast<T*>(gc_smem);        // chunk, row-major, rows of SR
  T* s_col = S + (int64_t)rmax * SR;           // the column to eliminate next, by parity
  const int total = gridDim.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    int k = 0;
    if (!CL) while (k + 1 < n_items && (int)blockIdx.x >= items[k + 1].b) ++k;
    s_item = CL ? blockIdx.x / csize : k;
  }
  for (int e = tid; e < (int)(sizeof(recv) / sizeof(uint32_t)); e += NT) reinterpret_cast<uint32_t*>(recv)[e] = 0;
  __syncthreads();
  const Item it = items[s_item];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, fs = f.fs, k0 = it.a;
  const int kb = min(nb, fs - k0);
  const int P = CL ? csize : it.c, q = CL ? (int)blockIdx.x % csize : (int)blockIdx.x - it.b;
  const int rows = n - k0;
  const int R = (rows + P - 1) / P;
  const int rbeg = k0 + q * R, rend = min(rbeg + R, n);   // my rows [rbeg, rend)
  const int nr_my = max(0, rend - rbeg);
  T* __restrict__ G = arena<T>(c) + f.off;
  // !CL: per parity, the candidates of all CTAs side by side (two words each); then
  // rows, per parity one per CTA and one per item (the row k0 + k)
  auto cand = [&](int par, int b) { return xbuf + 2 * ((int64_t)par * total + b); };
  auto rec = [&](int par, int b) { return xbuf + 4 * total + ((int64_t)par * (total + n_items) + b) * GC_REC; };
  // thread layout of the chunk: rows along lanes, ng groups of 4-column blocks
  const int rw = min(NT, (max(nr_my, 1) + 31) / 32 * 32), ng = NT / rw;
  const int tr = tid % rw, tg = tid / rw;
  uint64_t mk = 0;                             // this thread's best candidate of the next column
  int mr = LU_NONE;
  auto offer = [&](T v, int r) {
    const uint64_t key = LuBits<T>::key(v);
    if (v == v && (mr == LU_NONE || key > mk || (key == mk && r < mr))) { mk = key; mr = r; }
  };
  if (tg < ng)
    for (int j = tg; j < 64; j += ng)
      for (int r = tr; r < nr_my; r += rw) {
        const T v = j < kb ? G[(rbeg + r) + (int64_t)(k0 + j) * n] : T(0);
        S[r * SR + j] = v;
        if (j == 0) {
          s_col[r] = v;
          if (pivot && rbeg + r < fs) offer(v, rbeg + r);
        }
      }
  lu_best<T>(mk, mr);
  if (lane == 0) { s_key[warp] = mk; s_row[warp] = mr; }
  if (CL && csize > 1) lu_cluster_sync();      // every CTA of the cluster runs before anyone writes to it
  __syncthreads();
  for (int k = 0; k < kb; ++k) {
    const int gk = k0 + k, par = k & 1;
    const bool diag_mine = gk >= rbeg && gk < rend;
    LuRecv<T, CL>& rc = recv[par];
    // 1. this chunk's candidate, known to every warp
    uint64_t bk = lane < NW ? s_key[lane] : 0;
    int bi = lane < NW ? s_row[lane] : LU_NONE;
    lu_best<T>(bk, bi);
    const T* u;                                // the pivot's row and the old row k0 + k
    const T* old = rc.diag;
    int p = gk;
    if constexpr (CL) {
      // warp w serves CTA w
      if (warp < csize) {
        const T* cs = S + (bi == LU_NONE ? 0 : bi - rbeg) * SR + lane;
        const T* ds = S + (diag_mine ? gk - rbeg : 0) * SR + lane;
        const T c0 = cs[0], c1 = cs[32], d0 = ds[0], d1 = ds[32];
        const uint32_t a = lu_mapa(lu_smem(&rc), warp);
        const uint32_t ar = a + (uint32_t)offsetof(LuRecvT, row) + (uint32_t)sizeof(T) * (64 * q + lane);
        const uint32_t ad = a + (uint32_t)offsetof(LuRecvT, diag) + (uint32_t)sizeof(T) * lane;
        lu_put(ar, c0);
        lu_put(ar + 32 * (uint32_t)sizeof(T), c1);
        if (diag_mine) {
          lu_put(ad, d0);
          lu_put(ad + 32 * (uint32_t)sizeof(T), d1);
        }
        if (lane < 2)
          lu_put(a + (uint32_t)offsetof(LuRecvT, cand) + 16u * q + 8u * lane, lane ? (uint64_t)bi : bk);
      }
      if (csize > 1) lu_cluster_sync();
      else __syncthreads();
      // 2. the item's pivot
      uint64_t key = lane < csize ? rc.cand[lane][0] : 0;
      int r = lane < csize ? (int)rc.cand[lane][1] : LU_NONE, w = lane;
      lu_best<T>(key, r);
      if (r != LU_NONE) p = r;
      w = __ffs(__ballot_sync(0xffffffffu, lane < csize && (int)rc.cand[w & (GC_CLUSTER - 1)][1] == r)) - 1;
      u = p == gk ? rc.diag : rc.row[max(w, 0)];
    } else {
      const uint64_t tag56 = (uint64_t)(k + 1) << 56;
      bool ok = true;
      if (warp == 0) {
        uint64_t* cb = rec(par, blockIdx.x);
        if (lane < 2)
          // key bits 63..32 and the row (24 bits) in the first word, key bits 31..0 in the second
          gc_put(cand(par, blockIdx.x) + lane, tag56 | (lane == 0 ? (uint64_t)(bi == LU_NONE ? 0xFFFFFFu : (uint32_t)(bi - k0)) << 32 | (bk >> 32)
                                               : (bk & 0xFFFFFFFFull)));
        if (bi != LU_NONE)
          for (int w = lane; w < kb * WORDS; w += 32)
            gc_put(cb + w, tag56 | LuBits<T>::half(S[(bi - rbeg) * SR + w / WORDS], w % WORDS));
        // 2. the item's pivot
        uint64_t x0[GC_POLL], x1[GC_POLL], key = 0;
        int r = LU_NONE;
        ok = gc_poll2<GC_POLL>(cand(par, it.b), P, k + 1, x0, x1, err);
        if (ok) {
#pragma unroll
          for (int e = 0; e < GC_POLL; ++e) {
            if (lane + 32 * e >= P) continue;
            const uint64_t ck = x0[e] << 32 | (x1[e] & 0xFFFFFFFFull);
            const uint32_t row = (uint32_t)(x0[e] >> 32) & 0xFFFFFFu;
            const int cr = k0 + (int)row;
            if (row != 0xFFFFFFu && (r == LU_NONE || ck > key || (ck == key && cr < r))) { key = ck; r = cr; }
          }
        }
        ok = __all_sync(0xffffffffu, ok);
        lu_best<T>(key, r);
        if (r != LU_NONE) p = r;
        if (lane == 0) s_p = p;
        if (ok && p != gk) {
          if (p >= rbeg && p < rend) {
            for (int j = lane; j < kb; j += 32) rc.row[0][j] = S[(p - rbeg) * SR + j];
          } else {
            uint64_t x[2 * WORDS];
            ok = gc_poll<2 * WORDS>(rec(par, it.b + (p - k0) / R), kb * WORDS, k + 1, x, err);
#pragma unroll
            for (int e = 0; e < 2 * WORDS; ++e) {
              const uint32_t v = (uint32_t)x[e], lo = __shfl_down_sync(0xffffffffu, v, 1);
              const int t = lane + 32 * e;
              if (ok && t < kb * WORDS && t % WORDS == 0) rc.row[0][t / WORDS] = LuBits<T>::make(v, lo);
            }
          }
        }
      } else if (warp == 1) {
        // the old row k0 + k
        uint64_t* dr = rec(par, total + s_item);
        if (diag_mine) {
          for (int w = lane; w < kb * WORDS; w += 32)
            gc_put(dr + w, tag56 | LuBits<T>::half(S[(gk - rbeg) * SR + w / WORDS], w % WORDS));
          for (int j = lane; j < kb; j += 32) rc.diag[j] = S[(gk - rbeg) * SR + j];
        } else {
          uint64_t x[2 * WORDS];
          ok = gc_poll<2 * WORDS>(dr, kb * WORDS, k + 1, x, err);
#pragma unroll
          for (int e = 0; e < 2 * WORDS; ++e) {
            const uint32_t v = (uint32_t)x[e], lo = __shfl_down_sync(0xffffffffu, v, 1);
            const int t = lane + 32 * e;
            if (ok && t < kb * WORDS && t % WORDS == 0) rc.diag[t / WORDS] = LuBits<T>::make(v, lo);
          }
        }
      }
      if (__syncthreads_or(!ok)) return;
      p = s_p;
      u = p == gk ? rc.diag : rc.row[0];
    }
    if (q == 0 && tid == 0) c.piv[f.piv_off + gk] = p;
    T akk = u[k];
    if (akk == (T)0 || akk != akk) {
      if (q == 0 && tid == 0) set_status(c, it.front, akk != akk ? ST_NAN : ST_ZERO_PIVOT);
      akk = (T)1;
    }
    if (XsType<T>::field(akk) == 0) akk = lu_scale_up<T, NT>(s_col + par * rmax, nr_my, &rc.diag[k], akk);
    T rinv;
    if constexpr (sizeof(T) == 8) {            // a reciprocal costs every FP64 warp that takes it
      if (warp == 0) {
        rinv = lu_rcp(akk);
        if (lane == 0) s_rinv = rinv;
      }
      __syncthreads();
      rinv = s_rinv;
    } else {
      rinv = lu_rcp(akk);
    }
    // 3. rows from the pivot row on: the two rows swapped, multiplier and
    // rank-1 update of the panel's later columns below it; the 4-column
    // blocks from that of column k + 1 on in turn over the groups
    mk = 0;
    mr = LU_NONE;
    const int b0 = (k + 1) >> 2;
    if (tg < ng)
      for (int rl = max(rbeg, gk) - rbeg + tr; rl < nr_my; rl += rw) {
        const int r = rbeg + rl;
        T* __restrict__ row = S + rl * SR;
        if (r == gk) {
          if (p != gk)
            for (int j = tg; j < 64; j += ng) row[j] = u[j];
          continue;
        }
        T a[4], x[4];
        const bool sw = r == p;
        const T* __restrict__ src = sw ? old : row;
        const T l = (sw ? old[k] : s_col[par * rmax + rl]) * rinv;
        if (sw)
          for (int b = tg; b < b0; b += ng) {
            Vec4<T>::ld(old + 4 * b, a);
            if (4 * b + 3 == k) a[3] = l;
            Vec4<T>::st(row + 4 * b, a);
          }
        int b = b0 + tg;
        if (tg == 0) {
          if ((k & 3) == 3 && !sw) row[k] = l; // column k in the block before
          if (b < 16) {
            Vec4<T>::ld(src + 4 * b, a);
            Vec4<T>::ld(u + 4 * b, x);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int j = 4 * b + e;
              if (j > k) a[e] -= l * x[e];
              else if (j == k) a[e] = l;
            }
            Vec4<T>::st(row + 4 * b, a);
            const int e1 = (k + 1) & 3;
            const T v = e1 == 0 ? a[0] : e1 == 1 ? a[1] : e1 == 2 ? a[2] : a[3];
            s_col[(par ^ 1) * rmax + rl] = v;
            if (pivot && r < fs) offer(v, r);
          }
          b += ng;
        }
#pragma unroll 2
        for (; b < 16; b += ng) {
          Vec4<T>::ld(src + 4 * b, a);
          Vec4<T>::ld(u + 4 * b, x);
#pragma unroll
          for (int e = 0; e < 4; ++e) a[e] -= l * x[e];
          Vec4<T>::st(row + 4 * b, a);
        }
      }
    lu_best<T>(mk, mr);
    if (lane == 0) { s_key[warp] = mk; s_row[warp] = mr; }
    __syncthreads();
  }
  if (tg < ng)
    for (int j = tg; j < kb; j += ng)
      for (int r = tr; r < nr_my; r += rw) G[(rbeg + r) + (int64_t)(k0 + j) * n] = S[r * SR + j];
}

constexpr int GC_NT_CLUSTER = 512, GC_NT_GRID = 256;

template <typename T, bool CL>
static cudaError_t getrf_smem_t(const DevCtx& c, const Item* items, int n_items, int n_ctas, int csize, int nb,
                                int pivot, int rmax, uint64_t* xbuf, int* err, cudaStream_t s) {
  constexpr int NT = CL ? GC_NT_CLUSTER : GC_NT_GRID;
  const size_t smem = (size_t)rmax * (LuBits<T>::LD + 2) * sizeof(T);
  cudaFuncSetAttribute(k_getrf_smem<T, CL, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(n_ctas);
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  if (CL) {
    if (csize > 8) cudaFuncSetAttribute(k_getrf_smem<T, CL, NT>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = csize;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
  } else {
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = CL && csize == 1 ? 0 : 1;
  return cudaLaunchKernelEx(&cfg, k_getrf_smem<T, CL, NT>, c, items, n_items, nb, pivot, rmax, csize, xbuf, err);
}

void launch_getrf_smem(const DevCtx& c, const Item* items, int n_items, int n_ctas, int csize, int dtype, int nb,
                       int pivot, int rmax, uint64_t* xbuf, int* err, cudaStream_t s) {
  if (!n_items) return;
  if (nb > 64) throw std::invalid_argument("getrf_smem: panel wider than 64");
  if (csize > GC_CLUSTER) throw std::invalid_argument("getrf_smem: cluster too large");
  cudaError_t e;
  if (csize > 0) {
    e = dtype == F64 ? getrf_smem_t<double, true>(c, items, n_items, n_items * csize, csize, nb, pivot, rmax, nullptr, err, s)
                     : getrf_smem_t<float, true>(c, items, n_items, n_items * csize, csize, nb, pivot, rmax, nullptr, err, s);
  } else {
    if (n_ctas > GC_MAX_CTAS) throw std::invalid_argument("getrf_smem: too many CTAs");
    cudaMemsetAsync(xbuf, 0, sizeof(uint64_t) * (size_t)gc_words(n_ctas, n_items), s);
    e = dtype == F64 ? getrf_smem_t<double, false>(c, items, n_items, n_ctas, 0, nb, pivot, rmax, xbuf, err, s)
                     : getrf_smem_t<float, false>(c, items, n_items, n_ctas, 0, nb, pivot, rmax, xbuf, err, s);
  }
  if (e != cudaSuccess)
    throw std::runtime_error(std::string("LU panel launch failed: ") + cudaGetErrorString(e));
}

// Row interchanges of a panel (pivots of rows k0..k0+kb-1, kb = min(nb,
// fs - k0), applied in order) on the front's columns outside the panel and
// below a column limit.  Item: front, a = k0, b = first column of a
// 256-column chunk, c = column limit (0: n); one thread per column.  b = -1: no
// columns, but the front's row permutation, which the solves gather by.
constexpr int LASWP_THREADS = 256 + 32;

template <typename T>
__global__ void __launch_bounds__(LASWP_THREADS) k_laswp(DevCtx c, const Item* __restrict__ items, int nb) {
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, k0 = it.a;
  const int kb = min(nb, f.fs - k0);
  const int32_t* __restrict__ pv = c.piv + f.piv_off;
  if (threadIdx.x >= 256) {
    if (it.b >= 0) return;
    int32_t* __restrict__ perm = c.perm + f.piv_off;
    if (k0 == 0)
      for (int i = threadIdx.x - 256; i < f.fs; i += 32) perm[i] = i;
    __syncwarp();
    if (threadIdx.x == 256)
      for (int k = k0; k < k0 + kb; ++k) {
        const int p = pv[k];
        if (p != k) {
          const int32_t t = perm[k];
          perm[k] = perm[p];
          perm[p] = t;
        }
      }
    return;
  }
  const int j = it.b + threadIdx.x;
  const int jend = it.c > 0 ? min(it.c, n) : n;
  if (it.b < 0 || j >= jend || (j >= k0 && j < k0 + kb)) return;
  T* __restrict__ col = arena<T>(c) + f.off + (int64_t)j * n;
  for (int k = k0; k < k0 + kb; ++k) {
    const int p = pv[k];
    if (p != k) {
      const T t = col[k];
      col[k] = col[p];
      col[p] = t;
    }
  }
}

void launch_laswp(const DevCtx& c, const Item* items, int n_items, int dtype, int nb, cudaStream_t s) {
  if (!n_items) return;
  if (dtype == F64) k_laswp<double><<<n_items, LASWP_THREADS, 0, s>>>(c, items, nb);
  else k_laswp<float><<<n_items, LASWP_THREADS, 0, s>>>(c, items, nb);
}

constexpr int LUROW_CB = 16;   // columns per row-panel block

// A[k0:k0+kb, cols] <- L11^{-1} A[k0:k0+kb, cols]  (unit lower), cols >= k0+kb;
// item: front, a = k0, b = first column of the chunk, c = column limit (0: n);
// scale (null: not wanted): XsCtx::scale, raised by these columns
//
// Substitution in registers: Q lanes hold one column (lane q rows q, q+Q,
// ..), a step's solved entry goes to the others by one shuffle, L comes
// from shared memory in the lanes' order, and nothing waits at a block
// barrier after L is staged.  Bound by the
// multiply-adds (2016 per column; FP64 at about 2 per clock and SM, which
// is why the chunk is narrow: 16 columns spread a panel over every SM) and by the
// chain of 64 steps.  A warp's FP64 multiply-add takes its scheduler 64 clocks, so
// FP64 columns take eight lanes (four warps per CTA, one per scheduler, and half
// the multiply-adds between two steps), FP32 ones four.  Measured on GB300 against a
// column per thread (64
// columns per CTA, a block barrier per row): 24^3 p = 3 BF16-split LU, 534
// launches, 38.7 -> 7.9 ms; FP64, the smallest launches, four lanes 29 us, eight 18;
// 12^3 p = 3, 200 launches, 6.5 -> 5.0 ms.
template <typename T, int Q>
__global__ void __launch_bounds__(Q * LUROW_CB) k_lu_row_update(DevCtx c, const Item* __restrict__ items, int nb,
                                                                int* __restrict__ scale) {
  constexpr int NU = 64 / Q, LQ = NU + 2;      // rows per lane; their L entries' row in shared memory (no bank conflicts)
  constexpr int NT = Q * LUROW_CB;
  __shared__ __align__(16) T L[64 * Q * LQ];   // L[(Q k + q) LQ + u] = L11[q + Q u][k]
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, k0 = it.a;
  const int kb = min(nb, f.fs - k0);
  const int cend = it.c > 0 ? min(it.c, n) : n;    // columns < cend (item c; 0: all)
  T* __restrict__ G = arena<T>(c) + f.off;
  const int q = threadIdx.x & (Q - 1), col = it.b + threadIdx.x / Q;
  const bool in = col < cend;
  T* __restrict__ X = G + k0 + q + (int64_t)col * n;
  T x[NU];
#pragma unroll
  for (int u = 0; u < NU; ++u) x[u] = in && q + Q * u < kb ? X[Q * u] : T(0);
  {
    const int i = threadIdx.x & 63;            // row of L11
#pragma unroll 16
    for (int k = threadIdx.x >> 6; k < 64; k += NT / 64)
      L[(Q * k + (i & (Q - 1))) * LQ + i / Q] = i > k && i < kb ? G[(k0 + i) + (int64_t)(k0 + k) * n] : T(0);
  }
  __syncthreads();
#pragma unroll
  for (int b = 0; b < NU; ++b) {
#pragma unroll
    for (int r = 0; r < Q; ++r) {
      const T xk = __shfl_sync(0xffffffffu, x[b], r, Q);
      const T* __restrict__ l = L + (Q * (Q * b + r) + q) * LQ;
      if (q > r) x[b] -= l[b] * xk;
#pragma unroll
      for (int u = b + 1; u < NU; ++u) x[u] -= l[u] * xk;
    }
  }
#pragma unroll
  for (int u = 0; u < NU; ++u)
    if (in && q + Q * u < kb) X[Q * u] = x[u];
  if (!scale) return;
  // how near each row comes to a column's largest entry, over the CTA's columns
  int* s_e = reinterpret_cast<int*>(L);        // [row][column], rows of 17
  static_assert(sizeof(L) >= 64 * (LUROW_CB + 1) * sizeof(int), "room for the words");
  int e[NU], cm = 0;
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    e[u] = in && q + Q * u < kb ? XsType<T>::expo(x[u]) : 0;
    cm = max(cm, e[u]);
  }
#pragma unroll
  for (int o = 1; o < Q; o <<= 1) cm = max(cm, __shfl_xor_sync(0xffffffffu, cm, o));
  __syncthreads();                             // L has been read
#pragma unroll
  for (int u = 0; u < NU; ++u) s_e[(q + Q * u) * (LUROW_CB + 1) + threadIdx.x / Q] = e[u] ? XS_SCALE0 + e[u] - cm : 0;
  __syncthreads();
  if (threadIdx.x >= kb) return;
  int v = 0;
#pragma unroll
  for (int j = 0; j < LUROW_CB; ++j) v = max(v, s_e[threadIdx.x * (LUROW_CB + 1) + j]);
  if (v) atomicMax(scale + f.piv_off + k0 + threadIdx.x, v);
}

void launch_lu_row_update(const DevCtx& c, const Item* items, int n_items, int dtype, int nb, int* scale,
                          cudaStream_t s) {
  if (!n_items) return;
  if (nb != 64) throw std::invalid_argument("lu_row_update: panels are 64 columns wide");
  if (dtype == F64) k_lu_row_update<double, 8><<<n_items, 8 * LUROW_CB, 0, s>>>(c, items, nb, scale);
  else k_lu_row_update<float, 4><<<n_items, 4 * LUROW_CB, 0, s>>>(c, items, nb, scale);
}

// Inverses of a large LU front's diagonal blocks, for the flag-driven solves:
// L_bb (unit lower) and U_bb, 64 x 64, zero outside their triangles and past
// the block's kb rows.  Item: front, a = b.  Substitution in registers as in
// k_lu_row_update; U through its
// transpose, (U^T)^{-1} by rows being U^{-1} by columns.  One launch per level
// after its fronts are factored: every block of every front at once, eight CTAs
// each (L or U, 16 columns of the identity, whose rows above are zero and
// skipped).  Bound by the multiply-adds of a CTA: measured on GB300, FP64, 6^3
// p = 3 (25 and 19 blocks) 0.32 ms with one CTA per block, 0.15 so; 12^3 p = 3 0.77, 0.57.
template <typename T, int Q>
__global__ void __launch_bounds__(Q * LUROW_CB) k_lu_dinv(DevCtx c, const Item* __restrict__ items) {
  constexpr int NU = 64 / Q, LQ = NU + 2, NT = Q * LUROW_CB;
  __shared__ __align__(16) T L[64 * Q * LQ];   // L[(Q k + q) LQ + u] = M[q + Q u][k]
  __shared__ T rd[64];
  const Item it = items[blockIdx.x >> 3];
  const int upper = (blockIdx.x >> 2) & 1, first = LUROW_CB * (blockIdx.x & 3);     // first column
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, fs = f.fs, k0 = 64 * it.a;
  const int kb = min(64, fs - k0), nfb = (fs + 63) / 64;
  const T* __restrict__ G = arena<T>(c) + f.off + k0 + (int64_t)k0 * n;
  T* __restrict__ D = (sizeof(T) == 8 ? (T*)c.dinv64 : (T*)c.dinv32) + f.dinv_off + (int64_t)it.a * 4096;
  const int q = threadIdx.x & (Q - 1), col = first + threadIdx.x / Q;
#pragma unroll 8
  for (int e = threadIdx.x; e < 4096; e += NT) {
    const int i = e & 63, k = e >> 6;              // entry (i, k) of the block, column k
    const T v = i < kb && k < kb ? G[i + (int64_t)k * n] : (i == k ? T(1) : T(0));
    if (!upper) L[(Q * k + (i & (Q - 1))) * LQ + i / Q] = i > k ? v : T(0);
    else L[(Q * i + (k & (Q - 1))) * LQ + k / Q] = k > i ? v : T(0);   // U^T: entry (k, i)
    if (i == k) rd[i] = upper ? v : T(1);
  }
  __syncthreads();
  T x[NU];
#pragma unroll
  for (int u = 0; u < NU; ++u) x[u] = q + Q * u == col ? T(1) : T(0);
#pragma unroll
  for (int b = 0; b < NU; ++b) {
    if (Q * b < first) continue;                   // rows above the columns' first one are zero
#pragma unroll
    for (int r = 0; r < Q; ++r) {
      if (upper && q == r) x[b] /= rd[Q * b + r];
      const T xk = __shfl_sync(0xffffffffu, x[b], r, Q);
      const T* __restrict__ l = L + (Q * (Q * b + r) + q) * LQ;
      if (q > r) x[b] -= l[b] * xk;
#pragma unroll
      for (int u = b + 1; u < NU; ++u) x[u] -= l[u] * xk;
    }
  }
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    const int i = q + Q * u;                       // entry (i, col) of M^{-1}
    const T v = i < kb && col < kb && i >= col ? x[u] : T(0);
    if (!upper) D[col * 64 + i] = v;
    else D[(int64_t)nfb * 4096 + i * 64 + col] = v;
  }
}

void launch_lu_dinv(const DevCtx& c, const Item* items, int n_items, int dtype, cudaStream_t s) {
  if (!n_items) return;
  if (dtype == F64) k_lu_dinv<double, 8><<<8 * n_items, 8 * LUROW_CB, 0, s>>>(c, items);
  else k_lu_dinv<float, 4><<<8 * n_items, 4 * LUROW_CB, 0, s>>>(c, items);
}

// ---------------------------------------------------------------------------
// FP64 <-> FP32 panel conversion (mixed precision bookkeeping)
// ---------------------------------------------------------------------------
__global__ void k_convert(DevCtx c, const Item* __restrict__ items, int to_f32) {
  const Item it = items[blockIdx.y];
  const FrontDev f = c.fronts[it.front];
  const int64_t nn = (int64_t)f.n * f.n;
  const int64_t o64 = ((int64_t)it.a << 32) | (uint32_t)it.b;   // FP64 shadow offset
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nn;
       i += (int64_t)gridDim.x * blockDim.x) {
    if (to_f32) c.a32[f.off + i] = (float)c.a64[o64 + i];
    else c.a64[o64 + i] = (double)c.a32[f.off + i];
  }
}

void launch_convert_panels(const DevCtx& c, const Item* items, int n_items, int to_f32,
                           cudaStream_t s) {
  if (!n_items) return;
  dim3 g(64, n_items);
  k_convert<<<g, 256, 0, s>>>(c, items, to_f32);
}

}  // namespace uhm_gpu
