// Tree forward/backward solves and the element-wise residual.
//
// Reference steps restated here:
//   forward   solve_chol_1_hier / solve_lu_piv_1_hier + Helper_::merge_rhs_x
//             (UHM/src/matrix/uhm/fla/chol/solve.cxx:152-168,
//              fla/lu_piv/solve.cxx:161-187, helper.hxx:253-301)
//   backward  solve_chol_2_hier / solve_lu_piv_2_hier + Helper_::branch_rhs_x
//             (chol/solve.cxx:187-202, lu_piv/solve.cxx:211-231, helper.hxx:302-331)
// The right-hand side lives in a global vector in elimination order; the
// dofs eliminated at front f are g[g0 .. g0+fs).  A child's updated bottom
// block (xb) is gathered into its parent exactly like the matrix extend-add.
//
// Residual: r = b - sum_e P_e^T A_e P_e x on the retained FP64 element
// matrices (the unassembled operator), followed by a deterministic per-dof
// gather in element order.  This replaces the factor-based check_* of
// UHM/src/matrix/uhm/fla/chol/check.cxx:40-111.
#include "k_common.cuh"

namespace uhm_gpu {

// the empty value of the flag-driven solves' hand-off words (a signalling
// NaN: no arithmetic result or conversion produces it)
constexpr unsigned long long HAND_EMPTY = 0x7FF4DEAD7FF4DEADull;

// The gathers and stores between the global vector and the fronts' slabs go by
// groups of right-hand sides, a CTA each (grid.y): they are bound by the latency of
// their dependent loads.  Measured on GB300, 16 right-hand sides one after the
// other and so: forward gathers of two solves 2.57 -> 0.80 ms, stores 0.77 -> 0.13.

// z = [g[g0 .. g0+fs); 0] + sum over children of their xb (extend-add);
// item: front, a = first row, b = rows (0: all), c = 1 for a front of the
// 64-row flag-driven solves (LU with pivoting: its factor rows are gathered in
// the order of the front's row permutation)
template <int NQ>
__global__ void __launch_bounds__(256) k_fwd_gather(DevCtx c, const Item* __restrict__ items,
                                                    const double* __restrict__ g, int64_t ldg,
                                                    int method) {
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n;
  double* __restrict__ z = c.vec + f.voff;
  double* __restrict__ y = z + (int64_t)n * c.n_rhs;
  double* __restrict__ w = y + (int64_t)n * c.n_rhs;
  const int32_t* __restrict__ inv = c.inv + f.inv_off;
  // rows [it.a, it.a + it.b) of the front (it.b == 0: all rows; only then
  // are pivots applied, which needs the whole gathered vector)
  const int I0 = it.a, I1 = it.b > 0 ? min(n, it.a + it.b) : n;
  const int32_t* __restrict__ perm = method == M_LU_PIV && it.c ? c.perm + f.piv_off : nullptr;
  // the sources decoded once per CTA (in source order): a child's updated
  // bottom block and its leading dimension, null for an element source
  constexpr int GMAXSRC = 64;
  __shared__ const double* s_xb[GMAXSRC];
  __shared__ int s_ld[GMAXSRC];
  const int ns = min(f.nsrc, GMAXSRC);
  for (int s = threadIdx.x; s < ns; s += blockDim.x) {
    const SrcDev sd = c.srcs[f.src0 + s];
    if (sd.is_child) {
      const FrontDev ch = c.fronts[sd.slot];
      s_xb[s] = c.vec + ch.voff + ch.fs;
      s_ld[s] = ch.n;
    } else {
      s_xb[s] = nullptr;
      s_ld[s] = 0;
    }
  }
  __syncthreads();
  // right-hand sides q0 .. q0 + nq - 1 (grid.y), together: a row's maps are read once
  const int q0 = NQ == 1 ? 0 : NQ * blockIdx.y, nq = NQ == 1 ? 1 : min(NQ, c.n_rhs - q0);
  for (int R = I0 + threadIdx.x; R < I1; R += blockDim.x) {
    const int I = perm && R < f.fs ? perm[R] : R;
    double acc[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) acc[q] = q < nq && I < f.fs ? g[(f.g0 + I) + (q0 + q) * ldg] : 0.0;
    for (int s = 0; s < ns; ++s) {
      const double* xb = s_xb[s];
      if (!xb) continue;
      const int is = inv[(int64_t)s * n + I];
      if (is < 0) continue;
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        if (q < nq) acc[q] += xb[is + (int64_t)(q0 + q) * s_ld[s]];
    }
    for (int s = ns; s < f.nsrc; ++s) {
      const SrcDev sd = c.srcs[f.src0 + s];
      if (!sd.is_child) continue;
      const int is = inv[(int64_t)s * n + I];
      if (is < 0) continue;
      const FrontDev ch = c.fronts[sd.slot];
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        if (q < nq) acc[q] += c.vec[ch.voff + ch.fs + is + (int64_t)(q0 + q) * ch.n];
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      if (q >= nq) break;
      const int64_t at = R + (int64_t)(q0 + q) * n;
      z[at] = acc[q];
      // fronts of the 64-row flag-driven and chain solves: their y factor
      // rows (solutions) and w factor rows (partial sums) are forward
      // hand-offs, emptied here (the forward launch comes after)
      if (it.c && R < f.fs) {
        y[at] = __longlong_as_double((long long)HAND_EMPTY);
        w[at] = __longlong_as_double((long long)HAND_EMPTY);
      }
    }
  }
  __syncthreads();
  if (method == M_LU_PIV && it.b == 0 && threadIdx.x < nq) {
    // FLA_Apply_pivots(LEFT, NO_TRANSPOSE, p, xt): sequential interchanges
    const int32_t* __restrict__ piv = c.piv + f.piv_off;
    double* zq = z + (int64_t)(q0 + threadIdx.x) * n;
    for (int k = 0; k < f.fs; ++k) {
      const int p = piv[k];
      if (p != k) { double t = zq[k]; zq[k] = zq[p]; zq[p] = t; }
    }
  }
}

void launch_fwd_gather(const DevCtx& c, const Item* items, int n_items, const double* g,
                       int64_t ldg, int method, cudaStream_t s) {
  if (!n_items) return;
  if (c.n_rhs == 1) k_fwd_gather<1><<<n_items, 256, 0, s>>>(c, items, g, ldg, method);
  else k_fwd_gather<4><<<dim3(n_items, (c.n_rhs + 3) / 4), 256, 0, s>>>(c, items, g, ldg, method);
}

// whole-front forward sweep: z_t <- L^{-1} z_t ; z_b <- z_b - ABL z_t
template <typename T, int NT>
__global__ void __launch_bounds__(NT) k_fwd_small(DevCtx c, const Item* __restrict__ items,
                                                  int method) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* z = reinterpret_cast<double*>(smem_raw);
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, fs = f.fs, nr = c.n_rhs;
  const T* __restrict__ G = arena<T>(c) + f.off;
  double* __restrict__ zg = c.vec + f.voff;
  for (int idx = threadIdx.x; idx < n * nr; idx += NT) z[idx] = zg[idx];
  __syncthreads();
  const bool unit = method != M_CHOL;
  for (int j = 0; j < fs; ++j) {
    if (!unit) {
      const double d = (double)G[j + (int64_t)j * n];
      if (threadIdx.x < nr) z[j + threadIdx.x * n] /= d;
      __syncthreads();
    }
    const int h = n - j - 1;
    for (int idx = threadIdx.x; idx < h * nr; idx += NT) {
      const int i = j + 1 + idx % h, q = idx / h;
      z[i + q * n] -= (double)G[i + (int64_t)j * n] * z[j + q * n];
    }
    __syncthreads();
  }
  // y (second slab) receives the eliminated part, z keeps the updated bottom
  double* __restrict__ yg = zg + (int64_t)n * nr;
  for (int idx = threadIdx.x; idx < n * nr; idx += NT) {
    const int i = idx % n;
    if (i < fs) yg[idx] = z[idx];
    else zg[idx] = z[idx];
  }
}

// Cholesky small fronts with the factor panel (n x fs) staged in shared
// memory by one batch of loads: every column step then works on shared data
// (no global round trip per column).  The right-hand sides are solved in the
// factor's precision (as in the flag-driven solves of large fronts): FP32
// fronts take no FP64 arithmetic, which runs at a small fraction of the FP32 rate
// on this GPU; only where a launch's largest panel and right-hand sides pass
// SMALL_SOLVE_FP32 bytes do they, as without staging.  The pivots' reciprocals are formed once, all at a time (a
// division per column was most of an FP64 step); the solved entries are scaled by them
// where they are used.  From WARP_RHS right-hand sides on each warp takes its own
// ones and no block barrier is left in the sweep; below, the block shares
// the rows and crosses one per column.  Measured on GB300: 125-row FP64 front,
// one right-hand side, forward 121 -> 35 us, backward 172 -> 31 (its panel now
// staged too); 4,096 fronts of 125 (27) 106 -> 77 and 240 -> 68; 12 meshes, 16
// right-hand sides, FP32 1.08 -> 0.80 ms and 1.95 -> 1.03.
constexpr int WARP_RHS = 4;
constexpr int SMALL_SOLVE_FP32 = 96 * 1024;

// the front's factor columns into Ls (n x fs), the reciprocals of its pivots
// into rd, the slab v (n x n_rhs) into z
template <typename T, typename CT, int NT>
__device__ __forceinline__ void small_stage(const T* __restrict__ G, const double* __restrict__ v, int n, int fs,
                                            int nr, CT* z, CT* rd, T* Ls) {
  const int tot = n * fs;
  for (int i0 = 0; i0 < tot; i0 += 8 * NT) {
    T x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int idx = i0 + threadIdx.x + u * NT;
      x[u] = idx < tot ? G[idx] : T(0);        // columns 0..fs-1 are contiguous (ld n)
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int idx = i0 + threadIdx.x + u * NT;
      if (idx < tot) Ls[idx] = x[u];
    }
  }
  for (int idx = threadIdx.x; idx < n * nr; idx += NT) z[idx] = (CT)v[idx];
  for (int j = threadIdx.x; j < fs; j += NT) rd[j] = CT(1) / (CT)G[j + (int64_t)j * n];
  __syncthreads();
}

// this thread's right-hand sides q0, q0 + qs, .. and rows i0, i0 + is, .. of a sweep
struct SmallShare {
  int q0, qs, i0, is;
  bool warp;
  __device__ __forceinline__ SmallShare(int nr, int nt) {
    warp = nr >= WARP_RHS;
    q0 = warp ? threadIdx.x >> 5 : 0;
    qs = warp ? nt / 32 : 1;
    i0 = warp ? threadIdx.x & 31 : threadIdx.x;
    is = warp ? 32 : nt;
  }
  __device__ __forceinline__ void sync() const {
    if (warp) __syncwarp();
    else __syncthreads();
  }
};

template <typename T, typename CT, int NT>
__global__ void __launch_bounds__(NT) k_fwd_small_staged(DevCtx c, const Item* __restrict__ items) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, fs = f.fs, nr = c.n_rhs;
  CT* z = reinterpret_cast<CT*>(smem_raw);
  CT* rd = z + (size_t)n * nr;
  T* Ls = reinterpret_cast<T*>(rd + fs);
  double* __restrict__ zg = c.vec + f.voff;
  small_stage<T, CT, NT>(arena<T>(c) + f.off, zg, n, fs, nr, z, rd, Ls);
  const SmallShare sh(nr, NT);
  for (int q = sh.q0; q < nr; q += sh.qs) {
    CT* zq = z + q * n;
    for (int j = 0; j < fs; ++j) {
      const CT zj = zq[j] * rd[j];
      const T* col = Ls + j * n;
      for (int i = j + 1 + sh.i0; i < n; i += sh.is) zq[i] -= (CT)col[i] * zj;
      sh.sync();
    }
  }
  __syncthreads();
  double* __restrict__ yg = zg + (int64_t)n * nr;
  for (int q = 0; q < nr; ++q)
    for (int i = threadIdx.x; i < n; i += NT) {
      if (i < fs) yg[i + (int64_t)q * n] = (double)(z[i + q * n] * rd[i]);
      else zg[i + (int64_t)q * n] = (double)z[i + q * n];
    }
}

// x_F = L_FF^{-T} (y_F - L_SF^T x_S): the Schur-row products for all factor
// columns at once, then the small triangular solve column by column.
template <typename T, typename CT, int NT>
__global__ void __launch_bounds__(NT) k_bwd_small_staged(DevCtx c, const Item* __restrict__ items,
                                                         double* __restrict__ g, int64_t ldg) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, fs = f.fs, nr = c.n_rhs;
  CT* z = reinterpret_cast<CT*>(smem_raw);
  CT* rd = z + (size_t)n * nr;
  T* Ls = reinterpret_cast<T*>(rd + fs);
  const double* __restrict__ yg = c.vec + f.voff + (int64_t)n * nr;   // y slab
  small_stage<T, CT, NT>(arena<T>(c) + f.off, yg, n, fs, nr, z, rd, Ls);
  const SmallShare sh(nr, NT);
  for (int q = sh.q0; q < nr; q += sh.qs) {
    CT* zq = z + q * n;
    for (int j = sh.i0; j < fs; j += sh.is) {
      CT s0 = CT(0), s1 = CT(0);
      const T* col = Ls + (size_t)j * n;
      int i = fs;
      for (; i + 1 < n; i += 2) {
        s0 += (CT)col[i] * zq[i];
        s1 += (CT)col[i + 1] * zq[i + 1];
      }
      if (i < n) s0 += (CT)col[i] * zq[i];
      zq[j] -= s0 + s1;
    }
    sh.sync();
    for (int j = fs - 1; j > 0; --j) {
      const CT xj = zq[j] * rd[j];
      for (int i = sh.i0; i < j; i += sh.is) zq[i] -= (CT)Ls[j + i * n] * xj;
      sh.sync();
    }
  }
  __syncthreads();
  for (int q = 0; q < nr; ++q)
    for (int i = threadIdx.x; i < fs; i += NT) g[(f.g0 + i) + q * ldg] = (double)(z[i + q * n] * rd[i]);
}

void launch_fwd_small(const DevCtx& c, const Item* items, int n_items, int dtype, int method,
                      int staged_bytes, cudaStream_t s) {
  if (!n_items) return;
  if (method == M_CHOL && staged_bytes > 0) {
    const auto kernel = dtype == F64                       ? k_fwd_small_staged<double, double, 128>
                        : staged_bytes <= SMALL_SOLVE_FP32 ? k_fwd_small_staged<float, float, 128>
                                                           : k_fwd_small_staged<float, double, 128>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, staged_bytes);
    kernel<<<n_items, 128, staged_bytes, s>>>(c, items);
    return;
  }
  // the largest small front bounds the shared slab; 64 KB covers n*n_rhs <= 8192
  size_t sm = 8192 * sizeof(double);
  if (dtype == F64) {
    cudaFuncSetAttribute(k_fwd_small<double, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_fwd_small<double, 256><<<n_items, 256, sm, s>>>(c, items, method);
  } else {
    cudaFuncSetAttribute(k_fwd_small<float, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_fwd_small<float, 256><<<n_items, 256, sm, s>>>(c, items, method);
  }
}

// backward: xb <- g[schur dofs]
__global__ void __launch_bounds__(256) k_bwd_prepare(DevCtx c, const Item* __restrict__ items,
                                                     const double* __restrict__ g, int64_t ldg) {
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  double* __restrict__ y = c.vec + f.voff + (int64_t)f.n * c.n_rhs;
  const int32_t* __restrict__ sgi = c.sgi + f.sgi_off;
  const int q = blockIdx.y;
  for (int j = threadIdx.x; j < f.ss; j += blockDim.x) y[f.fs + j + (int64_t)q * f.n] = g[sgi[j] + q * ldg];
}

void launch_bwd_prepare(const DevCtx& c, const Item* items, int n_items, int dtype, int method,
                        const double* g, int64_t ldg, cudaStream_t s) {
  (void)dtype; (void)method;
  if (!n_items) return;
  k_bwd_prepare<<<dim3(n_items, c.n_rhs), 256, 0, s>>>(c, items, g, ldg);
}

template <int NT>
__device__ double block_sum(double v, double* s_red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if (lane == 0) s_red[warp] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0) {
    for (int w = 0; w < NT / 32; ++w) r += s_red[w];
    s_red[NT / 32] = r;
  }
  __syncthreads();
  r = s_red[NT / 32];
  __syncthreads();
  return r;
}

// whole-front backward sweep and store of x_t into g
template <typename T, int NT>
__global__ void __launch_bounds__(NT) k_bwd_small(DevCtx c, const Item* __restrict__ items,
                                                  int method, double* __restrict__ g, int64_t ldg) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double s_red[NT / 32 + 1];
  double* z = reinterpret_cast<double*>(smem_raw);
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, fs = f.fs, nr = c.n_rhs;
  const T* __restrict__ G = arena<T>(c) + f.off;
  double* __restrict__ zg = c.vec + f.voff + (int64_t)n * nr;   // y slab
  for (int idx = threadIdx.x; idx < n * nr; idx += NT) z[idx] = zg[idx];
  __syncthreads();
  const bool chol = method == M_CHOL;
  for (int q = 0; q < nr; ++q) {
    double* zq = z + q * n;
    for (int j = fs - 1; j >= 0; --j) {
      double part = 0.0;
      if (chol)
        for (int i = j + 1 + threadIdx.x; i < n; i += NT) part += (double)G[i + (int64_t)j * n] * zq[i];
      else
        for (int t = j + 1 + threadIdx.x; t < n; t += NT) part += (double)G[j + (int64_t)t * n] * zq[t];
      const double s = block_sum<NT>(part, s_red);
      if (threadIdx.x == 0) zq[j] = (zq[j] - s) / (double)G[j + (int64_t)j * n];
      __syncthreads();
    }
  }
  for (int q = 0; q < nr; ++q)
    for (int i = threadIdx.x; i < fs; i += NT) g[(f.g0 + i) + q * ldg] = z[i + q * n];
}

void launch_bwd_small(const DevCtx& c, const Item* items, int n_items, int dtype, int method,
                      double* g, int64_t ldg, int staged_bytes, cudaStream_t s) {
  if (!n_items) return;
  if (method == M_CHOL && staged_bytes > 0) {
    const auto kernel = dtype == F64                       ? k_bwd_small_staged<double, double, 128>
                        : staged_bytes <= SMALL_SOLVE_FP32 ? k_bwd_small_staged<float, float, 128>
                                                           : k_bwd_small_staged<float, double, 128>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, staged_bytes);
    kernel<<<n_items, 128, staged_bytes, s>>>(c, items, g, ldg);
    return;
  }
  size_t sm = 8192 * sizeof(double);
  if (dtype == F64) {
    cudaFuncSetAttribute(k_bwd_small<double, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_bwd_small<double, 256><<<n_items, 256, sm, s>>>(c, items, method, g, ldg);
  } else {
    cudaFuncSetAttribute(k_bwd_small<float, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_bwd_small<float, 256><<<n_items, 256, sm, s>>>(c, items, method, g, ldg);
  }
}

__global__ void __launch_bounds__(256) k_bwd_store(DevCtx c, const Item* __restrict__ items,
                                                   double* __restrict__ g, int64_t ldg) {
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const double* __restrict__ z = c.vec + f.voff + (int64_t)f.n * c.n_rhs;   // y slab
  const int q = blockIdx.y;
  for (int i = threadIdx.x; i < f.fs; i += blockDim.x) g[(f.g0 + i) + q * ldg] = z[i + (int64_t)q * f.n];
}

void launch_bwd_store(const DevCtx& c, const Item* items, int n_items, double* g, int64_t ldg,
                      cudaStream_t s) {
  if (!n_items) return;
  k_bwd_store<<<dim3(n_items, c.n_rhs), 256, 0, s>>>(c, items, g, ldg);
}

// ---------------------------------------------------------------------------
// element-wise residual
// ---------------------------------------------------------------------------
// y_e = A_e x_e  for every element (one CTA per element and group of NQ right-hand
// sides, which share A's entries and keep NQ independent sums going per row)
template <int NQ>
__global__ void __launch_bounds__(128) k_elem_gemv(const double* __restrict__ emat,
                                                   const int64_t* __restrict__ emat_off,
                                                   const int* __restrict__ elem_m,
                                                   const int64_t* __restrict__ emap_off,
                                                   const int32_t* __restrict__ emap,
                                                   const double* __restrict__ x, int64_t ldx,
                                                   double* __restrict__ y,
                                                   const int64_t* __restrict__ y_off, int n_rhs) {
  __shared__ double s_x[1024][NQ];
  const int e = blockIdx.x, q0 = NQ == 1 ? 0 : NQ * blockIdx.y, nq = NQ == 1 ? 1 : min(NQ, n_rhs - q0);
  const int m = elem_m[e];
  const double* __restrict__ A = emat + emat_off[e];
  const int32_t* __restrict__ map = emap + emap_off[e];
  double* __restrict__ ye = y + y_off[e] + (int64_t)q0 * m;
  for (int j0 = 0; j0 < m; j0 += 1024) {
    const int jn = min(1024, m - j0);
    __syncthreads();
    for (int j = threadIdx.x; j < jn; j += blockDim.x) {
      const double* xj = x + map[j0 + j] + q0 * ldx;
#pragma unroll
      for (int q = 0; q < NQ; ++q) s_x[j][q] = q < nq ? xj[q * ldx] : 0.0;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
      double acc[NQ];
#pragma unroll
      for (int q = 0; q < NQ; ++q) acc[q] = j0 && q < nq ? ye[i + (int64_t)q * m] : 0.0;
      for (int j = 0; j < jn; ++j) {
        const double a = A[i + (int64_t)(j0 + j) * m];
#pragma unroll
        for (int q = 0; q < NQ; ++q)
          if (q < nq) acc[q] += a * s_x[j][q];
      }
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        if (q < nq) ye[i + (int64_t)q * m] = acc[q];
    }
  }
}

void launch_elem_gemv(const double* emat, const int64_t* emat_off, const int* elem_m,
                      const int64_t* emap_off, const int32_t* emap, const double* x, int64_t ldx,
                      double* y, const int64_t* y_off, int n_elem, int n_rhs, cudaStream_t s) {
  if (!n_elem) return;
  if (n_rhs == 1)
    k_elem_gemv<1><<<n_elem, 128, 0, s>>>(emat, emat_off, elem_m, emap_off, emap, x, ldx, y, y_off, n_rhs);
  else if (n_rhs == 2)
    k_elem_gemv<2><<<n_elem, 128, 0, s>>>(emat, emat_off, elem_m, emap_off, emap, x, ldx, y, y_off, n_rhs);
  else
    k_elem_gemv<4><<<dim3(n_elem, (n_rhs + 3) / 4), 128, 0, s>>>(emat, emat_off, elem_m, emap_off, emap, x, ldx, y,
                                                                 y_off, n_rhs);
}

// r[i] = (sub_from_b ? b[i] - sum : sum), sum over the (element, row) list of dof i in order.
// idx entries index the flattened per-element y buffer (offset of row 0 of rhs 0 + row).
template <int NQ>
__global__ void k_dof_gather(const int64_t* __restrict__ ptr, const int64_t* __restrict__ idx,
                             const double* __restrict__ y, const double* __restrict__ b,
                             int64_t ldb, double* __restrict__ r, int64_t N, int n_rhs,
                             int sub_from_b) {
  const int q0 = NQ == 1 ? 0 : NQ * blockIdx.y, nq = NQ == 1 ? 1 : min(NQ, n_rhs - q0);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N;
       i += (int64_t)gridDim.x * blockDim.x) {
    double s[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) s[q] = 0.0;
    for (int64_t k = ptr[i]; k < ptr[i + 1]; ++k) {
      // idx encodes (element y offset + row) and the element's row count in the high bits
      const int64_t v = idx[k];
      const int64_t off = v & ((1LL << 40) - 1);
      const int64_t m = v >> 40;
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        if (q < nq) s[q] += y[off + (q0 + q) * m];
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      if (q < nq) r[i + (q0 + q) * ldb] = sub_from_b ? b[i + (q0 + q) * ldb] - s[q] : s[q];
  }
}

void launch_dof_gather(const int64_t* ptr, const int64_t* idx, const double* y, const double* b,
                       int64_t ldb, double* r, int64_t N, int n_rhs, int sub_from_b,
                       cudaStream_t s) {
  if (!N) return;
  int blocks = (int)std::min<int64_t>((N + 255) / 256, 152 * 16);
  if (n_rhs == 1) k_dof_gather<1><<<blocks, 256, 0, s>>>(ptr, idx, y, b, ldb, r, N, n_rhs, sub_from_b);
  else if (n_rhs == 2) k_dof_gather<2><<<blocks, 256, 0, s>>>(ptr, idx, y, b, ldb, r, N, n_rhs, sub_from_b);
  else
    k_dof_gather<4><<<dim3(blocks, (n_rhs + 3) / 4), 256, 0, s>>>(ptr, idx, y, b, ldb, r, N, n_rhs, sub_from_b);
}

// out[0] = max |v| (single-pass, deterministic: per-block max then a final block)
// max(a, b) of non-negative values that keeps a NaN (fmax drops it), so that
// a NaN anywhere in the vector reaches the result
__device__ __forceinline__ double nanmax(double a, double b) { return (b > a || b != b) ? b : a; }

__global__ void k_absmax_partial(const double* __restrict__ v, int64_t n, double* __restrict__ part) {
  __shared__ double s[256];
  double m = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    m = nanmax(m, fabs(v[i]));
  s[threadIdx.x] = m;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) s[threadIdx.x] = nanmax(s[threadIdx.x], s[threadIdx.x + o]);
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = s[0];
}

__global__ void k_absmax_final(const double* __restrict__ part, int np, double* __restrict__ out) {
  __shared__ double s[256];
  double m = 0.0;
  for (int i = threadIdx.x; i < np; i += blockDim.x) m = nanmax(m, part[i]);
  s[threadIdx.x] = m;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) s[threadIdx.x] = nanmax(s[threadIdx.x], s[threadIdx.x + o]);
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = s[0];
}

// out must hold 1 + 304 doubles (result, then partials)
void launch_absmax(const double* v, int64_t n, double* out, cudaStream_t s) {
  const int np = 304;
  k_absmax_partial<<<np, 256, 0, s>>>(v, n, out + 1);
  k_absmax_final<<<1, 256, 0, s>>>(out + 1, np, out);
}

// Maximum |v| per tree of a forest.  v holds n_rhs columns of ng dofs;
// tree[i] is the tree of dof i.  The dofs of one tree are not contiguous
// (numbering runs generation by generation over all trees) but come in long
// runs (a front's factor dofs are consecutive), so each thread scans 32
// consecutive entries and flushes its running maximum with one atomicMax on
// the bit pattern (non-negative doubles order like their bits; NaN, kept by
// the comparison below, orders above every number) whenever the tree changes.
// out[t] must be zeroed before the launch.
__global__ void k_absmax_tree(const double* __restrict__ v, int64_t nv, int64_t ng,
                              const int* __restrict__ tree, unsigned long long* __restrict__ out) {
  const int64_t i0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) * 32;
  if (i0 >= nv) return;
  const int64_t i1 = i0 + 32 < nv ? i0 + 32 : nv;
  int64_t row = i0 % ng;
  int cur = -1;
  double m = 0.0;
  for (int64_t i = i0; i < i1; ++i) {
    const int t = tree[row];
    if (t != cur) {
      if (cur >= 0) atomicMax(&out[cur], (unsigned long long)__double_as_longlong(m));
      cur = t;
      m = 0.0;
    }
    const double a = fabs(v[i]);
    if (a > m || a != a) m = a;
    if (++row == ng) row = 0;
  }
  atomicMax(&out[cur], (unsigned long long)__double_as_longlong(m));
}

void launch_absmax_tree(const double* v, int64_t nv, int64_t ng, const int* tree, int n_trees,
                        unsigned long long* out, cudaStream_t s) {
  cudaMemsetAsync(out, 0, sizeof(unsigned long long) * n_trees, s);
  if (!nv) return;
  const int64_t threads = (nv + 31) / 32;
  k_absmax_tree<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(v, nv, ng, tree, out);
}

__global__ void k_axpy(double* __restrict__ y, const double* __restrict__ x, int64_t n, double a) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    y[i] += a * x[i];
}

void launch_axpy(double* y, const double* x, int64_t n, double alpha, cudaStream_t s) {
  if (!n) return;
  int blocks = (int)std::min<int64_t>((n + 255) / 256, 152 * 8);
  k_axpy<<<blocks, 256, 0, s>>>(y, x, n, alpha);
}

}  // namespace uhm_gpu

namespace uhm_gpu {

// ||A||_inf of the assembled operator A = sum_e P_e^T A_e P_e, exactly, on the
// device.  Entry (i, J) of A is summed over the elements that contain both
// dofs; the element of smallest index among them (the "owner") computes that
// sum and adds |A(i, J)| to its partial row sum for row i.  Partial sums are
// then gathered per dof in element order (k_dof_gather), so the result is
// deterministic.  dof_el lists, per dof, (element, local row) sorted by element.
__global__ void __launch_bounds__(128) k_anorm_partial(const double* __restrict__ emat,
                                                       const int64_t* __restrict__ emat_off,
                                                       const int* __restrict__ elem_m,
                                                       const int64_t* __restrict__ emap_off,
                                                       const int32_t* __restrict__ emap,
                                                       const int64_t* __restrict__ dof_ptr,
                                                       const int2* __restrict__ dof_el,
                                                       double* __restrict__ part,
                                                       const int64_t* __restrict__ y_off) {
  const int e = blockIdx.x;
  const int m = elem_m[e];
  const int32_t* __restrict__ map = emap + emap_off[e];
  for (int l = threadIdx.x; l < m; l += blockDim.x) {
    const int32_t i = map[l];
    const int64_t a0 = dof_ptr[i], a1 = dof_ptr[i + 1];
    double s = 0.0;
    for (int j = 0; j < m; ++j) {
      const int32_t J = map[j];
      const int64_t b0 = dof_ptr[J], b1 = dof_ptr[J + 1];
      // merge-intersect the two element lists
      int64_t a = a0, b = b0;
      int owner = -1;
      double v = 0.0;
      while (a < a1 && b < b1) {
        const int2 pa = dof_el[a], pb = dof_el[b];
        if (pa.x < pb.x) ++a;
        else if (pb.x < pa.x) ++b;
        else {
          if (owner < 0) owner = pa.x;
          const int me = elem_m[pa.x];
          v += emat[emat_off[pa.x] + pa.y + (int64_t)pb.y * me];
          ++a;
          ++b;
        }
      }
      if (owner == e) s += fabs(v);
    }
    part[y_off[e] + l] = s;
  }
}

void launch_anorm_partial(const double* emat, const int64_t* emat_off, const int* elem_m,
                          const int64_t* emap_off, const int32_t* emap, const int64_t* dof_ptr,
                          const int2* dof_el, double* part, const int64_t* y_off, int n_elem,
                          cudaStream_t s) {
  if (!n_elem) return;
  k_anorm_partial<<<n_elem, 128, 0, s>>>(emat, emat_off, elem_m, emap_off, emap, dof_ptr, dof_el,
                                         part, y_off);
}

}  // namespace uhm_gpu

namespace uhm_gpu {

// ===========================================================================
// Flag-driven level solves of large Cholesky fronts.
//
// One launch covers every large front of a level.  The rows of a front are cut
// into 64-row blocks: factor blocks [64b, min(64b+64, fs)) and ABL blocks
// starting at fs.  A CTA takes a ticket (atomic counter) and processes the
// item of that rank; items are ordered so that each CTA only waits for blocks
// owned by CTAs with smaller tickets, which are already running -- progress
// is guaranteed whatever the residency.  A finished block's solution is
// published as self-validating hand-off words (below).  Every wait is bounded (error
// flag, no hang).
// Forward:  x_b = L_bb^{-1} (z_b - sum_{j<b} L_bj x_j)
// Backward: x_b = L_bb^{-T} (y_b - sum_{r > block b} L_rb^T x_r)
// with L_bb^{-1} precomputed at factorisation (64 x 64, dinv arenas).
// ===========================================================================
constexpr int FB = 64;
constexpr int SF_NR = FLAG_NR;    // right-hand sides per launch (256-row and chain kernels)

UHM_DEFINE_WAIT_LIMIT(set_wait_limit_solve, 1u << 22)

template <typename T> __device__ __forceinline__ const T* dinv_arena(const DevCtx& c);
template <> __device__ __forceinline__ const double* dinv_arena<double>(const DevCtx& c) { return c.dinv64; }
template <> __device__ __forceinline__ const float* dinv_arena<float>(const DevCtx& c) { return c.dinv32; }

// Hand-off words of the 64-row flag-driven solves.  A block's solution is
// published as plain FP64 words that carry their own completion: before the
// launch every word of the hand-off holds HAND_EMPTY, a signalling NaN that
// no arithmetic result or conversion can produce, and the solving CTA
// overwrites it with the value (one relaxed 8-byte store per entry, single-
// copy atomic).  A reader polls the words themselves: once none of them is
// HAND_EMPTY it holds the values, with no flag, no fence on the writer's side
// and no second round trip on the reader's.  The forward hand-off is the y
// slab's factor rows (filled by the gather before the launch), the backward
// one the z slab's factor rows (filled by the forward CTA of the block, after
// its last read of them).
__device__ __forceinline__ unsigned long long ld_hand(const double* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_hand(double* p, double v) {
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(__double_as_longlong(v)) : "memory");
}

// Where the first hand-off wait of a solve gave up (0: none): kind * 10^8 +
// awaited block * 10^4 + the waiting block (kind 1 forward rows, 2 backward
// columns, 3 forward chain, 4 backward chain), read and cleared by the host
// with the error word.
__device__ int g_solve_where = 0;
__device__ __forceinline__ int wait_code(int kind, int awaited, int own) {
  return kind * 100000000 + min(awaited, 9999) * 10000 + min(own, 9999);
}
int solve_wait_where() {
  int v = 0;
  const int zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_solve_where, sizeof(int)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(g_solve_where, &zero, sizeof(int));
  return v;
}

// One warp: the 64 hand-off words of one block and right-hand side
// (entries lane and lane + 32; entries at or past kb read as 0).
struct HandWords {
  unsigned long long w0, w1;
  __device__ __forceinline__ void load(const double* base, int kb) {
    const int lane = threadIdx.x & 31;
    w0 = lane < kb ? ld_hand(base + lane) : 0ull;
    w1 = lane + 32 < kb ? ld_hand(base + lane + 32) : 0ull;
  }
  __device__ __forceinline__ bool full() const {
    return __all_sync(0xffffffffu, w0 != HAND_EMPTY && w1 != HAND_EMPTY);
  }
  // bounded wait until every word is written; false (and *err = 2, where
  // recorded) when the limit runs out
  __device__ __forceinline__ bool wait(const double* base, int kb, int* err, int where) {
    const uint32_t lim = g_wait_limit;
    for (uint32_t i = 0; !full(); ++i) {
      if (i >= lim) {
        if ((threadIdx.x & 31) == 0) {
          atomicExch(err, 2);
          atomicCAS(&g_solve_where, 0, where);
        }
        return false;
      }
      __nanosleep(32);
      load(base, kb);
    }
    return true;
  }
  template <typename CT>
  __device__ __forceinline__ void stage(CT* dst) const {
    const int lane = threadIdx.x & 31;
    dst[lane] = (CT)__longlong_as_double(w0);
    dst[lane + 32] = (CT)__longlong_as_double(w1);
  }
};

// The hand-off words of one block for NQ right-hand sides: warp q < nq polls and
// stages right-hand side q (with one warp polling them in turn, each took a round
// trip of its own on the chain of hand-offs).
struct HandWarp {
  HandWords hw;
  bool mine, live;       // live: false once a wait has run out (no more waiting)
  const double* base;    // this warp's right-hand side
  __device__ __forceinline__ HandWarp(const double* slab, int n, int q0, int nq) {
    const int q = threadIdx.x >> 5;
    mine = live = q < nq;
    base = slab + (int64_t)(q0 + (mine ? q : 0)) * n;
  }
  __device__ __forceinline__ void load(int j, int kb) {
    if (mine) hw.load(base + j * FB, kb);
  }
  template <typename CT, int NQ>
  __device__ __forceinline__ void take(int j, int kb, int* err, int where, CT (&dst)[NQ][FB]) {
    if (!mine) return;
    if (live) live = hw.wait(base + j * FB, kb, err, where);
    hw.stage(dst[threadIdx.x >> 5]);
  }
};

// acc[q] += sum over the column blocks j < jend of L[row, block j] y_j for
// the CTA's rows (thread: row lane tid % 64, column group tid / 64), y_j read
// from its hand-off words (HandWarp), the other warps waiting at the block barrier.
template <typename T, int NQ>
__device__ __forceinline__ void fwd_gather_blocks(const DevCtx& c, const FrontDev& f, int row, bool rv, int jend,
                                                  int q0, int nq, int* err, T (&acc)[NQ], T (*ysh)[NQ][FB]) {
  using CT = T;
  const int n = f.n, fs = f.fs, g = threadIdx.x / FB;
  const T* __restrict__ G = arena<T>(c) + f.off;
  const double* __restrict__ y = c.vec + f.voff + (int64_t)n * c.n_rhs;
  // The factor tile of block column j does not depend on y: it is loaded one
  // block ahead, so that only the loads of y_j follow the wait.
  CT tile[16];
  auto load_tile = [&](int j) {
    const int kbj = min(FB, fs - j * FB);
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int cc = g * 16 + u;
      tile[u] = (rv && cc < kbj) ? (CT)G[row + (int64_t)(j * FB + cc) * n] : CT(0);
    }
  };
  HandWarp hand(y, n, q0, nq);
  if (jend > 0) {
    load_tile(0);
    hand.load(0, min(FB, fs));
  }
  for (int j = 0; j < jend; ++j) {
    const int buf = j & 1;
    // y_j is read by every later block of the front at once: one warp per CTA
    // and right-hand side polls and stages it (the next block's words already in flight)
    hand.take(j, min(FB, fs - j * FB), err, wait_code(1, j, row / FB), ysh[buf]);
    if (j + 1 < jend) hand.load(j + 1, min(FB, fs - (j + 1) * FB));
    CT cur[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) cur[u] = tile[u];
    if (j + 1 < jend) load_tile(j + 1);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 16; ++u) {
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        if (q < nq) acc[q] += cur[u] * ysh[buf][q][g * 16 + u];
    }
  }
}

// item: front, a = block index (factor blocks 0..nfb-1, ABL blocks nfb..);
// a CTA per group of NQ right-hand sides (flags_nq), so that a launch for one
// right-hand side issues no products for absent ones
template <typename T, int NQ>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 2) k_fwd_flags(DevCtx c, const Item* __restrict__ items,
                                                   int* ticket, int* err, int ng) {
  using CT = T;
  __shared__ int s_t;
  __shared__ CT red[4][FB][NQ];
  __shared__ CT v[FB][NQ];
  __shared__ T dsh[FB * (FB + 1)];     // inverse diagonal block, staged before any wait
  // y_j staged by warp 0, two buffers alternating by block: one barrier per block
  __shared__ CT ysh[2][NQ][FB];
  if (threadIdx.x == 0) s_t = atomicAdd(ticket, 1);
  __syncthreads();
  const Item it = items[s_t / ng];
  const int q0 = (s_t % ng) * NQ;
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, fs = f.fs, nr = c.n_rhs, b = it.a;
  const int nq = min(NQ, nr - q0);
  const int nfb = (fs + FB - 1) / FB;
  const bool factor_block = b < nfb;
  if (factor_block) {
    const T* __restrict__ Dg = dinv_arena<T>(c) + f.dinv_off + (int64_t)b * FB * FB;
    for (int idx = threadIdx.x; idx < FB * FB; idx += 256) dsh[(idx / FB) * (FB + 1) + idx % FB] = Dg[idx];
  }
  const int r0 = factor_block ? b * FB : fs + (b - nfb) * FB;
  const int r1 = factor_block ? min(r0 + FB, fs) : min(r0 + FB, n);
  double* __restrict__ z = c.vec + f.voff;
  double* __restrict__ y = z + (int64_t)n * nr;
  const int i = threadIdx.x % FB, g = threadIdx.x / FB;
  const int row = r0 + i;
  const bool rv = row < r1;
  CT acc[NQ], zr[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    acc[q] = CT(0);
    zr[q] = (rv && q < nq && g == 0) ? (CT)z[row + (int64_t)(q0 + q) * n] : CT(0);   // before any wait
  }
  // the factor rows of z are not read again: they become the backward
  // solve's hand-off words for this block
  if (factor_block && rv && g == 0) {
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      if (q < nq) z[row + (int64_t)(q0 + q) * n] = __longlong_as_double((long long)HAND_EMPTY);
  }
  fwd_gather_blocks<T, NQ>(c, f, row, rv, factor_block ? b : nfb, q0, nq, err, acc, ysh);
#pragma unroll
  for (int q = 0; q < NQ; ++q) red[g][i][q] = acc[q];
  __syncthreads();
  if (threadIdx.x < FB) {
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      v[i][q] = (rv && q < nq) ? zr[q] - (red[0][i][q] + red[1][i][q] + red[2][i][q] + red[3][i][q]) : CT(0);
  }
  __syncthreads();
  if (factor_block) {
    // y = Dinv v on all 256 threads: column group g sums t in [16 g, 16 g + 16),
    // then the four partial sums are added in group order; this takes the
    // 64-step dependent chain of one thread per row off the hand-off to the
    // next block.  The stored inverse is zero above its diagonal and past the
    // block's kb rows and columns, so every thread runs the same unbranched
    // loop (its loads issued together) and the sums equal the skipped-term
    // ones exactly.
    CT xp[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) xp[q] = CT(0);
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int t = g * 16 + u;
      const CT d = (CT)dsh[t * (FB + 1) + i];     // Dinv[i][t], column t staged as row t
#pragma unroll
      for (int q = 0; q < NQ; ++q) xp[q] += d * v[t][q];
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) red[g][i][q] = xp[q];
    __syncthreads();
    if (threadIdx.x < FB && rv) {
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        if (q < nq)
          st_hand(y + row + (int64_t)(q0 + q) * n,
                  (double)(red[0][i][q] + red[1][i][q] + red[2][i][q] + red[3][i][q]));
    }
  } else if (threadIdx.x < FB && rv) {
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      if (q < nq) z[row + (int64_t)(q0 + q) * n] = (double)v[i][q];
  }
}

// Forward solve of large Cholesky fronts with 256-row CTAs.  Item: front,
// a = B: B < nfb4 (= ceil(nfb / 4)) the factor rows 256 B .. (64-row blocks
// 4 B .. 4 B + 3, solved here in turn), otherwise the ABL rows
// fs + 256 (B - nfb4) ...  One thread per row; the row's 64 factor entries of
// the next column block are loaded into registers before that block's
// solution is waited for.  Column blocks left of the CTA come from other
// CTAs as hand-off words (warp 0 polls and stages them, the next block's
// words already in flight); the CTA's own blocks are solved in turn on all
// its threads (v = z - sum on the block's rows, y = Dinv v by four column
// groups, summed in group order), each published at once as hand-off words,
// and every later row of the CTA adds its product with y.  One hand-off
// between CTAs per 256 rows instead of per 64.  Tickets in item order: every
// CTA waits only on smaller tickets.
constexpr int F4_ROWS = 256;

template <typename T>
__global__ void __launch_bounds__(256, 1) k_fwd_hand4(DevCtx c, const Item* __restrict__ items, int* ticket, int* err,
                                                      int q0) {
  using CT = T;
  extern __shared__ __align__(16) unsigned char f4_dyn[];
  T* dsh = reinterpret_cast<T*>(f4_dyn);          // own inverse diagonal blocks, dsh[s][t * 65 + i] = Dinv_s[i][t]
  __shared__ int s_t;
  __shared__ CT ysh[2][SF_NR][FB];
  __shared__ CT vsh[SF_NR][FB];
  __shared__ CT red[4][FB][SF_NR];
  const int tid = threadIdx.x;
  if (tid == 0) s_t = atomicAdd(ticket, 1);
  __syncthreads();
  const Item it = items[s_t];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, fs = f.fs, nr = c.n_rhs;
  const int nq = min(SF_NR, nr - q0);
  const int nfb = (fs + FB - 1) / FB, nfb4 = (nfb + 3) / 4;
  const bool factor_cta = it.a < nfb4;
  const int b0 = factor_cta ? 4 * it.a : nfb;                 // first own 64-row block (factor CTAs)
  const int ns = factor_cta ? min(4, nfb - b0) : 0;           // own blocks
  const int r0 = factor_cta ? F4_ROWS * it.a : fs + F4_ROWS * (it.a - nfb4);
  const int r1 = factor_cta ? min(r0 + F4_ROWS, fs) : min(r0 + F4_ROWS, n);
  const int row = r0 + tid;
  const bool rv = row < r1;
  const int sub = tid >> 6;                                   // own block of this row (factor CTAs)
  const T* __restrict__ G = arena<T>(c) + f.off;
  double* __restrict__ z = c.vec + f.voff;
  double* __restrict__ y = z + (int64_t)n * nr;
  if (factor_cta) {
    const T* __restrict__ Dg = dinv_arena<T>(c) + f.dinv_off + (int64_t)b0 * FB * FB;
    for (int idx = tid; idx < ns * FB * FB; idx += 256) {
      const int s2 = idx / (FB * FB), e = idx % (FB * FB);
      dsh[s2 * FB * (FB + 1) + (e / FB) * (FB + 1) + e % FB] = Dg[idx];
    }
  }
  CT acc[SF_NR], zr[SF_NR];
#pragma unroll
  for (int q = 0; q < SF_NR; ++q) {
    acc[q] = CT(0);
    zr[q] = (rv && q < nq) ? (CT)z[row + (int64_t)(q0 + q) * n] : CT(0);
  }
  // the factor rows of z are not read again: they become the backward
  // solve's hand-off words
  if (factor_cta && rv) {
#pragma unroll
    for (int q = 0; q < SF_NR; ++q)
      if (q < nq) z[row + (int64_t)(q0 + q) * n] = __longlong_as_double((long long)HAND_EMPTY);
  }
  const int jext = b0;                    // column blocks solved by other CTAs
  // the row's entries of column block j, where this row needs them
  CT tile[FB];
  auto load_tile = [&](int j) {
    const bool need = rv && (j < jext || sub > j - b0);
    const int kbj = min(FB, fs - j * FB);
#pragma unroll
    for (int u = 0; u < FB; ++u) tile[u] = (need && u < kbj) ? (CT)G[row + (int64_t)(j * FB + u) * n] : CT(0);
  };
  const int jlast = factor_cta ? b0 + ns - 1 : nfb;          // tiles needed: blocks 0 .. jlast - 1
  if (jlast > 0) load_tile(0);
  const bool w0 = tid < 32;
  HandWords hw;
  bool live = true;      // warp 0: false once a wait has run out (no more waiting)
  if (jext > 0 && w0) hw.load(y + (int64_t)q0 * n, min(FB, fs));
  for (int j = 0; j < jext; ++j) {
    const int buf = j & 1;
    if (w0) {
      const int kbj = min(FB, fs - j * FB);
      const double* yj = y + j * FB;
      if (live) live = hw.wait(yj + (int64_t)q0 * n, kbj, err, wait_code(1, j, b0));
      hw.stage(ysh[buf][0]);
      for (int q = 1; q < nq; ++q) {
        HandWords hq;
        hq.load(yj + (int64_t)(q0 + q) * n, kbj);
        if (live) live = hq.wait(yj + (int64_t)(q0 + q) * n, kbj, err, wait_code(1, j, b0));
        hq.stage(ysh[buf][q]);
      }
      if (j + 1 < jext) hw.load(y + (j + 1) * FB + (int64_t)q0 * n, min(FB, fs - (j + 1) * FB));
    }
    __syncthreads();
    if constexpr (sizeof(T) == 4) {
      // FP32: the next block's loads are issued before this block's products
      CT cur[FB];
#pragma unroll
      for (int u = 0; u < FB; ++u) cur[u] = tile[u];
      if (j + 1 < jlast) load_tile(j + 1);
      if (rv) {
#pragma unroll
        for (int u = 0; u < FB; ++u)
#pragma unroll
          for (int q = 0; q < SF_NR; ++q) acc[q] += cur[u] * ysh[buf][q][u];
      }
    } else {
      // FP64 (register budget): products first, then the next block's loads
      if (rv) {
#pragma unroll
        for (int u = 0; u < FB; ++u)
#pragma unroll
          for (int q = 0; q < SF_NR; ++q) acc[q] += tile[u] * ysh[buf][q][u];
      }
      if (j + 1 < jlast) load_tile(j + 1);
    }
  }
  // own blocks s: v = z - acc on its rows, y = Dinv_s v, published; the rows
  // below add their products with y
  for (int s = 0; s < ns; ++s) {
    const int j = b0 + s, kbj = min(FB, fs - j * FB);
    if (sub == s) {
#pragma unroll
      for (int q = 0; q < SF_NR; ++q) vsh[q][tid & 63] = rv ? zr[q] - acc[q] : CT(0);
    }
    // FP32: the next block's tile is loaded before this block's solve (the
    // rows below need it right after); FP64 (register budget) loads it after
    // the products
    CT cur[sizeof(T) == 4 ? FB : 1];
    if constexpr (sizeof(T) == 4) {
#pragma unroll
      for (int u = 0; u < FB; ++u) cur[u] = tile[u];
      if (j + 1 < jlast) load_tile(j + 1);
    }
    __syncthreads();
    {
      // y = Dinv v: column group g sums t in [16 g, 16 g + 16) (Dinv is
      // lower triangular: t <= i)
      const int i = tid & 63, g = tid >> 6;
      const T* Ds = dsh + s * FB * (FB + 1);
      CT xp[SF_NR];
#pragma unroll
      for (int q = 0; q < SF_NR; ++q) xp[q] = CT(0);
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int t = g * 16 + u;
        if (t <= i && t < kbj) {
          const CT d = (CT)Ds[t * (FB + 1) + i];
#pragma unroll
          for (int q = 0; q < SF_NR; ++q) xp[q] += d * vsh[q][t];
        }
      }
#pragma unroll
      for (int q = 0; q < SF_NR; ++q) red[g][i][q] = xp[q];
    }
    __syncthreads();
    if (tid < FB) {
      const int i = tid, r = r0 + FB * s + i;
#pragma unroll
      for (int q = 0; q < SF_NR; ++q) {
        const CT yv = red[0][i][q] + red[1][i][q] + red[2][i][q] + red[3][i][q];
        ysh[0][q][i] = i < kbj ? yv : CT(0);
        if (i < kbj && q < nq) st_hand(y + r + (int64_t)(q0 + q) * n, (double)yv);
      }
    }
    __syncthreads();
    if constexpr (sizeof(T) == 4) {
      if (rv && sub > s) {
#pragma unroll
        for (int u = 0; u < FB; ++u)
#pragma unroll
          for (int q = 0; q < SF_NR; ++q) acc[q] += cur[u] * ysh[0][q][u];
      }
    } else {
      (void)cur;
      if (rv && sub > s) {
#pragma unroll
        for (int u = 0; u < FB; ++u)
#pragma unroll
          for (int q = 0; q < SF_NR; ++q) acc[q] += tile[u] * ysh[0][q][u];
      }
      if (j + 1 < jlast) load_tile(j + 1);
    }
  }
  if (!factor_cta && rv) {
#pragma unroll
    for (int q = 0; q < SF_NR; ++q)
      if (q < nq) z[row + (int64_t)(q0 + q) * n] = (double)(zr[q] - acc[q]);
  }
}

void launch_fwd_flags4(const DevCtx& c, const Item* items, int n_items, int dtype, int* ticket, int* err, int q0,
                       cudaStream_t s) {
  if (!n_items) return;
  cudaMemsetAsync(ticket, 0, sizeof(int), s);
  if (dtype == F64) {
    const int sm = (int)(sizeof(double) * 4 * FB * (FB + 1));
    cudaFuncSetAttribute(k_fwd_hand4<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    k_fwd_hand4<double><<<n_items, 256, sm, s>>>(c, items, ticket, err, q0);
  } else {
    const int sm = (int)(sizeof(float) * 4 * FB * (FB + 1));
    cudaFuncSetAttribute(k_fwd_hand4<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    k_fwd_hand4<float><<<n_items, 256, sm, s>>>(c, items, ticket, err, q0);
  }
}

// Backward: item: front, a = factor block index, tickets in descending block
// order, a CTA per group of NQ right-hand sides.  The 64-row blocks below the
// factor block, the ABL rows (x known from the parent) first, then the factor
// blocks from the last one up as their hand-off words arrive, pass through two
// shared-memory tiles: loaded by rows (a warp's loads are consecutive rows of a
// column), a block ahead in registers, and read by columns, so that a thread
// sums a quarter of one column per right-hand side in NQ registers.  (With 16 NQ
// sums per thread, one row each, only one CTA fitted an SM, and adding the 64 rows
// up was on the chain of hand-offs.)
template <typename T, int NQ>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 2) k_bwd_flags(DevCtx c, const Item* __restrict__ items,
                                                   int* ticket, int* err, int ng) {
  using CT = T;
  extern __shared__ __align__(16) unsigned char bwd_dyn[];
  CT (*ts)[FB][FB + 1] = reinterpret_cast<CT (*)[FB][FB + 1]>(bwd_dyn);      // two tiles [row][column]
  CT* dsh = reinterpret_cast<CT*>(bwd_dyn) + 2 * FB * (FB + 1);             // inverse diagonal block
  __shared__ int s_t;
  __shared__ CT red[4][FB][NQ];
  __shared__ CT v[FB][NQ];
  __shared__ CT xsh[2][NQ][FB];
  if (threadIdx.x == 0) s_t = atomicAdd(ticket, 1);
  __syncthreads();
  const Item it = items[s_t / ng];
  const int q0 = (s_t % ng) * NQ;
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, fs = f.fs, nr = c.n_rhs, b = it.a;
  const int nq = min(NQ, nr - q0), nfb = (fs + FB - 1) / FB;
  const int c0 = b * FB, kb = min(FB, fs - c0);
  const T* __restrict__ G = arena<T>(c) + f.off;
  {
    const T* __restrict__ Dg = dinv_arena<T>(c) + f.dinv_off + (int64_t)b * FB * FB;
    for (int idx = threadIdx.x; idx < FB * FB; idx += 256) dsh[(idx / FB) * (FB + 1) + idx % FB] = Dg[idx];
  }
  double* __restrict__ hx = c.vec + f.voff;                  // hand-off: the z slab's factor rows
  double* __restrict__ y = hx + (int64_t)n * nr;
  // thread: column i (row i of a tile when loading), quarter g
  const int i = threadIdx.x % FB, g = threadIdx.x / FB;
  CT acc[NQ], yb[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    acc[q] = CT(0);
    // this block's right-hand sides, loaded before any wait
    yb[q] = (threadIdx.x < kb && q < nq) ? (CT)y[c0 + threadIdx.x + (int64_t)(q0 + q) * n] : CT(0);
  }
  // FP64: the ABL rows without the tiles, a row per thread and 16 columns, the
  // rows added up before any wait (the tiles' barriers and 64-bit accesses cost the
  // levels that are bound by the FP64 products a quarter of their time)
  constexpr bool ROWS = sizeof(T) == 8 && NQ == 1;
  if constexpr (ROWS) {
    if (fs < n) {
      CT ar[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) ar[u] = CT(0);
      for (int rs = fs; rs < n; rs += 2 * FB) {
        CT xr[2], gv[2][16];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = rs + h * FB + i;
          xr[h] = r < n ? (CT)y[r + (int64_t)q0 * n] : CT(0);
#pragma unroll
          for (int u = 0; u < 16; ++u) {
            const int cc = g * 16 + u;
            gv[h][u] = (r < n && cc < kb) ? (CT)G[r + (int64_t)(c0 + cc) * n] : CT(0);
          }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int u = 0; u < 16; ++u) ar[u] += gv[h][u] * xr[h];
      }
#pragma unroll
      for (int u = 0; u < 16; ++u) ts[1][i][g * 16 + u] = ar[u];
      __syncthreads();
#pragma unroll
      for (int r = 0; r < 16; ++r) acc[0] += ts[1][g * 16 + r][i];
    }
  }
  const int na = ROWS ? 0 : (n - fs + FB - 1) / FB, nblk = na + nfb - 1 - b;
  auto first_row = [&](int k) { return k < na ? fs + k * FB : (nfb - 1 - (k - na)) * FB; };
  auto rows_of = [&](int k) { return min(FB, (k < na ? n : fs) - first_row(k)); };
  CT tile[16];
  auto load_tile = [&](int k) {
    const int r = first_row(k) + i;
    const bool in = i < rows_of(k);
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int cc = g * 16 + u;
      tile[u] = (in && cc < kb) ? (CT)G[r + (int64_t)(c0 + cc) * n] : CT(0);
    }
  };
  HandWarp hand(hx, n, q0, nq);
  const double* const ya = y + (int64_t)(q0 + (hand.mine ? threadIdx.x >> 5 : 0)) * n;
  const int lane = threadIdx.x & 31;
  auto load_x = [&](int k) {
    if (!hand.mine) return;
    const int r = first_row(k), m = rows_of(k);
    if (k < na) {
      hand.hw.w0 = lane < m ? (unsigned long long)__double_as_longlong(ya[r + lane]) : 0ull;
      hand.hw.w1 = lane + 32 < m ? (unsigned long long)__double_as_longlong(ya[r + lane + 32]) : 0ull;
    } else {
      hand.hw.load(hand.base + r, m);
    }
  };
  if (nblk > 0) {
    load_tile(0);
    load_x(0);
  }
  for (int k = 0; k < nblk; ++k) {
    const int buf = k & 1;
#pragma unroll
    for (int u = 0; u < 16; ++u) ts[buf][i][g * 16 + u] = tile[u];
    if (k + 1 < nblk) load_tile(k + 1);
    if (hand.mine) {
      const int r = first_row(k);
      if (k >= na && hand.live) hand.live = hand.hw.wait(hand.base + r, rows_of(k), err, wait_code(2, r / FB, b));
      hand.hw.stage(xsh[buf][threadIdx.x >> 5]);
    }
    if (k + 1 < nblk) load_x(k + 1);
    __syncthreads();
    // (a tile's sum by itself: n / 64 + 16 roundings in a row instead of n / 4)
    CT p[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) p[q] = CT(0);
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const CT t = ts[buf][g * 16 + u][i];
#pragma unroll
      for (int q = 0; q < NQ; ++q) p[q] += t * xsh[buf][q][g * 16 + u];
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) acc[q] += p[q];
  }
#pragma unroll
  for (int q = 0; q < NQ; ++q) red[g][i][q] = acc[q];
  __syncthreads();
  if (threadIdx.x < FB) {
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      v[i][q] = (i < kb && q < nq) ? yb[q] - (red[0][i][q] + red[1][i][q] + red[2][i][q] + red[3][i][q]) : CT(0);
  }
  __syncthreads();
  // x = Dinv^T v : x_i = sum_{t >= i} Dinv[t, i] v_t   (column i of Dinv, staged at start),
  // on all 256 threads: group g sums t in [16 g, 16 g + 16), partial sums
  // added in group order; Dinv[t][i] is zero for t < i and past kb: the
  // unbranched sum is exact
  CT xp[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) xp[q] = CT(0);
#pragma unroll
  for (int u = 0; u < 16; ++u) {
    const CT d = dsh[i * (FB + 1) + g * 16 + u];
#pragma unroll
    for (int q = 0; q < NQ; ++q) xp[q] += d * v[g * 16 + u][q];
  }
#pragma unroll
  for (int q = 0; q < NQ; ++q) red[g][i][q] = xp[q];
  __syncthreads();
  if (threadIdx.x < kb) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      if (q >= nq) break;
      const double x = (double)(red[0][i][q] + red[1][i][q] + red[2][i][q] + red[3][i][q]);
      y[c0 + i + (int64_t)(q0 + q) * n] = x;
      st_hand(hx + c0 + i + (int64_t)(q0 + q) * n, x);
    }
  }
}

// Right-hand sides per CTA; the other groups run beside it (consecutive
// tickets: their reads of a tile of the factor meet in L2).  FP64: one, since its
// products, 64 x 64 per block and right-hand side at about 1.1 us each, are
// on the chain of hand-offs twice per block.  FP32: up to four (with eight the
// levels of large fronts took 543 instead of 351 us forward and 316 instead of 195
// backward, those of many fronts 120 to 300 instead of 160 to 340).
// Measured on GB300, a launch per group before, forward and backward: 12^3 p = 4
// FP64, 4 right-hand sides, root 12,698 rows: 2.69 + 3.86 -> 1.30 + 1.42 ms; FP32, 16
// right-hand sides, 11,427 fronts up to 6,938 rows, two solves: 6.8 + 10.3 -> 2.1 +
// 2.4; one right-hand side, 16^3 p = 4 FP64: 1.15 + 1.52 -> 1.15 + 1.35.
template <typename T> static int flags_nq(int nr) { return sizeof(T) == 8 || nr == 1 ? 1 : nr == 2 ? 2 : 4; }

template <typename T>
static void fwd_flags_t(const DevCtx& c, const Item* items, int n_items, int* ticket, int* err, cudaStream_t s) {
  const int nq = flags_nq<T>(c.n_rhs), ng = (c.n_rhs + nq - 1) / nq;
  if (nq == 1) k_fwd_flags<T, 1><<<n_items * ng, 256, 0, s>>>(c, items, ticket, err, ng);
  else if constexpr (sizeof(T) == 4) {
    if (nq == 2) k_fwd_flags<T, 2><<<n_items * ng, 256, 0, s>>>(c, items, ticket, err, ng);
    else k_fwd_flags<T, 4><<<n_items * ng, 256, 0, s>>>(c, items, ticket, err, ng);
  }
}

void launch_fwd_flags(const DevCtx& c, const Item* items, int n_items, int dtype, int* ticket, int* err,
                      cudaStream_t s) {
  if (!n_items) return;
  cudaMemsetAsync(ticket, 0, sizeof(int), s);
  if (dtype == F64) fwd_flags_t<double>(c, items, n_items, ticket, err, s);
  else fwd_flags_t<float>(c, items, n_items, ticket, err, s);
}

template <typename T, int NQ>
static void bwd_flags_nq(const DevCtx& c, const Item* items, int n_items, int* ticket, int* err, int ng,
                         cudaStream_t s) {
  const size_t dyn = 3 * sizeof(T) * FB * (FB + 1);
  cudaFuncSetAttribute(k_bwd_flags<T, NQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
  k_bwd_flags<T, NQ><<<n_items * ng, 256, dyn, s>>>(c, items, ticket, err, ng);
}

template <typename T>
static void bwd_flags_t(const DevCtx& c, const Item* items, int n_items, int* ticket, int* err, cudaStream_t s) {
  const int nq = flags_nq<T>(c.n_rhs), ng = (c.n_rhs + nq - 1) / nq;
  if (nq == 1) bwd_flags_nq<T, 1>(c, items, n_items, ticket, err, ng, s);
  else if constexpr (sizeof(T) == 4) {
    if (nq == 2) bwd_flags_nq<T, 2>(c, items, n_items, ticket, err, ng, s);
    else bwd_flags_nq<T, 4>(c, items, n_items, ticket, err, ng, s);
  }
}

void launch_bwd_flags(const DevCtx& c, const Item* items, int n_items, int dtype, int* ticket, int* err,
                      cudaStream_t s) {
  if (!n_items) return;
  cudaMemsetAsync(ticket, 0, sizeof(int), s);
  if (dtype == F64) bwd_flags_t<double>(c, items, n_items, ticket, err, s);
  else bwd_flags_t<float>(c, items, n_items, ticket, err, s);
}

// ===========================================================================
// Backward flag-driven solve of large LU fronts: x_b = U_bb^{-1} (y_b - sum_{c
// right of block b} U_bc x_c), the forward kernel's row blocks from the last
// one up.  Item: front, a = factor block, tickets in descending block order.
// The columns right of the factor block (x known from the parent) come
// first, then the factor blocks as their hand-off words arrive.  U_bb^{-1}
// is formed at factorisation (k_lu_dinv).  Bound by the chain of hand-offs
// as the Cholesky solves are; measured on GB300 (24^3 p = 3, root 14,911
// rows, FP32): 1.9 ms for the two backward solves of a step against 44
// for a launch per 64 columns with the block substituted by one warp.
// ===========================================================================
template <typename T, int NQ>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 2) k_lu_bwd_flags(DevCtx c, const Item* __restrict__ items,
                                                                              int* ticket, int* err, int ng) {
  __shared__ int s_t;
  __shared__ T red[4][FB][NQ];
  __shared__ T v[FB][NQ];
  __shared__ T dsh[FB * (FB + 1)];
  __shared__ T xsh[2][NQ][FB];
  if (threadIdx.x == 0) s_t = atomicAdd(ticket, 1);
  __syncthreads();
  const Item it = items[s_t / ng];
  const int q0 = (s_t % ng) * NQ;
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, fs = f.fs, nr = c.n_rhs, b = it.a;
  const int nq = min(NQ, nr - q0), nfb = (fs + FB - 1) / FB;
  const T* __restrict__ G = arena<T>(c) + f.off;
  {
    const T* __restrict__ Dg = dinv_arena<T>(c) + f.dinv_off + (int64_t)(nfb + b) * FB * FB;
    for (int idx = threadIdx.x; idx < FB * FB; idx += 256) dsh[(idx / FB) * (FB + 1) + idx % FB] = Dg[idx];
  }
  double* __restrict__ hx = c.vec + f.voff;                  // hand-off: the z slab's factor rows
  double* __restrict__ y = hx + (int64_t)n * nr;
  const int i = threadIdx.x % FB, g = threadIdx.x / FB;
  const int row = b * FB + i;
  const bool rv = row < fs;
  T acc[NQ], yb[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    acc[q] = T(0);
    yb[q] = (rv && q < nq && g == 0) ? (T)y[row + (int64_t)(q0 + q) * n] : T(0);   // before any wait
  }
  // columns fs .. n-1: group g takes 16 of every 64, all loads of a round in flight
  for (int cs = fs; cs < n; cs += FB) {
    T gv[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int cc = cs + g * 16 + u;
      gv[u] = rv && cc < n ? G[row + (int64_t)cc * n] : T(0);
    }
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int cc = min(cs + g * 16 + u, n - 1);
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        if (q < nq) acc[q] += gv[u] * (T)y[cc + (int64_t)(q0 + q) * n];
    }
  }
  T tile[16];
  auto load_tile = [&](int j) {
    const int kbj = min(FB, fs - j * FB);
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int cc = g * 16 + u;
      tile[u] = (rv && cc < kbj) ? G[row + (int64_t)(j * FB + cc) * n] : T(0);
    }
  };
  HandWarp hand(hx, n, q0, nq);
  if (nfb - 1 > b) {
    load_tile(nfb - 1);
    hand.load(nfb - 1, min(FB, fs - (nfb - 1) * FB));
  }
  for (int j = nfb - 1; j > b; --j) {
    const int buf = j & 1;
    hand.take(j, min(FB, fs - j * FB), err, wait_code(2, j, b), xsh[buf]);
    if (j - 1 > b) hand.load(j - 1, min(FB, fs - (j - 1) * FB));
    T cur[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) cur[u] = tile[u];
    if (j - 1 > b) load_tile(j - 1);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 16; ++u)
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        if (q < nq) acc[q] += cur[u] * xsh[buf][q][g * 16 + u];
  }
#pragma unroll
  for (int q = 0; q < NQ; ++q) red[g][i][q] = acc[q];
  __syncthreads();
  if (threadIdx.x < FB) {
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      v[i][q] = (rv && q < nq) ? yb[q] - (red[0][i][q] + red[1][i][q] + red[2][i][q] + red[3][i][q]) : T(0);
  }
  __syncthreads();
  // x = Uinv v by four column groups (zero below its diagonal and past the block)
  T xp[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) xp[q] = T(0);
#pragma unroll
  for (int u = 0; u < 16; ++u) {
    const int t = g * 16 + u;
    const T d = dsh[t * (FB + 1) + i];     // Uinv[i][t], column t staged as row t
#pragma unroll
    for (int q = 0; q < NQ; ++q) xp[q] += d * v[t][q];
  }
#pragma unroll
  for (int q = 0; q < NQ; ++q) red[g][i][q] = xp[q];
  __syncthreads();
  if (threadIdx.x < FB && rv) {
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      if (q < nq) {
        const double x = (double)(red[0][i][q] + red[1][i][q] + red[2][i][q] + red[3][i][q]);
        y[row + (int64_t)(q0 + q) * n] = x;
        st_hand(hx + row + (int64_t)(q0 + q) * n, x);
      }
  }
}

template <typename T>
static void lu_bwd_flags_t(const DevCtx& c, const Item* items, int n_items, int* ticket, int* err, cudaStream_t s) {
  const int nq = flags_nq<T>(c.n_rhs), ng = (c.n_rhs + nq - 1) / nq;
  if (nq == 1) k_lu_bwd_flags<T, 1><<<n_items * ng, 256, 0, s>>>(c, items, ticket, err, ng);
  else if constexpr (sizeof(T) == 4) {
    if (nq == 2) k_lu_bwd_flags<T, 2><<<n_items * ng, 256, 0, s>>>(c, items, ticket, err, ng);
    else k_lu_bwd_flags<T, 4><<<n_items * ng, 256, 0, s>>>(c, items, ticket, err, ng);
  }
}

void launch_lu_bwd_flags(const DevCtx& c, const Item* items, int n_items, int dtype, int* ticket, int* err,
                         cudaStream_t s) {
  if (!n_items) return;
  cudaMemsetAsync(ticket, 0, sizeof(int), s);
  if (dtype == F64) lu_bwd_flags_t<double>(c, items, n_items, ticket, err, s);
  else lu_bwd_flags_t<float>(c, items, n_items, ticket, err, s);
}

// ===========================================================================
// Chain solves of large FP32 Cholesky fronts.
//
// In the flag-driven solves every 64-row block waits for its neighbour's
// solution to cross from one SM to another (a store, the reader's poll, its
// load): that latency is paid once per block along the whole diagonal.  Here
// one CTA per front (the chain) solves all diagonal blocks in turn from its
// own shared memory, and other CTAs (helpers) feed it:
//
//   forward   x_b = Dinv_b (z_b - P_b - sum_{j = b-K}^{b-1} L_bj x_j)
//             P_b = sum_{j < b-K} L_bj x_j            (helper of row block b)
//   backward  x_b = Dinv_b^T (y_b - P_b - sum_{r = b+1}^{b+K} L_rb^T x_r)
//             P_b = sum_{r > b+K} L_rb^T x_r + (ABL rows) (helper of column block b)
//
// The chain applies the K = CH_K blocks next to the diagonal itself, so a
// helper's partial sum for block b needs solutions at least K + 1 blocks
// back: it has K chain steps to arrive.  Solutions and partial sums travel
// as hand-off words (HAND_EMPTY until written): x in y's factor rows
// (forward) and z's (backward), P in the third slab w.  The chain stages its
// window of blocks and the diagonal inverse with cp.async, CH_STAGES - 1
// steps ahead (asking L2 for them CH_L2_AHEAD steps ahead), and loads each
// step's right-hand side and partial sum a step ahead; the helpers stream their blocks through shared memory CH_HS - 1
// ahead.  Rows of ABL (forward) are finished by their own CTAs once every
// x_j is out.
//
// Items: front, a = block, b = role.  Tickets: the chains first, then the
// helpers in the order their sums are needed, then the ABL rows.  A chain
// waits on helpers with larger tickets, but a helper needs only chain steps
// that in turn need only helpers with smaller tickets: as long as the
// chains and one more CTA fit on the GPU together (at most CH_MAX_CHAINS
// chains per launch, one CTA per SM), the lowest unfinished helper can
// always run and finish, and every wait ends.
// ===========================================================================
constexpr int CH_STAGES = 3;
constexpr int CH_LD = 68;           // floats per staged block column: 64 + room for the 16-byte alignment shift
constexpr int CH_TILE = 64 * CH_LD;
constexpr int CH_HS = 8;            // shared-memory stages of a helper's blocks
constexpr int CH_HW = 4;            // blocks of hand-off words warp 0 of a helper keeps in flight
constexpr int CH_L2_AHEAD = 12;     // steps ahead whose blocks the chain asks L2 for

struct ChainSmem {
  float L[CH_STAGES][CH_K + 1][CH_TILE];   // per stage: the window's blocks, the diagonal inverse (slot CH_K)
  float xs[CH_K][SF_NR][FB];               // the window's solutions (block j at j % CH_K)
  float ts[SF_NR][FB];
};
struct ChainRowSmem {
  float L[CH_HS][CH_TILE];
  float vsh[2][SF_NR][FB];          // the staged solution values of the current block
  float red[4][FB][SF_NR];
  float redb[FB][FB + 1];
};
constexpr size_t CH_SMEM = sizeof(ChainSmem) > sizeof(ChainRowSmem) ? sizeof(ChainSmem) : sizeof(ChainRowSmem);

__device__ __forceinline__ void ch_cp16(float* dst, const float* src) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(src) : "memory");
}
__device__ __forceinline__ void ch_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void ch_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void ch_l2(const float* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// The 64 x 64 block of the panel G (ld n) at rows r0.., columns c0.. (c0 a
// multiple of 64), its first ncols columns staged as columns of CH_LD
// floats: column cc starts at the 16-byte boundary at or before entry
// (r0, c0 + cc), so entry (i, cc) is at dst[cc * CH_LD + ch_sh(r0, cc, n) + i].
// Two columns per warp and pass, 17 chunks of 16 bytes each.  Callers stage
// only columns left of column n - 1 with r0 < n, n > 66: the up to 3 extra
// entries either side lie in the neighbouring columns of the same panel.
__device__ __forceinline__ void ch_stage_block(float* dst, const float* G, int64_t r0, int64_t c0, int64_t n,
                                               int ncols = 64) {
  const int lane = threadIdx.x & 31, p = lane & 15;
  for (int k = threadIdx.x >> 5; 2 * k < ncols; k += blockDim.x >> 5) {
    const int cc = 2 * k + (lane >> 4);
    if (cc < ncols) {
      const int64_t s0 = r0 + (c0 + cc) * n;
      const float* src = G + (s0 & ~(int64_t)3);
      float* d = dst + cc * CH_LD;
      ch_cp16(d + 4 * p, src + 4 * p);
      if (p == 0) ch_cp16(d + 64, src + 64);
    }
  }
}
// the alignment shift of staged column cc (c0 a multiple of 4)
__device__ __forceinline__ int ch_sh(int64_t r0, int cc, int64_t n) {
  return (int)(((r0 & 3) + (int64_t)(cc & 3) * (n & 3)) & 3);
}
// the lower triangle of the 64 x 64 diagonal inverse (column-major, 16-byte
// aligned): entry (i, t), i >= t, at dst[t * CH_LD + i]; the 16-byte chunks
// wholly above the diagonal are not copied
__device__ __forceinline__ void ch_stage_dinv(float* dst, const float* D) {
  for (int e = threadIdx.x; e < 64 * 16; e += blockDim.x) {
    const int t = e >> 4, p = e & 15;
    if (4 * p + 3 >= t) ch_cp16(dst + t * CH_LD + 4 * p, D + 4 * e);
  }
}
__device__ __forceinline__ void ch_l2_dinv(const float* D) {
  for (int e = threadIdx.x; e < 128; e += blockDim.x) ch_l2(D + 32 * e);
}
__device__ __forceinline__ void ch_l2_block(const float* G, int64_t r0, int64_t c0, int64_t n) {
  for (int e = threadIdx.x; e < 64 * 3; e += blockDim.x) {
    const int cc = e / 3, p = e - 3 * cc;
    ch_l2(G + r0 + (c0 + cc) * n + (p == 2 ? 63 : 32 * p));
  }
}
__device__ __forceinline__ float ch_sum4(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// Bounded wait of a warp until the lanes' hand-off words (w[q], q < cnt,
// where need) are written; reloads the missing ones.  Returns false (and
// sets *err) when the limit runs out.
template <int NQ>
__device__ __forceinline__ bool ch_wait_words(unsigned long long (&w)[NQ], const double* const (&p)[NQ], int cnt,
                                              bool need, int* err, int where) {
  const uint32_t lim = g_wait_limit;
  for (uint32_t it = 0;; ++it) {
    bool ok = true;
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      if (need && q < cnt && w[q] == HAND_EMPTY) ok = false;
    if (__all_sync(0xffffffffu, ok)) return true;
    if (it >= lim) {
      if ((threadIdx.x & 31) == 0) {
        atomicExch(err, 2);
        atomicCAS(&g_solve_where, 0, where);
      }
      return false;
    }
    __nanosleep(32);
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      if (need && q < cnt && w[q] == HAND_EMPTY) w[q] = ld_hand(p[q]);
  }
}

// forward chain of one front (thread: row i = tid / 4, column phase g = tid % 4);
// right-hand sides q0 .. q0 + nq - 1, nq <= NQ
template <int NQ>
__device__ void fwd_chain(const DevCtx& c, const FrontDev& f, int q0, int nq, int* err, ChainSmem& S) {
  const int tid = threadIdx.x, i = tid >> 2, g = tid & 3;
  const int64_t n = f.n;
  const int fs = f.fs, nr = c.n_rhs, nfb = (fs + FB - 1) / FB;
  const float* __restrict__ G = c.a32 + f.off;
  const float* __restrict__ Dg = c.dinv32 + f.dinv_off;
  double* __restrict__ z = c.vec + f.voff;
  double* __restrict__ y = z + n * nr;
  double* __restrict__ w = y + n * nr;
  // every column this thread reads in a staged block (cc = 4 u + g) has the same shift
  const int sh = ch_sh(0, g, n);
  auto stage = [&](int b) {
    if (b >= nfb) return;
    float* St = &S.L[b % CH_STAGES][0][0];
    for (int k = 0; k < CH_K && b - 1 - k >= 0; ++k)
      ch_stage_block(St + k * CH_TILE, G, (int64_t)b * FB, (int64_t)(b - 1 - k) * FB, n);
    ch_stage_dinv(St + CH_K * CH_TILE, Dg + (int64_t)b * FB * FB);
  };
  auto l2_ahead = [&](int b) {
    if (b >= nfb) return;
    for (int k = 0; k < CH_K && b - 1 - k >= 0; ++k) ch_l2_block(G, (int64_t)b * FB, (int64_t)(b - 1 - k) * FB, n);
    ch_l2_dinv(Dg + (int64_t)b * FB * FB);
  };
  for (int b = CH_STAGES - 1; b < CH_L2_AHEAD; ++b) l2_ahead(b);
  for (int b = 0; b < CH_STAGES - 1; ++b) {
    stage(b);
    ch_commit();
  }
  // the right-hand side and the helper's words of a step are loaded a step
  // ahead, so that their round trip is off the chain
  double zn[NQ];
  unsigned long long pn[NQ];
  auto load_rhs = [&](int b) {
    const int row = b * FB + i;
    const bool on = b < nfb && g == 0 && i < min(FB, fs - b * FB);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      zn[q] = (on && q < nq) ? z[row + (int64_t)(q0 + q) * n] : 0.0;
      pn[q] = (on && q < nq && b > CH_K) ? ld_hand(w + row + (int64_t)(q0 + q) * n) : 0ull;
    }
  };
  load_rhs(0);
  bool live = true;
  for (int b = 0; b < nfb; ++b) {
    const int kb = min(FB, fs - b * FB), row = b * FB + i;
    const bool rv = i < kb, lead = g == 0, helped = b > CH_K;
    double zq[NQ];
    unsigned long long pw[NQ];
    const double* pp[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      pp[q] = w + row + (int64_t)(q0 + q) * n;
      zq[q] = zn[q];
      pw[q] = pn[q];
    }
    load_rhs(b + 1);
    ch_wait<CH_STAGES - 2>();
    __syncthreads();                      // step b's blocks staged, x of step b - 1 visible, stage (b - 1) free
    stage(b + CH_STAGES - 1);
    ch_commit();
    l2_ahead(b + CH_L2_AHEAD);
    const float* St = &S.L[b % CH_STAGES][0][0];
    float acc[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) acc[q] = 0.f;
    for (int k = 0; k < CH_K; ++k) {
      const int j = b - 1 - k;
      if (j < 0) break;
      const float* T = St + k * CH_TILE + sh + i;
      const float* xj = &S.xs[j % CH_K][0][0];
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int cc = 4 * u + g;
        const float l = T[cc * CH_LD];
#pragma unroll
        for (int q = 0; q < NQ; ++q) acc[q] += l * xj[q * FB + cc];
      }
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) acc[q] = ch_sum4(acc[q]);
    if (helped && live) live = ch_wait_words<NQ>(pw, pp, nq, lead && rv, err, wait_code(3, b, b));
    if (lead) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const bool on = rv && q < nq;
        const float p = helped ? (float)__longlong_as_double((long long)pw[q]) : 0.f;
        S.ts[q][i] = on ? (float)zq[q] - p - acc[q] : 0.f;
        if (on) {
          // the right-hand side and the partial sum are consumed: their words
          // become the backward solve's hand-offs
          z[row + (int64_t)(q0 + q) * n] = __longlong_as_double((long long)HAND_EMPTY);
          w[row + (int64_t)(q0 + q) * n] = __longlong_as_double((long long)HAND_EMPTY);
        }
      }
    }
    __syncthreads();
    // x_b = Dinv_b t (Dinv lower triangular)
    const float* Dm = St + CH_K * CH_TILE + i;
    float xp[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) xp[q] = 0.f;
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int t = 4 * u + g;
      if (t <= i) {
        const float d = Dm[t * CH_LD];
#pragma unroll
        for (int q = 0; q < NQ; ++q) xp[q] += d * S.ts[q][t];
      }
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) xp[q] = ch_sum4(xp[q]);
    if (lead) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const bool on = rv && q < nq;
        S.xs[b % CH_K][q][i] = on ? xp[q] : 0.f;
        if (on) st_hand(y + row + (int64_t)(q0 + q) * n, (double)xp[q]);
      }
    }
  }
  ch_wait<0>();
}

// backward chain of one front (thread: column cc = tid / 4 of the block, row phase g = tid % 4)
template <int NQ>
__device__ void bwd_chain(const DevCtx& c, const FrontDev& f, int q0, int nq, int* err, ChainSmem& S) {
  const int tid = threadIdx.x, cc = tid >> 2, g = tid & 3;
  const int64_t n = f.n;
  const int fs = f.fs, nr = c.n_rhs, nfb = (fs + FB - 1) / FB;
  const float* __restrict__ G = c.a32 + f.off;
  const float* __restrict__ Dg = c.dinv32 + f.dinv_off;
  double* __restrict__ hx = c.vec + f.voff;       // backward hand-off: the z slab's factor rows
  double* __restrict__ y = hx + n * nr;
  double* __restrict__ w = y + n * nr;
  const bool has_abl = fs < f.n;
  const int sh = ch_sh(0, cc, n);                 // this thread's column in every staged block
  // step s solves block b = nfb - 1 - s; its window: row blocks b + 1 .. b + CH_K
  auto stage = [&](int s) {
    const int b = nfb - 1 - s;
    if (b < 0) return;
    float* St = &S.L[s % CH_STAGES][0][0];
    for (int k = 0; k < CH_K && b + 1 + k < nfb; ++k)
      ch_stage_block(St + k * CH_TILE, G, (int64_t)(b + 1 + k) * FB, (int64_t)b * FB, n);
    ch_stage_dinv(St + CH_K * CH_TILE, Dg + (int64_t)b * FB * FB);
  };
  auto l2_ahead = [&](int s) {
    const int b = nfb - 1 - s;
    if (b < 0) return;
    for (int k = 0; k < CH_K && b + 1 + k < nfb; ++k) ch_l2_block(G, (int64_t)(b + 1 + k) * FB, (int64_t)b * FB, n);
    ch_l2_dinv(Dg + (int64_t)b * FB * FB);
  };
  for (int s = CH_STAGES - 1; s < CH_L2_AHEAD; ++s) l2_ahead(s);
  for (int s = 0; s < CH_STAGES - 1; ++s) {
    stage(s);
    ch_commit();
  }
  // the forward solution and the helper's words of a step, a step ahead
  double yn[NQ];
  unsigned long long pn[NQ];
  auto load_rhs = [&](int s) {
    const int b = nfb - 1 - s, col = b * FB + cc;
    const bool on = b >= 0 && g == 0 && cc < min(FB, fs - b * FB);
    const bool helped = has_abl || b + CH_K + 1 <= nfb - 1;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      yn[q] = (on && q < nq) ? y[col + (int64_t)(q0 + q) * n] : 0.0;
      pn[q] = (on && q < nq && helped) ? ld_hand(w + col + (int64_t)(q0 + q) * n) : 0ull;
    }
  };
  load_rhs(0);
  bool live = true;
  for (int s = 0; s < nfb; ++s) {
    const int b = nfb - 1 - s;
    const int kb = min(FB, fs - b * FB), col = b * FB + cc;
    const bool cv = cc < kb, lead = g == 0;
    const bool helped = has_abl || b + CH_K + 1 <= nfb - 1;
    double yq[NQ];
    unsigned long long pw[NQ];
    const double* pp[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      pp[q] = w + col + (int64_t)(q0 + q) * n;
      yq[q] = yn[q];
      pw[q] = pn[q];
    }
    load_rhs(s + 1);
    ch_wait<CH_STAGES - 2>();
    __syncthreads();
    stage(s + CH_STAGES - 1);
    ch_commit();
    l2_ahead(s + CH_L2_AHEAD);
    const float* St = &S.L[s % CH_STAGES][0][0];
    float acc[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) acc[q] = 0.f;
    for (int k = 0; k < CH_K; ++k) {
      const int r = b + 1 + k;
      if (r >= nfb) break;
      const int kbr = min(FB, fs - r * FB);
      const float* T = St + k * CH_TILE + cc * CH_LD + sh;
      const float* xr = &S.xs[r % CH_K][0][0];
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int ii = 4 * u + g;
        // rows past the factor block hold other data: skipped, not multiplied by 0
        const float l = ii < kbr ? T[ii] : 0.f;
#pragma unroll
        for (int q = 0; q < NQ; ++q) acc[q] += l * xr[q * FB + ii];
      }
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) acc[q] = ch_sum4(acc[q]);
    if (helped && live) live = ch_wait_words<NQ>(pw, pp, nq, lead && cv, err, wait_code(4, b, b));
    if (lead) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const bool on = cv && q < nq;
        const float p = helped ? (float)__longlong_as_double((long long)pw[q]) : 0.f;
        S.ts[q][cc] = on ? (float)yq[q] - p - acc[q] : 0.f;
      }
    }
    __syncthreads();
    // x_b = Dinv_b^T t: x[cc] = sum_{t >= cc} Dinv[t][cc] t[t]
    const float* Dm = St + CH_K * CH_TILE + cc * CH_LD;
    float xp[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) xp[q] = 0.f;
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int t = 4 * u + g;
      if (t >= cc) {
        const float d = Dm[t];
#pragma unroll
        for (int q = 0; q < NQ; ++q) xp[q] += d * S.ts[q][t];
      }
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) xp[q] = ch_sum4(xp[q]);
    if (lead) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const bool on = cv && q < nq;
        S.xs[b % CH_K][q][cc] = on ? xp[q] : 0.f;
        if (on) {
          y[col + (int64_t)(q0 + q) * n] = (double)xp[q];
          st_hand(hx + col + (int64_t)(q0 + q) * n, (double)xp[q]);
        }
      }
    }
  }
  ch_wait<0>();
}

// Helper and ABL rows of the forward chain: acc[q] = sum over column blocks
// j < jend of L[row, block j] x_j for the CTA's 64 rows r0.. (thread: row
// lane tid % 64, column group tid / 64).  The blocks stream through
// shared memory CH_HS - 1 ahead (cp.async); warp 0 keeps the hand-off words
// of CH_HW blocks in flight, waits (bounded) for each block's words and
// stages their values.
template <int NQ>
__device__ __forceinline__ void chain_fwd_rows(const DevCtx& c, const FrontDev& f, int r0, int jend, int q0, int nq,
                                               int* err, float (&acc)[NQ], ChainRowSmem& S) {
  const int64_t n = f.n;
  const int fs = f.fs, i = threadIdx.x % FB, g = threadIdx.x / FB;
  const float* __restrict__ G = c.a32 + f.off;
  const double* __restrict__ y = c.vec + f.voff + n * c.n_rhs;
  const bool w0 = threadIdx.x < 32;
  int sh[4];                        // shift of the staged columns cc with cc % 4 = 0, 1, 2, 3
#pragma unroll
  for (int k = 0; k < 4; ++k) sh[k] = ch_sh(r0, k, n);
  auto kbj = [&](int j) { return min(FB, fs - j * FB); };
  auto stage = [&](int j) {
    if (j < jend) ch_stage_block(S.L[j % CH_HS], G, r0, (int64_t)j * FB, n, kbj(j));
  };
  for (int j = 0; j < CH_HS - 1; ++j) {
    stage(j);
    ch_commit();
  }
  HandWords hw[CH_HW];
  bool live = true;
  if (w0) {
#pragma unroll
    for (int u = 0; u < CH_HW; ++u)
      if (u < jend) hw[u].load(y + u * FB + (int64_t)q0 * n, kbj(u));
  }
  for (int J = 0; J < jend; J += CH_HW) {
#pragma unroll
    for (int u = 0; u < CH_HW; ++u) {
      const int j = J + u;
      if (j >= jend) break;
      const int kb = kbj(j);
      if (w0) {
        const double* yj = y + j * FB;
        if (live) live = hw[u].wait(yj + (int64_t)q0 * n, kb, err, wait_code(1, j, r0 / FB));
        hw[u].stage(S.vsh[j & 1][0]);
        for (int q = 1; q < nq; ++q) {
          HandWords hq;
          hq.load(yj + (int64_t)(q0 + q) * n, kb);
          if (live) live = hq.wait(yj + (int64_t)(q0 + q) * n, kb, err, wait_code(1, j, r0 / FB));
          hq.stage(S.vsh[j & 1][q]);
        }
        if (j + CH_HW < jend) hw[u].load(y + (j + CH_HW) * FB + (int64_t)q0 * n, kbj(j + CH_HW));
      }
      ch_wait<CH_HS - 2>();
      __syncthreads();
      stage(j + CH_HS - 1);
      ch_commit();
      const float* T = S.L[j % CH_HS] + i;
      const float* v = &S.vsh[j & 1][0][0];
#pragma unroll
      for (int uu = 0; uu < 16; ++uu) {
        const int cc = g * 16 + uu;
        // columns past the factor block hold other data: skipped
        const float l = cc < kb ? T[cc * CH_LD + sh[uu & 3]] : 0.f;
#pragma unroll
        for (int q = 0; q < NQ; ++q) acc[q] += l * v[q * FB + cc];
      }
    }
  }
  ch_wait<0>();
}

// Helper rows of the backward chain for column block b: acc[q][u] = sum over
// the row blocks below the chain's window (the ABL rows, x from the parent,
// then the factor blocks nfb - 1 down to b + CH_K + 1, x from the hand-off
// words) of L[r, 64 b + 16 g + u] x_r (thread: row lane tid % 64, column
// group tid / 64); staged as in chain_fwd_rows.
template <int NQ>
__device__ __forceinline__ void chain_bwd_rows(const DevCtx& c, const FrontDev& f, int b, int q0, int nq, int* err,
                                               float (&acc)[NQ][16], ChainRowSmem& S) {
  const int64_t n = f.n;
  const int fs = f.fs, nfb = (fs + FB - 1) / FB, rl = threadIdx.x % FB, g = threadIdx.x / FB;
  const int kbc = min(FB, fs - b * FB);
  const float* __restrict__ G = c.a32 + f.off;
  const double* __restrict__ hx = c.vec + f.voff;
  const double* __restrict__ y = hx + n * c.n_rhs;
  const int nab = (int)((n - fs + FB - 1) / FB);
  const int nfar = max(0, nfb - 1 - (b + CH_K));
  const int tend = nab + nfar;
  // row block t: the ABL blocks first, then factor blocks from the last one up
  auto r0_of = [&](int t) { return t < nab ? fs + t * FB : (nfb - 1 - (t - nab)) * FB; };
  auto rend_of = [&](int t) { return t < nab ? (int)n : min((nfb - 1 - (t - nab)) * FB + FB, fs); };
  auto src_of = [&](int t) -> const double* { return t < nab ? y : hx; };
  auto stage = [&](int t) {
    if (t < tend) ch_stage_block(S.L[t % CH_HS], G, r0_of(t), (int64_t)b * FB, n, kbc);
  };
  for (int t = 0; t < CH_HS - 1; ++t) {
    stage(t);
    ch_commit();
  }
  const bool w0 = threadIdx.x < 32;
  HandWords hw[CH_HW];
  bool live = true;
  if (w0) {
#pragma unroll
    for (int u = 0; u < CH_HW; ++u)
      if (u < tend) hw[u].load(src_of(u) + r0_of(u) + (int64_t)q0 * n, rend_of(u) - r0_of(u));
  }
  for (int T0 = 0; T0 < tend; T0 += CH_HW) {
#pragma unroll
    for (int u = 0; u < CH_HW; ++u) {
      const int t = T0 + u;
      if (t >= tend) break;
      const int r0 = r0_of(t), kr = rend_of(t) - r0;
      if (w0) {
        const double* xr = src_of(t) + r0;
        if (live) live = hw[u].wait(xr + (int64_t)q0 * n, kr, err, wait_code(2, r0 / FB, b));
        hw[u].stage(S.vsh[t & 1][0]);
        for (int q = 1; q < nq; ++q) {
          HandWords hq;
          hq.load(xr + (int64_t)(q0 + q) * n, kr);
          if (live) live = hq.wait(xr + (int64_t)(q0 + q) * n, kr, err, wait_code(2, r0 / FB, b));
          hq.stage(S.vsh[t & 1][q]);
        }
        if (t + CH_HW < tend)
          hw[u].load(src_of(t + CH_HW) + r0_of(t + CH_HW) + (int64_t)q0 * n, rend_of(t + CH_HW) - r0_of(t + CH_HW));
      }
      ch_wait<CH_HS - 2>();
      __syncthreads();
      stage(t + CH_HS - 1);
      ch_commit();
      if (rl < kr) {
        // rows past the block (or the front) hold other data: skipped
        const float* Tt = S.L[t % CH_HS] + rl;
        int sh[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) sh[k] = ch_sh(r0, k, n);
        float xv[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) xv[q] = S.vsh[t & 1][q][rl];
#pragma unroll
        for (int uu = 0; uu < 16; ++uu) {
          const int cc = g * 16 + uu;
          const float l = cc < kbc ? Tt[cc * CH_LD + sh[uu & 3]] : 0.f;
#pragma unroll
          for (int q = 0; q < NQ; ++q) acc[q][uu] += l * xv[q];
        }
      }
    }
  }
  ch_wait<0>();
}

template <int NQ>
__device__ __forceinline__ void fwd_chain_cta(const DevCtx& c, const Item& it, const FrontDev& f, int q0, int nq,
                                              int* err, unsigned char* raw) {
  if (it.b == CH_CHAIN) {
    fwd_chain<NQ>(c, f, q0, nq, err, *reinterpret_cast<ChainSmem*>(raw));
    return;
  }
  ChainRowSmem& H = *reinterpret_cast<ChainRowSmem*>(raw);
  const int n = f.n, fs = f.fs, nfb = (fs + FB - 1) / FB, b = it.a;
  const bool helper = it.b == CH_HELPER;      // else CH_ABL
  const int r0 = helper ? b * FB : fs + (b - nfb) * FB;
  const int r1 = helper ? min(r0 + FB, fs) : min(r0 + FB, n);
  const int i = threadIdx.x % FB, gg = threadIdx.x / FB, row = r0 + i;
  const bool rv = row < r1;
  double* __restrict__ z = c.vec + f.voff;
  double* __restrict__ w = z + 2 * (int64_t)n * c.n_rhs;
  if (helper) {
    // the chain reads this row block's CH_K blocks next to the diagonal and
    // its inverse from one SM: start them towards L2 long before
    for (int k = 1; k <= CH_K; ++k) ch_l2_block(c.a32 + f.off, (int64_t)b * FB, (int64_t)(b - k) * FB, n);
    ch_l2_dinv(c.dinv32 + f.dinv_off + (int64_t)b * FB * FB);
  }
  float zr[NQ], acc[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    acc[q] = 0.f;
    zr[q] = (!helper && rv && q < nq && gg == 0) ? (float)z[row + (int64_t)(q0 + q) * n] : 0.f;
  }
  chain_fwd_rows<NQ>(c, f, r0, helper ? b - CH_K : nfb, q0, nq, err, acc, H);
#pragma unroll
  for (int q = 0; q < NQ; ++q) H.red[gg][i][q] = acc[q];
  __syncthreads();
  if (threadIdx.x < FB && rv) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      if (q >= nq) break;
      const float sum = H.red[0][i][q] + H.red[1][i][q] + H.red[2][i][q] + H.red[3][i][q];
      if (helper) st_hand(w + row + (int64_t)(q0 + q) * n, (double)sum);
      else z[row + (int64_t)(q0 + q) * n] = (double)(zr[q] - sum);
    }
  }
}

template <int NQ>
__device__ __forceinline__ void bwd_chain_cta(const DevCtx& c, const Item& it, const FrontDev& f, int q0, int nq,
                                              int* err, unsigned char* raw) {
  if (it.b == CH_CHAIN) {
    bwd_chain<NQ>(c, f, q0, nq, err, *reinterpret_cast<ChainSmem*>(raw));
    return;
  }
  ChainRowSmem& H = *reinterpret_cast<ChainRowSmem*>(raw);
  const int n = f.n, fs = f.fs, b = it.a;
  const int c0 = b * FB, kb = min(FB, fs - c0);
  double* __restrict__ w = c.vec + f.voff + 2 * (int64_t)n * c.n_rhs;
  const int rl = threadIdx.x % FB, gg = threadIdx.x / FB;
  {
    // the chain's blocks below this column block's diagonal and its inverse, towards L2
    const int nfb = (fs + FB - 1) / FB;
    for (int k = 1; k <= CH_K && b + k < nfb; ++k) ch_l2_block(c.a32 + f.off, (int64_t)(b + k) * FB, (int64_t)b * FB, n);
    ch_l2_dinv(c.dinv32 + f.dinv_off + (int64_t)b * FB * FB);
  }
  float acc[NQ][16];
#pragma unroll
  for (int q = 0; q < NQ; ++q)
#pragma unroll
    for (int u = 0; u < 16; ++u) acc[q][u] = 0.f;
  chain_bwd_rows<NQ>(c, f, b, q0, nq, err, acc, H);
  // column sums over the 64 row lanes, one right-hand side at a time
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    if (q >= nq) break;
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 16; ++u) H.redb[rl][gg * 16 + u] = acc[q][u];
    __syncthreads();
    if (threadIdx.x < kb) {
      float s = 0.f;
      for (int r = 0; r < FB; ++r) s += H.redb[r][threadIdx.x];
      st_hand(w + c0 + threadIdx.x + (int64_t)(q0 + q) * n, (double)s);
    }
  }
}

// item: front, a = block, b = role; right-hand sides q0 .. q0 + SF_NR - 1
__global__ void __launch_bounds__(256, 1) k_fwd_chain(DevCtx c, const Item* __restrict__ items, int* ticket, int* err,
                                                      int q0) {
  extern __shared__ __align__(16) unsigned char ch_raw[];
  __shared__ int s_t;
  if (threadIdx.x == 0) s_t = atomicAdd(ticket, 1);
  __syncthreads();
  const Item it = items[s_t];
  const FrontDev f = c.fronts[it.front];
  const int nq = min(SF_NR, c.n_rhs - q0);
  if (nq == 1) fwd_chain_cta<1>(c, it, f, q0, nq, err, ch_raw);
  else if (nq == 2) fwd_chain_cta<2>(c, it, f, q0, nq, err, ch_raw);
  else fwd_chain_cta<SF_NR>(c, it, f, q0, nq, err, ch_raw);
}

// item: front, a = column block, b = role (chain or helper); right-hand sides q0 .. q0 + SF_NR - 1
__global__ void __launch_bounds__(256, 1) k_bwd_chain(DevCtx c, const Item* __restrict__ items, int* ticket, int* err,
                                                      int q0) {
  extern __shared__ __align__(16) unsigned char ch_raw[];
  __shared__ int s_t;
  if (threadIdx.x == 0) s_t = atomicAdd(ticket, 1);
  __syncthreads();
  const Item it = items[s_t];
  const FrontDev f = c.fronts[it.front];
  const int nq = min(SF_NR, c.n_rhs - q0);
  if (nq == 1) bwd_chain_cta<1>(c, it, f, q0, nq, err, ch_raw);
  else if (nq == 2) bwd_chain_cta<2>(c, it, f, q0, nq, err, ch_raw);
  else bwd_chain_cta<SF_NR>(c, it, f, q0, nq, err, ch_raw);
}

void launch_fwd_chain(const DevCtx& c, const Item* items, int n_items, int* ticket, int* err, int q0,
                      cudaStream_t s) {
  if (!n_items) return;
  cudaMemsetAsync(ticket, 0, sizeof(int), s);
  cudaFuncSetAttribute(k_fwd_chain, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CH_SMEM);
  k_fwd_chain<<<n_items, 256, CH_SMEM, s>>>(c, items, ticket, err, q0);
}

void launch_bwd_chain(const DevCtx& c, const Item* items, int n_items, int* ticket, int* err, int q0,
                      cudaStream_t s) {
  if (!n_items) return;
  cudaMemsetAsync(ticket, 0, sizeof(int), s);
  cudaFuncSetAttribute(k_bwd_chain, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CH_SMEM);
  k_bwd_chain<<<n_items, 256, CH_SMEM, s>>>(c, items, ticket, err, q0);
}

}  // namespace uhm_gpu
