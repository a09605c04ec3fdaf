// Tensor-core Schur update for FP32 fronts: C -= A21 * A21^T (Cholesky) with
// BF16-split operands on the 5th-generation tensor cores (tcgen05).
//
// The update restates the trailing SYRK of the front's blocked Cholesky
// (LINAL/src/dense/chol.cxx:78-82 and the front-level syrk of
// UHM/src/matrix/uhm/fla/chol/decompose.cxx:94-95).
//
// Split precision: every FP32 entry a = hi + lo + (mid) with hi, lo (, mid)
// BF16 (round to nearest); the product a*b is taken as the sum of BF16
// products hi*hi + hi*lo + lo*hi ("bf16x3", ~2^-17 relative) or, with three
// parts, the six terms of order <= 2^-16 ("bf16x6", FP32-class), all
// accumulated in FP32 in tensor memory.
//
// Kernel: one persistent CTA per SM walks the 128 x 128 output tiles; warp 16
// issues TMA loads (128-byte swizzle) into a shared-memory ring guarded by
// mbarriers, warp 17 issues tcgen05.mma (M=128, N=128, K=16) into one of two
// 128-column TMEM accumulators, warps 0-15 (a 32-lane quarter and 32 columns
// each) read TMEM back (tcgen05.ld) and apply C -= acc to the FP32 panel while
// the next tile accumulates in the other buffer.  Every wait is bounded: a wait
// that gives up records an error flag and the CTA skips its stores.
//
// Bound by the memory traffic of C (read and written once: K = 256 leaves 24 flops
// per byte) and by the operands' way from L2.  A ring slot holds every part of a
// 64-column chunk of A and of B, so that a part used by two terms is loaded once
// (256 KB instead of 384 per tile in bf16x3); a warp's 32 loads of C go out
// before it waits for the products, 64 KB per SM, where eight warps staging C
// through shared memory 16 loads at a time had 16 KB.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <cstdio>
#include <stdexcept>

#include "k_common.cuh"
#include "k_tc.cuh"
#include "k_tc_ptx.cuh"

namespace uhm_gpu {

constexpr int TC_BM = 128, TC_BN = 128, TC_BK = 64;
constexpr int TC_EPI_WARPS = 16;
constexpr int TC_THREADS = 32 * (TC_EPI_WARPS + 2);     // epilogue, TMA producer, MMA issuer
constexpr uint32_t TC_TILE_BYTES = TC_BM * TC_BK * 2;   // 16 KB (A and B tiles alike)
constexpr uint32_t TC_RING = 12 * TC_TILE_BYTES;        // slots of 2 x parts tiles: 3 (bf16x3) or 2 (bf16x6)
constexpr int TC_SLOTS_MAX = 3;
constexpr uint32_t TC_SMEM = 1024 + TC_RING + 256;

UHM_DEFINE_WAIT_LIMIT(set_wait_limit_tc, 1u << 24)

// bounded wait: false (and error flag) when the barrier never completes
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                          int* err) {
  return mbar_wait_lim(bar, parity, abort_flag, err, 1, g_wait_limit);
}

// item: front, a = K0 (outer step start), b = tile row, c = tile col
// (tiles counted from the trailing block's first row K0 + KB).
// Operand parts: A 0 .. PARTS - 1, B pb0 .. pb0 + PARTS - 1; the products of parts p
// and q, p + q < PARTS (three terms for two parts, six for three).
//
// Persistent: one CTA per SM walks the tile list with stride gridDim.x.  The
// TMA ring (full / empty barriers) runs continuously across tiles; TMEM holds
// two 128-column accumulators, so the epilogue of tile i (TMEM -> registers
// -> C in global memory) overlaps the mainloop of tile i + 1.  acc_full[b]
// is committed by the MMA warp when accumulator b holds a finished tile;
// acc_empty[b] collects the epilogue warps once they have read it.
// Measured on GB300, the LU trailing updates of 24^3 p = 3 (BF16X3, K = 256):
// 21.7 -> 15.6 ms; 13,000 tiles 513 -> 379 us, of which C's traffic alone is 251 (420
// before the next tile's C was asked into L2 while a tile's products run and a part
// of A was kept in the collector buffer).
template <int PARTS>
__global__ void __launch_bounds__(TC_THREADS, 1)
k_tc_syrk(DevCtx c, const __grid_constant__ CUtensorMap wsmap, const int64_t* __restrict__ ws_off,
          const int64_t* __restrict__ ws_stride, const Item* __restrict__ items, int n_items, int nbo,
          int pb0, int lower_only, int* err) {
  extern __shared__ __align__(1024) uint8_t tc_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + TC_RING);
  uint64_t* empty = bars + TC_SLOTS_MAX;
  uint64_t* acc_full = empty + TC_SLOTS_MAX;
  uint64_t* acc_empty = acc_full + 2;
  uint64_t* drain_bar = acc_empty + 2;
  volatile int* s_abort = reinterpret_cast<volatile int*>(drain_bar + 1);
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(drain_bar + 2);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int parts = PARTS;
  constexpr uint32_t slot_bytes = 2 * (uint32_t)parts * TC_TILE_BYTES;
  constexpr int slots = TC_RING / slot_bytes;
  static_assert(slots >= 2 && slots <= TC_SLOTS_MAX, "ring");

  if (threadIdx.x == 0) {
    for (int s = 0; s < TC_SLOTS_MAX; ++s) {
      mbar_init(smem_u32(&bars[s]), 1);
      mbar_init(smem_u32(&empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&acc_full[b]), 1);
      mbar_init(smem_u32(&acc_empty[b]), TC_EPI_WARPS);
    }
    mbar_init(smem_u32(drain_bar), 1);
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)),
                 "r"(2 * TC_BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *s_tmem;

  if (warp == TC_EPI_WARPS) {
    if (lane == 0) {
      // TMA producer
      int s = 0;
      uint32_t ph = 1;               // parity of the empty wait (the first round passes)
      uint32_t issued = 0;           // chunks
      bool live = true;
      for (int t = blockIdx.x; t < n_items && live; t += gridDim.x) {
        const Item it = items[t];
        const int KB = min(nbo, c.fronts[it.front].fs - it.a);
        const int nk = (KB + TC_BK - 1) / TC_BK;
        // the whole BF16 workspace is one 2D tensor of rows of nbo elements;
        // part p of this front starts at row (ws_off + p * ws_stride) / nbo
        const int prow = (int)(ws_stride[it.front] / nbo);
        const int ra = (int)(ws_off[it.front] / nbo) + it.b * TC_BM;
        const int rb = (int)(ws_off[it.front] / nbo) + pb0 * prow + it.c * TC_BN;
        for (int kk = 0; kk < nk; ++kk) {
          if (issued >= (uint32_t)slots && !mbar_wait(smem_u32(&empty[s]), ph, s_abort, err)) {
            live = false;
            break;
          }
          const uint32_t fb = smem_u32(&bars[s]), st = smem_u32(smem) + s * slot_bytes;
          mbar_expect_tx(fb, slot_bytes);
          for (int p = 0; p < parts; ++p) {
            tma_load_2d(st + p * TC_TILE_BYTES, &wsmap, kk * TC_BK, ra + p * prow, fb);
            tma_load_2d(st + (parts + p) * TC_TILE_BYTES, &wsmap, kk * TC_BK, rb + p * prow, fb);
          }
          ++issued;
          if (++s == slots) { s = 0; ph ^= 1; }
        }
      }
      // the last loads issued (one chunk per slot at most) have landed before
      // the CTA exits, whether or not the MMA warp consumed them
      const uint32_t cnt = issued < (uint32_t)slots ? issued : (uint32_t)slots;
      for (uint32_t q = issued - cnt; q < issued; ++q) mbar_drain(smem_u32(&bars[q % slots]), (q / slots) & 1);
    }
  } else if (warp == TC_EPI_WARPS + 1) {
    // MMA issuer: the whole warp, one elected lane issuing
    const uint32_t elected = elect_one();
    const uint32_t idesc = idesc_bf16_f32(TC_BM, TC_BN);
    const uint32_t ring = smem_u32(smem), bar0 = smem_u32(bars), empty0 = smem_u32(empty);
    auto wait = [&](uint32_t bar, uint32_t parity) {
      return __all_sync(0xffffffffu, mbar_wait(bar, parity, s_abort, err)) != 0;
    };
    int s = 0, i = 0;
    uint32_t ph = 0;
    bool live = true;
    for (int t = blockIdx.x; t < n_items && live; t += gridDim.x, ++i) {
      const Item it = items[t];
      const int nk = __shfl_sync(0xffffffffu, (min(nbo, c.fronts[it.front].fs - it.a) + TC_BK - 1) / TC_BK, 0);
      const int b = i & 1, u = i >> 1;
      if (u >= 1 && !wait(smem_u32(&acc_empty[b]), (u - 1) & 1)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t acc = tmem + b * TC_BN;
      uint32_t on = 0;
      for (int kk = 0; kk < nk; ++kk) {
        live = wait(bar0 + 8 * s, ph);
        if (!live) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a0 = sdesc_lo(ring + (uint32_t)s * slot_bytes);
        const uint32_t b0 = sdesc_lo(ring + (uint32_t)s * slot_bytes + (uint32_t)parts * TC_TILE_BYTES);
        // per 16 columns, part of A by part of A: its products with parts 0 .. PARTS -
        // 1 - p of B; A is read from shared memory once (collector buffer)
#pragma unroll
        for (int k = 0; k < TC_BK / 16; ++k)
#pragma unroll
          for (int p = 0; p < PARTS; ++p)
#pragma unroll
            for (int q = 0; q < PARTS - p; ++q) {
              const uint32_t at = a0 + p * (TC_TILE_BYTES >> 4) + 2 * k, bt = b0 + q * (TC_TILE_BYTES >> 4) + 2 * k;
              if (k == 0 && p == 0 && q == 0) {
                umma_bf16_w(elected, acc, at, bt, SDESC_SW128_HI, idesc, on);
                on = 1u;
              } else if (k == 0 && p == 0 || p == PARTS - 1) {
                umma_bf16_w(elected, acc, at, bt, SDESC_SW128_HI, idesc, 1u);
              } else if (q == 0) {
                umma_bf16_wa<UMMA_A_FILL>(elected, acc, at, bt, SDESC_SW128_HI, idesc);
              } else if (q < PARTS - p - 1) {
                umma_bf16_wa<UMMA_A_USE>(elected, acc, at, bt, SDESC_SW128_HI, idesc);
              } else {
                umma_bf16_wa<UMMA_A_LAST>(elected, acc, at, bt, SDESC_SW128_HI, idesc);
              }
            }
        umma_commit_w(elected, empty0 + 8 * s);
        if (++s == slots) { s = 0; ph ^= 1; }
      }
      if (live) umma_commit_w(elected, smem_u32(&acc_full[b]));
    }
    // every MMA issued has completed before TMEM is freed
    umma_commit_w(elected, smem_u32(drain_bar));
    mbar_drain(smem_u32(drain_bar), 0);
  } else {
    // epilogue: warp w reads TMEM lanes [32 (w % 4), +32) (its lane quarter =
    // tile rows) and handles the columns [32 (w / 4), +32); the entries of C are
    // loaded while the products run
    constexpr int NC = TC_BN / 4;
    static_assert(NC == 32, "a lane per column of the prefetch");
    const int quarter = warp & 3, cg = warp >> 2;
    // columns c0 + j, j < cend, of this thread's row are updated, entry 0 at G
    struct Geo { float* G; int n, cend; };
    auto geo_of = [&](int t) {
      const Item it = items[t];
      const FrontDev& f = c.fronts[it.front];
      const int n = f.n, base = it.a + min(nbo, f.fs - it.a);
      const int row = base + it.b * TC_BM + quarter * 32 + lane, c0 = base + it.c * TC_BN + cg * NC;
      return Geo{c.a32 + f.off + row + (int64_t)c0 * n, n, row < n ? (lower_only ? min(n, row + 1) : n) - c0 : 0};
    };
    int i = 0;
    Geo cur = {};
    if ((int)blockIdx.x < n_items) cur = geo_of(blockIdx.x);
    for (int t = blockIdx.x; t < n_items; t += gridDim.x, ++i) {
      const int n = cur.n, cend = cur.cend;
      float* __restrict__ G = cur.G;
      float v[NC];
#pragma unroll
      for (int j = 0; j < NC; ++j) v[j] = j < cend ? __ldcg(G + (int64_t)j * n) : 0.0f;
      // the next tile's C towards L2: lane j asks for the rows of column j, at its
      // first and its last row
      if (t + (int)gridDim.x < n_items) {
        cur = geo_of(t + gridDim.x);
        const float* p0 = cur.G - lane + (int64_t)lane * cur.n;
        const int most = __reduce_max_sync(0xffffffffu, cur.cend);
        const unsigned rows = __ballot_sync(0xffffffffu, cur.cend > 0);
        if (lane < most) {
          asm volatile("prefetch.global.L2 [%0];" ::"l"(p0 + __ffs(rows) - 1));
          asm volatile("prefetch.global.L2 [%0];" ::"l"(p0 + 31 - __clz(rows)));
        }
      }
      const int b = i & 1, u = i >> 1;
      const bool ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&acc_full[b]), u & 1, s_abort, err));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t a[NC];
      TC_LD32(tmem + ((uint32_t)(quarter * 32) << 16) + b * TC_BN + cg * NC, a);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      // accumulator b may be overwritten from here on
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&acc_empty[b]));
      if (!*s_abort) {
#pragma unroll
        for (int j = 0; j < NC; ++j)
          if (j < cend) G[(int64_t)j * n] = v[j] - __uint_as_float(a[j]);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * TC_BN));
  }
}

// Split the panel A[K0+KB : n, K0 : K0+KB] (FP32, column-major, ld n) into
// BF16 parts stored row-major with row length nbo (zero beyond KB):
// part p row r = round-to-nearest BF16 of the p-th residual.
// item: front, a = K0, b = row block (64 rows)
// trans = 1 packs U12^T instead: row r is column base + r of the front, rows
// K0..K0+KB (the LU panel's U block right of the outer panel), into parts
// poff.. (the B operand of the LU trailing update).
__global__ void __launch_bounds__(256) k_tc_pack(DevCtx c, const Item* __restrict__ items, int nbo,
                                                 int nparts, __nv_bfloat16* __restrict__ ws,
                                                 const int64_t* __restrict__ ws_off,
                                                 const int64_t* __restrict__ ws_stride, int trans, int poff) {
  __shared__ float tile[64][65];
  const Item it = items[blockIdx.x];
  const FrontDev f = c.fronts[it.front];
  const int n = f.n, K0 = it.a;
  const int KB = min(nbo, f.fs - K0);
  const int base = K0 + KB;
  const int r0 = it.b * 64;
  const float* __restrict__ G = c.a32 + f.off;
  __nv_bfloat16* __restrict__ W = ws + ws_off[it.front];
  const int64_t pstride = ws_stride[it.front];
  for (int k0 = 0; k0 < nbo; k0 += 64) {
    // one batch of 16 independent loads per thread (coalesced along the
    // column), then the shared-memory transpose
    float v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int idx = threadIdx.x + 256 * u;
      const int r = trans ? idx / 64 : idx % 64, k = trans ? idx % 64 : idx / 64;
      const int gr = base + r0 + r, gk = k0 + k;
      v[u] = (gr < n && gk < KB) ? (trans ? G[(K0 + gk) + (int64_t)gr * n] : G[gr + (int64_t)(K0 + gk) * n])
                                 : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int idx = threadIdx.x + 256 * u;
      const int r = trans ? idx / 64 : idx % 64, k = trans ? idx % 64 : idx / 64;
      tile[r][k] = v[u];
    }
    __syncthreads();
    // each thread converts 8 consecutive k of one row and writes every part
    // as one 16-byte store
#pragma unroll
    for (int h2 = 0; h2 < 2; ++h2) {
      const int idx = threadIdx.x + 256 * h2, r = idx / 8, k8 = (idx % 8) * 8;
      if (base + r0 + r >= n) continue;
      float x[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) x[q] = tile[r][k8 + q];
      for (int p = 0; p < nparts; ++p) {
        __align__(16) __nv_bfloat16 hb[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          hb[q] = __float2bfloat16_rn(x[q]);
          x[q] -= __bfloat162float(hb[q]);
        }
        *reinterpret_cast<uint4*>(W + (p + poff) * pstride + (int64_t)(r0 + r) * nbo + k0 + k8) =
            *reinterpret_cast<const uint4*>(hb);
      }
    }
  }
}

// ---- host side ---------------------------------------------------------------
static PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;

static bool get_encoder() {
  if (g_encode) return true;
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) !=
          cudaSuccess ||
      q != cudaDriverEntryPointSuccess || !fn) {
    cudaGetLastError();
    return false;
  }
  g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  return true;
}

// 2D map over a row-major rows x nbo BF16 matrix, box 64 (K) x 128 (rows)
bool tc_encode_part(CUtensorMap* map, void* base, int64_t rows, int nbo) {
  if (!get_encoder()) return false;
  cuuint64_t dims[2] = {(cuuint64_t)nbo, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)nbo * 2};
  cuuint32_t box[2] = {TC_BK, TC_BM};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

void launch_tc_pack(const DevCtx& c, const Item* items, int n_items, int nbo, int nparts, void* ws,
                    const int64_t* ws_off, const int64_t* ws_stride, int trans, int poff, cudaStream_t s) {
  if (!n_items) return;
  k_tc_pack<<<n_items, 256, 0, s>>>(c, items, nbo, nparts, (__nv_bfloat16*)ws, ws_off, ws_stride, trans, poff);
}

void launch_tc_syrk(const DevCtx& c, const CUtensorMap& wsmap, const int64_t* ws_off,
                    const int64_t* ws_stride, const Item* items, int n_items, int nbo, int parts, int pb0,
                    int lower_only, int cap, int* err, cudaStream_t s) {
  if (!n_items) return;
  if (parts != 2 && parts != 3) throw std::invalid_argument("tc_syrk: operands of two or three parts");
  static int n_sm = 0;
  if (!n_sm) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
    if (n_sm <= 0) n_sm = 1;
  }
  const auto kernel = parts == 2 ? k_tc_syrk<2> : k_tc_syrk<3>;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM);
  const int sms = cap > 0 && cap < n_sm ? cap : n_sm;
  const int grid = n_items < sms ? n_items : sms;   // one persistent CTA per SM
  kernel<<<grid, TC_THREADS, TC_SMEM, s>>>(c, wsmap, ws_off, ws_stride, items, n_items, nbo, pb0, lower_only, err);
}

int tc_tile() { return TC_BM; }

}  // namespace uhm_gpu
