// Launchers of the sliced tensor-core updates of FP64 and FP32 fronts (k_xs.cu).
#pragma once
#include <cuda.h>
#include <cstdint>
#include "kernels.cuh"

namespace uhm_gpu {

constexpr int XS_NBO = 256;       // outer panel width: columns whose slices share a row exponent at most
constexpr int XS_TILE = 128;      // update tiles: XS_TILE rows, XS_TILE or 64 columns
constexpr int xs_pack_rows(int nb) { return nb == 64 ? 64 : 16; }   // rows per pack item
constexpr int XS_TRSM_ROWS = 16;  // rows per item of the FP64 panel TRSM
constexpr int XS_S64 = 8, XS_S32 = 4;   // slices of an FP64 / FP32 front's operands
constexpr int XS_SPARE_ROWS = 256;      // workspace rows past the last front's (tiles run over)
// LU: entries within 2^XS_NEAR of their row's maximum count as near it (k_xs.cu)
constexpr int XS_NEAR64 = 6, XS_NEAR32 = 6;
constexpr int XS_SCALE0 = 1 << 12;      // (a word of scale that nothing has raised is zero)
constexpr int XS_USES = 3;        // pairs of operands of a panel column: the update's region (0, 1, 2)

// Where the operand slices live: 128-byte rows of four slices x 16 columns (BF16),
// row ((group of slices) (16-column chunks) + chunk) n + r, per front first
// row row0[front] (A and, Cholesky, B) and row0b[front] (LU: B = U12^T), one
// exponent per front row at exp0[front] / exp0 + nb_off.
struct XsCtx {
  void* ws;
  const int64_t* row0;
  const int64_t* row0b;
  const int64_t* exp0;     // first exponent of the front's A rows; its B rows follow at + n
  int* exps;
  // LU (otherwise null), what scales and checks the slices (k_xs.cu): per use (the
  // update's region, scale_n words each) and factor column (at the front's pivots)
  // XS_SCALE0 plus the power of two of its row of U12; per row of exps XS_NBO bits, one for
  // each of the panel's columns near the row's maximum; per use, side (A, B), group
  // (own, shared rows) and front the union of these over its rows, near_n words each,
  // from near0[front] on
  int* scale;
  int64_t scale_n;
  uint32_t* masks;
  uint32_t* near;
  int64_t near_n;
  const int64_t* near0;
};

// 2D maps over the workspace's 128-byte rows: boxes of 128 and of 64 rows, 128-byte swizzle
struct XsMaps {
  CUtensorMap m128, m64;
};
bool xs_encode(XsMaps* maps, void* base, int64_t rows);
// slices of xs_pack_rows(nb) panel rows, columns K0 .. K0 + W, W = min(nb, fs - K0), nb 64 or XS_NBO (item:
// front, a = K0, b = first row, c = 0; c = 1: the rows are the front's
// columns (U12^T: entries (K0 + k, row)), written to the B region); use: the
// region of the update that takes them
void launch_xs_pack(const DevCtx& c, const XsCtx& x, const Item* items, int n_items, int dtype, int nb, int use,
                    cudaStream_t s);
// LU, nb = XS_NBO: the powers of two that the slices of U12 are scaled by, from its 32
// columns at a time (item: front, a = K0, b = first column)
constexpr int XS_SCALE_COLS = 32;
void launch_xs_scale(const DevCtx& c, const XsCtx& x, const Item* items, int n_items, int dtype, cudaStream_t s);
// FP64 Cholesky: panel rows times the inverse of the diagonal block and, c = 1,
// their slices for an update with nb = 64 (item: front, a = k0, b = first row)
void launch_xs_trsm(const DevCtx& c, const XsCtx& x, const Item* items, int n_items, cudaStream_t s);
// C -= A B^T over 128 x tile_n tiles (item: front, a = first row, b = first
// column, c = K0 of the packed columns, W = min(nb, fs - K0)); lower: B is A
// and only entries col <= row are updated.  region as for k_tile_update: 0
// every entry, 1 columns below the outer panel's end, 2 rows below it; cap:
// CTAs (0: one per SM)
void launch_xs_update(const DevCtx& c, const XsCtx& x, const XsMaps& maps, const Item* items, int n_items,
                      int dtype, int nb, int region, int lower, int tile_n, int cap, int* err, cudaStream_t s);

}  // namespace uhm_gpu
