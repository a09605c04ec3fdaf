// Tensor-core (tcgen05) Schur update: operand maps and launchers.
#pragma once
#include <cuda.h>
#include <cstdint>
#include "kernels.cuh"

namespace uhm_gpu {

constexpr int TC_NBO = 256;   // default outer panel width of fronts updated on tensor cores

bool tc_encode_part(CUtensorMap* map, void* base, int64_t rows, int nbo);
// trans = 0: the panel rows below the outer panel (A operand, parts poff..);
// trans = 1: the LU panel's U block right of it, transposed (B operand)
void launch_tc_pack(const DevCtx& c, const Item* items, int n_items, int nbo, int nparts, void* ws,
                    const int64_t* ws_off, const int64_t* ws_stride, int trans, int poff, cudaStream_t s);
// C -= A B^T, operands in BF16 parts: A 0 .. parts - 1, B pb0 .. pb0 + parts - 1, the
// terms p + q < parts; cap: CTAs (0: one per SM)
void launch_tc_syrk(const DevCtx& c, const CUtensorMap& wsmap, const int64_t* ws_off,
                    const int64_t* ws_stride, const Item* items, int n_items, int nbo, int parts, int pb0,
                    int lower_only, int cap, int* err, cudaStream_t s);
int tc_tile();

}  // namespace uhm_gpu
