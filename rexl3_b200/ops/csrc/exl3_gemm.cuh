// The persistent EXL3 GEMM of exl3_gemm_grouped.cu, as the entry points of the other EXL3 GEMMs call it.
#pragma once
#include <cuda_runtime.h>

namespace rx {

// Whether gemm_persistent takes the product: widths with a column decoder (twice the bits: 6 or 8), up to 128 rows a tile or 256 without splits, splits of 128 k and more.
bool gemm_persistent_takes(int K, int twice, int splits, int brows);

// part[split][row][n]; `cut`: K is split at multiples of 64 or 128.  tile_tab: device int32 [max_tiles][3] = {expert, first row, rows}, nullptr: the
// max_tiles row tiles of a plain product.
int gemm_persistent(const void* xs, int rows, int K, const void* trellis, size_t expert_words, int N, int twice, int codebook, void* part, int splits, int cut,
                    const int* tile_tab, int max_tiles, int brows, int* status, cudaStream_t st);

}  // namespace rx
