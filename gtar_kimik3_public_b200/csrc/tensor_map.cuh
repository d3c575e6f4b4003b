// Tensor maps of bfloat16 matrices for TMA loads.
#pragma once

#include <cuda.h>

#include "common.cuh"

// A K-major matrix [rows, k] with `ld` elements between rows, in boxes of box_rows x box_k; `swizzle`: boxes of 64 entries a row in the
// 128-byte swizzle, else as they lie in memory.  The base, the rows' distance and a box's rows are multiples of 16 bytes.
int gk_matrix_map(CUtensorMap* map, const void* base, long long rows, int k, long long ld, int box_k, int box_rows, bool swizzle);
