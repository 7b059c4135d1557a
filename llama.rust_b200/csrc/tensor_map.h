// Tensor maps for TMA loads of matrix operands.
#pragma once
#include <cuda.h>

#include <cstdint>

namespace b200 {

// rows of k 16-bit elements ld apart (base and ld * 2 multiples of 16 bytes), in boxes of 64 elements x box_rows with the 128-byte
// swizzle; what lies outside reads as zero.  Defined in gemm_bf16_tcgen05.cu
int rows_map(CUtensorMap *map, CUtensorMapDataType type, const void *base, int64_t k, int64_t rows, int64_t ld, int box_rows);

}  // namespace b200
