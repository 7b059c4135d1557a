// Tensor maps for TMA loads of matrix operands.
#pragma once
#include <cuda.h>

#include <cstdint>

namespace b200 {

// rows of k 16-bit elements ld apart (base and ld * 2 multiples of 16 bytes), in boxes of 64 elements x box_rows with the 128-byte
// swizzle; what lies outside reads as zero.  Defined in gemm_bf16_tcgen05.cu
int rows_map(CUtensorMap *map, CUtensorMapDataType type, const void *base, int64_t k, int64_t rows, int64_t ld, int box_rows);
// a cache of n_pos positions x heads x d 16-bit floats (nb1 bytes from position to position, nb2 from head to head, both and the base
// multiples of 16), in boxes of 64 elements x box_pos positions of one head with the 128-byte swizzle.  false: refused by the driver
bool cache_tile_map(CUtensorMap *map, const void *base, int64_t d, int64_t heads, int64_t n_pos, int64_t nb1, int64_t nb2, int box_pos);

}  // namespace b200
