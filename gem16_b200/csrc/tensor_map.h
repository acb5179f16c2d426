// Internal: tensor maps for TMA, encoded by the driver (gemm.cu).
#pragma once

#include <cuda.h>

#include <cstdint>

namespace gemb {

// Byte matrix [rows, row_bytes] row-major -> tiles of 128 bytes x box_rows rows, 128-byte swizzle.
int32_t make_byte_map(const char* op, CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes, uint32_t box_rows);
// Matrix [rows, cols] of words of two or four bytes, row-major -> tiles of box_cols x box_rows; with the 128-byte swizzle (box_cols
// words are 128 bytes then) or as they lie.
int32_t make_word_map(const char* op, CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint32_t word_bytes, uint32_t box_cols,
                      uint32_t box_rows, bool swizzle);

}  // namespace gemb
