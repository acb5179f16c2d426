// Internal: tensor maps for TMA, encoded by the driver (gemm.cu).
#pragma once

#include <cuda.h>

#include <cstdint>

namespace gemb {

// Byte matrix [rows, row_bytes] row-major -> tiles of 128 bytes x box_rows rows, 128-byte swizzle.
int32_t make_byte_map(const char* op, CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes, uint32_t box_rows);

}  // namespace gemb
