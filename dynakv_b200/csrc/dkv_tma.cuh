// Tensor maps for the TMA-fed tcgen05 kernels.
#pragma once

#include <cuda.h>
#include <stdint.h>

namespace dkv {

// [rows, cols] 16-bit matrix with a row pitch in elements, boxes of 64 columns x box_rows rows in the 128-byte swizzle;
// false when the driver does not export the encoder or refuses the map (implemented in dkv_project.cu)
bool tensor_map_16bit(CUtensorMap* m, int dtype, const void* base, uint64_t rows, uint64_t cols, uint64_t pitch, uint32_t box_rows);

}  // namespace dkv
