// Byte geometry of NVFP4 tensors (E2M1 codes two per byte, one E4M3 scale per 16 values - or a 4-bit index into a table of 16 -
// and one FP32 scale per tensor).
#pragma once

#include <stdint.h>

namespace nvfp4 {

__host__ __device__ inline uint64_t align256(uint64_t v) { return (v + 255ull) & ~255ull; }

// Byte geometry of a tensor (tools/euhedral_artifacts/nvfp4.py:49-57; native/src/host/nvfp4_linear.c:79-91).
struct Geometry {
    uint64_t row_bytes, row_scales, scale_row_bytes, scale_offset, global_offset, size;
    __host__ __device__ Geometry(uint32_t rows, uint32_t k) {
        const uint64_t kp = ((uint64_t)k + 127u) / 128u * 128u;
        row_bytes = kp / 2u;
        row_scales = scale_row_bytes = kp / 16u;
        scale_offset = align256((uint64_t)rows * row_bytes);
        global_offset = align256(scale_offset + (uint64_t)rows * row_scales);
        size = global_offset + 4u;
    }
};

// Byte geometry of a tensor whose block scales are 4-bit indices into a table of 16 E4M3 codes (layout
// row-split-k128-sd4-v1, tools/euhedral_artifacts/nvfp4.py:60-69): the index plane is half the scale plane (two indices
// per byte, the even block in the low nibble), then the table, then the FP32 tensor scale.
struct GeometrySd4 {
    uint64_t row_bytes, scale_row_bytes, scale_offset, table_offset, global_offset, size;
    __host__ __device__ GeometrySd4(uint32_t rows, uint32_t k) {
        const uint64_t kp = ((uint64_t)k + 127u) / 128u * 128u;
        row_bytes = kp / 2u;
        scale_row_bytes = kp / 32u;
        scale_offset = align256((uint64_t)rows * row_bytes);
        table_offset = align256(scale_offset + (uint64_t)rows * scale_row_bytes);
        global_offset = table_offset + 16u;
        size = table_offset + 20u;
    }
};

}  // namespace nvfp4
