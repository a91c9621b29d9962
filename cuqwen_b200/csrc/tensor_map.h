// Tensor maps of weight matrices (kernels.cu).
#pragma once
#include <cuda.h>
#include <stddef.h>

namespace cq {

// Byte-typed 4-D map of `layers` equal row-major matrices, layer_stride bytes apart, each seen as [rows][64-byte chunks]: a box of box_rows rows x piece_bytes of one
// of them lands in shared memory chunk-major; rows and chunks beyond the matrix arrive as zeros.
int encode_layer_map(CUtensorMap* m, const void* w, size_t row_bytes, size_t rows, int layers, size_t layer_stride, int piece_bytes, int box_rows);

// Map of `rows` fp16 cache rows of hd values (64 or 128): a box of `keys` rows lands as hd / 64 blocks [key][64 values], 128-byte swizzled.
int encode_cache_map(CUtensorMap* m, const void* cache, size_t rows, int hd, int keys);

}  // namespace cq
