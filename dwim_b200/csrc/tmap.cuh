// Tensor maps (gemm.cu holds the encoder).
#pragma once
#include <cuda.h>
#include "common.cuh"

namespace dwim {
int encode_nd(dwim_b200_ctx *ctx, CUtensorMap *map, CUtensorMapDataType type, const void *ptr, int rank, const uint64_t *dims,
              const uint64_t *pitches, const uint32_t *box, CUtensorMapSwizzle swizzle, const char *what);
int encode_2d(dwim_b200_ctx *ctx, CUtensorMap *map, CUtensorMapDataType type, const void *ptr, uint64_t inner, uint64_t outer,
              uint64_t pitch_bytes, uint32_t box_inner, uint32_t box_outer, CUtensorMapSwizzle swizzle, const char *what);
}  // namespace dwim
