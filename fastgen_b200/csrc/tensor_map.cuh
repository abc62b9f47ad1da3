// Tensor maps (TMA descriptors), encoded by the driver's function, which is looked up at run time.
#pragma once

#include <cuda.h>

#include "common.cuh"

// A map of `rank` dimensions over `base` with a 128-byte swizzle and a 128-byte promotion in L2; elements beyond the
// tensor read as zeros.  Returns 0, or stores a message and returns a negative code.
int fg_encode_tensor_map(CUtensorMap* map, CUtensorMapDataType type, int rank, const void* base, const cuuint64_t* dims,
                         const cuuint64_t* strides, const cuuint32_t* box);
