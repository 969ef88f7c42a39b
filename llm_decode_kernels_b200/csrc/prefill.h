// Shared by the kernels of the prompt path.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace b200 {

// Tensor map of activations X fp16 [T, K]: boxes of 64 columns x box_rows tokens, 128-byte swizzle, zeros past T. False if the
// driver refuses (alignment).
bool encode_activation_map(CUtensorMap* map, const void* X, int T, int K, int box_rows);

}  // namespace b200
