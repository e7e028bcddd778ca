// The engine's weight matrices (engine.cu) as the loader (model_load.cu) fills them.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "../../include/fnx_b200.h"

namespace fnxb {
// fills matrix `index` of the engine's tensor `name` (stacked expert tensors hold several) from its GGML blocks in device memory, in
// whichever layout the tensor is held
int engine_put_matrix(fnx_engine* e, const std::string& name, int index, size_t rows, size_t cols, const uint8_t* ggml, cudaStream_t st);
}  // namespace fnxb
