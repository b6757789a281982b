// What the bindings of the model-side kernels share (binding_ops.cpp).
#pragma once

#include <ATen/core/Tensor.h>
#include <c10/util/Optional.h>
#include <cuda_runtime_api.h>

#include <cstdint>

namespace hvd {

// Throws unless t is 4-D, 16-bit, on a GPU and contiguous in channels_last.
void CheckActivations(const at::Tensor& t, const char* what);
// t, checked, or a copy of it that starts on a 16-byte boundary.
at::Tensor Activations(const at::Tensor& t, const char* what);
const float* FloatPtrOrNull(const c10::optional<at::Tensor>& t, int64_t channels,
                            const char* what);
// `count` doubles that are zero when the next kernel of the stream runs. `own` has to
// live until the last kernel that uses them is launched; until then no other request
// clears them.
double* ZeroedDoubles(int64_t count, const at::Tensor& like, cudaStream_t stream,
                      at::Tensor* own);

}  // namespace hvd
