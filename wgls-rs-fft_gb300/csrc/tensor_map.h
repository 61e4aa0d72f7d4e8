// The CUDA driver's tensor-map encoder, looked up through the runtime.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>

namespace gbfft {

// Null where the driver does not provide it.
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder();

}  // namespace gbfft
