// The driver's tensor-map encoder, looked up at run time so that the library has no link-time dependency on libcuda.
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>

namespace b200q {

// nullptr when the driver does not have it.
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder();

}  // namespace b200q
