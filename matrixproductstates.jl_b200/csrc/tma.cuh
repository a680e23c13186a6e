// Access to the driver's tensor map encoder.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>

namespace mpsb {
// cuTensorMapEncodeTiled, looked up once per process; null when the driver does not have it
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder();
}  // namespace mpsb
