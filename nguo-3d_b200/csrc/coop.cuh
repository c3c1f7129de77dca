// Cooperative launches that a device or its current share of SMs cannot take.
#pragma once
#include <cuda_runtime_api.h>

namespace mg {

// Whether a cooperative launch was refused because its grid cannot be resident at once (an MPS client's
// or a partition's share of the SMs is smaller than the device's count): nothing ran, and another
// path can still solve the system. Other errors are the context's.
inline bool coop_refused(cudaError_t e) {
  return e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources || e == cudaErrorNotSupported;
}

}  // namespace mg
