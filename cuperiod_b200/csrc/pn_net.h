// What the proposal network's translation units share (host side).
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

namespace blsb200 {
namespace pn {

// cuTensorMapEncodeTiled, once load_encode() has returned cudaSuccess.
extern PFN_cuTensorMapEncodeTiled_v12000 g_encode;
cudaError_t load_encode();

}  // namespace pn
}  // namespace blsb200
