// host_stage.h -- copies between the caller's arrays and the device, and the
// finite test of a caller's arrays.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <initializer_list>
#include <memory>
#include <utility>

namespace b200fem {

// true when every value is finite: a NaN or an infinity in a caller's array
// is refused with B200FEM_ERR_INVALID_ARG before it reaches the device
bool all_finite(const double* a, size_t n);
// The same of several arrays (null: none), large ones by several threads.
bool all_finite_arrays(std::initializer_list<std::pair<const double*, size_t>> arrays);

struct HostStage;

// One array of a host copy (host null: none).
struct HostCopy {
  void* host;
  void* dev;
  size_t bytes;
};

// Copies between host arrays and the device, ordered behind the work on
// `stream`.  Staged copies are complete on return, others are asynchronous on
// `stream`: the caller synchronises it before it reads.  `stage`: the
// engine's hold on the device's stage, made on the first staged copy.
cudaError_t stage_copy(int device, cudaStream_t stream, std::shared_ptr<HostStage>& stage,
                       std::initializer_list<HostCopy> list, bool to_host);

}  // namespace b200fem
