// Host interface of the small-window kernel (hdb_small.cu).
#pragma once
#include <cuda_runtime.h>

#include "hdb_args.h"

namespace hdb {

// Whether windows of n points and D dims, among `windows` of a batch on `sms` SMs,
// belong to the kernel (unit_core: min_samples <= 2).
bool small_window(int precision, int n, int D, bool unit_core, int windows, int sms);

// Raises the dynamic shared-memory limit for windows of up to nmax points.
cudaError_t small_prepare(int precision, int nmax);

// One CTA for each of the `windows` windows of f.queue, at most nmax points each.
cudaError_t small_launch(int precision, const ForwardArgs& f, const SmallArgs& s, int windows, int nmax,
                         cudaStream_t stream, int priority);

}  // namespace hdb
