// Host interface of the sparse path (hdb_sparse.cu): one launcher per stage.
#pragma once
#include <cuda_runtime.h>

#include "hdb_args.h"

namespace hdb {

enum class SparseStage { kNarrow, kTiles, kRows, kCore, kForest, kBetween, kTree, kLight, kStar, kWeights, kPrim };

// Launches `stage` for the windows of `a`; `f` is the forward's argument block
// (kPrim only).  precision: 0 float32, 1 float64 (kNarrow, kCore and kWeights
// belong to bounded distances, SparseArgs::approx).
cudaError_t sparse_launch(int precision, SparseStage stage, const SparseArgs& a, const ForwardArgs* f,
                          cudaStream_t stream, int priority);

// Raises the dynamic shared-memory limits for windows of up to n points; false
// in *fits when a window of that size does not fit in `budget` bytes.
cudaError_t sparse_prepare(int precision, int n, size_t budget, bool* fits);

// Whether windows of D dims take tensor-core products.
bool sparse_gram(int D);

// Whether the bound of the distances holds for windows of D dims.
bool sparse_dims(bool approx, int D);

// Row stride of the neighbour lists for min_samples ms (0: not supported) and
// the entries used of them.
int sparse_list(bool approx, bool gram, int ms, int* keep);

}  // namespace hdb
