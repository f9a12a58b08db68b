// Launchers of the sparse path (hdb_sparse.cuh).
#include "hdb_sparse.h"

#include "hdb_launch.h"
#include "hdb_registry.h"
#include "hdb_sparse.cuh"

namespace hdb {
namespace {

// Threads of the one-CTA-a-window kernels.
int window_threads(int nmax) { return nmax <= 128 ? 64 : (nmax <= 512 ? 128 : (nmax <= 1024 ? 256 : 512)); }

unsigned blocks(int n, int per) { return (unsigned)((n + per - 1) / per); }

template <typename Real>
cudaError_t launch_rows(const SparseArgs& a, cudaStream_t s, int priority) {
    const unsigned grid = (unsigned)a.n_windows * blocks(a.nmax, kSparseRowsCta);
    const unsigned threads = 32 * kCoreRowsWarps;
    if (a.gram && a.list <= 32) return launch_ex(hdb_sparse_gram_rows_kernel<Real>, grid, threads, 0, s, priority, 1, a);
    switch (a.list) {
        case 8: return launch_ex(hdb_sparse_rows_kernel<Real, 8>, grid, threads, 0, s, priority, 1, a);
        case 16: return launch_ex(hdb_sparse_rows_kernel<Real, 16>, grid, threads, 0, s, priority, 1, a);
        case 32: return launch_ex(hdb_sparse_rows_kernel<Real, 32>, grid, threads, 0, s, priority, 1, a);
        default: return launch_ex(hdb_sparse_rows_kernel<Real, 64>, grid, threads, 0, s, priority, 1, a);
    }
}

template <typename Real>
cudaError_t launch_stage(SparseStage stage, const SparseArgs& a, const ForwardArgs* f, cudaStream_t s, int priority) {
    const unsigned W = (unsigned)a.n_windows;
    switch (stage) {
        case SparseStage::kRows:
            return launch_rows<Real>(a, s, priority);
        case SparseStage::kTiles: {
            const unsigned t = blocks(a.nmax, 128);
            if (a.gram)
                return launch_ex(hdb_sparse_gram_kernel<Real>, W * (t * (t + 1) / 2), 256, 2 * kGramStage, s, priority, 1, a);
            return launch_ex(hdb_sparse_tiles_kernel<Real>, W * (t * (t + 1) / 2), 256, 0, s, priority, 1, a);
        }
        case SparseStage::kForest:
            return launch_ex(hdb_sparse_forest_kernel<Real>, W, (unsigned)window_threads(a.nmax),
                             sparse_forest_smem(a.nmax), s, priority, 1, a);
        case SparseStage::kBetween:
            return launch_ex(hdb_sparse_between_kernel<Real>, W * blocks(a.nmax, kBetweenRows), 256,
                             sparse_between_smem(a.nmax), s, priority, 1, a);
        case SparseStage::kTree:
            return launch_ex(hdb_sparse_tree_kernel<Real>, W, (unsigned)window_threads(a.nmax), sparse_tree_smem(a.nmax),
                             s, priority, 1, a);
        case SparseStage::kLight:
            return launch_ex(hdb_sparse_light_kernel<Real>, W * blocks(a.nmax, kLightRows), 256,
                             (size_t)sparse_round(a.nmax) * sizeof(float), s, priority, 1, a);
        case SparseStage::kStar:
            return launch_ex(hdb_sparse_star_kernel<Real>, W * blocks(a.nmax, kSparseRowsCta), 256, 0, s, priority, 1, a);
        case SparseStage::kPrim:
            return launch_ex(hdb_sparse_prim_kernel<Real>, W, (unsigned)window_threads(a.nmax),
                             SparsePrimLayout<Real>::bytes(a.nmax), s, priority, 1, a, *f);
        default:
            break;
    }
    switch (stage) {
        case SparseStage::kNarrow:
            if (a.gram)
                return launch_ex(hdb_sparse_split_kernel<Real>, W * blocks(a.nmax, kSplitRows), 256, 0, s, priority, 1, a);
            if constexpr (sizeof(Real) == 8)
                return launch_ex(hdb_sparse_narrow_kernel, W * blocks(a.nmax, kNarrowRows), 256, 0, s, priority, 1, a);
            break;
        case SparseStage::kCore:
            return launch_ex(hdb_sparse_core_kernel<Real>, W * blocks(a.nmax, 128), 128, 0, s, priority, 1, a);
        case SparseStage::kWeights:
            return launch_ex(hdb_sparse_weights_kernel<Real>, W * kWeightsPerWindow, 128, 0, s, priority, 1, a);
        default:
            break;
    }
    return cudaErrorInvalidValue;
}

template <typename Real>
cudaError_t prepare(int n, size_t budget, bool* fits) {
    const size_t need[5] = {2 * kGramStage, sparse_forest_smem(n), sparse_between_smem(n), sparse_tree_smem(n),
                            SparsePrimLayout<Real>::bytes(n)};
    const void* func[5] = {(const void*)hdb_sparse_gram_kernel<Real>,
                           (const void*)hdb_sparse_forest_kernel<Real>, (const void*)hdb_sparse_between_kernel<Real>,
                           (const void*)hdb_sparse_tree_kernel<Real>,
                           (const void*)hdb_sparse_prim_kernel<Real>};
    *fits = true;
    for (int i = 0; i < 5; ++i) {
        cudaFuncAttributes attr;
        cudaError_t e = cudaFuncGetAttributes(&attr, func[i]);
        if (e != cudaSuccess) return e;
        if (need[i] + attr.sharedSizeBytes + 1024 > budget) { *fits = false; return cudaSuccess; }
        e = raise_dynamic_smem(func[i], need[i]);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace

cudaError_t sparse_launch(int precision, SparseStage stage, const SparseArgs& a, const ForwardArgs* f,
                          cudaStream_t stream, int priority) {
    return precision == 0 ? launch_stage<float>(stage, a, f, stream, priority)
                          : launch_stage<double>(stage, a, f, stream, priority);
}

cudaError_t sparse_prepare(int precision, int n, size_t budget, bool* fits) {
    return precision == 0 ? prepare<float>(n, budget, fits) : prepare<double>(n, budget, fits);
}

bool sparse_gram(int D) { return D >= kGramMinDims && D <= kGramMaxDims; }

bool sparse_dims(bool approx, int D) { return !approx || D <= kNarrowMaxDims; }

int sparse_list(bool approx, bool gram, int ms, int* keep) {
    // Entries past position ms - 1 show where the star ends and bound the
    // uncertain range, which is wider for products.
    const int want = ms <= 2 ? 8 : (gram ? ms + ms / 4 + 10 : (approx ? ms + 3 : ms + 1));
    const int need = ms <= 2 ? 8 : (gram ? ms + 6 : (approx ? ms + 2 : ms + 1));
    for (int k : {8, 16, 32, 64})
        if (want <= k || (need <= k && k == 64)) {
            *keep = ms <= 2 ? 8 : (want < k ? (want < 8 ? 8 : want) : k);
            return k;
        }
    return 0;
}

}  // namespace hdb
