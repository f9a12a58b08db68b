// Producer stage: encoder embeddings in bfloat16 / float16 (or the compute
// type) to the compute type, optionally L2-normalised per point, in one pass.
//
// No reference counterpart: the reference takes float32/float64 input only
// (hdbscan_gpu/_cuda.py:95-97 casts on the host side of CuPy).  Conversion
// from bfloat16/float16 to float32 is exact.  Normalisation is defined
// exactly: s = 0; for k in 0..D-1: s = s + x_k*x_k (round-to-nearest, no
// FMA); r = sqrt_rn(s); x_k' = x_k / r (round-to-nearest); a zero vector is
// left as it is (as scikit-learn's normalize does).  The
// result goes to the workspace and every later stage reads it, so the
// normalisation is computed once per point rather than once per distance tile.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "hdb_common.cuh"

namespace hdb {

enum InputType : int { kInputCompute = 0, kInputBF16 = 1, kInputF16 = 2 };

template <typename Real, typename In>
__device__ __forceinline__ Real to_compute(In v) {
    if constexpr (std::is_same<In, __nv_bfloat16>::value) return (Real)__bfloat162float(v);
    else if constexpr (std::is_same<In, __half>::value) return (Real)__half2float(v);
    else return (Real)v;
}

constexpr int kPreparePoints = 32;   // points per CTA
constexpr int kPrepareChunk = 128;   // coordinates staged at a time

// A point's sum of squares is one serial chain, so a warp holds 32 of them side
// by side; its operands come through shared memory, where every global load
// and store is coalesced.  Memory-bound apart from the chains.  (One thread a
// point straight from global memory read 32 rows with every load: 392 us for
// 47,952 x 384 bfloat16 values.)
template <typename Real, typename In>
__global__ void __launch_bounds__(256) hdb_prepare_kernel(const In* __restrict__ X, Real* __restrict__ out,
                                                          int64_t points, int D, int normalize) {
    using T = RealTraits<Real>;
    __shared__ Real s_x[kPreparePoints][kPrepareChunk + 1];
    __shared__ Real s_norm[kPreparePoints];
    const int64_t i0 = (int64_t)blockIdx.x * kPreparePoints;
    const int rows = (int)(points - i0 < kPreparePoints ? points - i0 : kPreparePoints);
    const In* x = X + i0 * D;
    Real* y = out + i0 * D;
    const int64_t total = (int64_t)rows * D;
    if (!normalize) {
        for (int64_t t = threadIdx.x; t < total; t += 256) y[t] = to_compute<Real>(x[t]);
        return;
    }
    Real s = Real(0);
    for (int k0 = 0; k0 < D; k0 += kPrepareChunk) {
        const int width = D - k0 < kPrepareChunk ? D - k0 : kPrepareChunk;
        for (int r = threadIdx.x / kPrepareChunk; r < rows; r += 256 / kPrepareChunk) {
            const int k = threadIdx.x % kPrepareChunk;
            if (k < width) s_x[r][k] = to_compute<Real>(x[(int64_t)r * D + k0 + k]);
        }
        __syncthreads();
        if ((int)threadIdx.x < rows) {
#pragma unroll 8
            for (int k = 0; k < width; ++k) {
                const Real v = s_x[threadIdx.x][k];
                s = T::add(s, T::mul(v, v));
            }
        }
        __syncthreads();
    }
    if ((int)threadIdx.x < rows) s_norm[threadIdx.x] = T::sqrt_rn(s);
    __syncthreads();
    for (int r = threadIdx.x >> 5; r < rows; r += 8) {
        const Real norm = s_norm[r];
        for (int k = threadIdx.x & 31; k < D; k += 32) {
            const Real v = to_compute<Real>(x[(int64_t)r * D + k]);
            y[(int64_t)r * D + k] = norm > Real(0) ? T::div(v, norm) : v;
        }
    }
}

}  // namespace hdb
