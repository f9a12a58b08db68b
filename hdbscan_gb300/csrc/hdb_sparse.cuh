// Sparse path: the exact minimum spanning tree without a dense Prim loop.
//
// Prim over the dense graph is a serial chain of n-1 row reads and block-wide
// argmins (matrix variant, float32: 1.0 us a step at 2048 points, 1.4 us at
// 4096), and float64 distances are bound by the FP64 pipe.  Both go away once
// the few edges that can matter are known:
//   1. a spanning tree T', minimal up to roundings, is built from each point's
//      nearest neighbours by rounds of component merging (Boruvka), and from one
//      pass over the distances between the components whose lists are used up;
//   2. an edge heavier than the largest edge on the T' path between its ends
//      lies in no minimum spanning tree (the filter of Karger, Klein and
//      Tarjan 1995), so one pass over all pairs keeps only the light ones.  The
//      path maximum comes from the merge rounds alone: the tree whose nodes are
//      the components of every round, with the edge each component chose as the
//      weight to its parent, has the same path maxima as T' (King 1997);
//   3. Prim's vertex order follows from the light edges: every edge of minimal
//      weight across any cut is light, so each step sees the same minimum and
//      the same lowest vertex of that weight as over the dense graph.  A
//      vertex's source (strict '<' keeps the older one) is then the first
//      visited end of its light edges of that weight.
//
// Most light edges are ties: max(core_x, core_u, d) = core_x for every point u
// among x's ms nearest with a smaller core (x's star).  They need no distance,
// they are in the neighbour lists, and one of them for each component that the
// star touches below core_x is enough for the order (hdb_sparse_star_kernel).
//
// float64 windows and wide float32 ones: the pass over all pairs and the
// neighbour lists use float32 distances with a proven bound (sparse_bound), for
// wide points from tensor-core products; every comparison that decides something
// takes the safe side, and all weights, core distances and ties come from exact
// arithmetic in the window's own precision on the few pairs that remain.
// float32 windows of few dims: the distance blocks are exact, the bounds zero.
//
// A window that does not fit (more light edges than the workspace holds, as
// with many equal distances; neighbours that the bound cannot tell apart;
// values outside the range of the bound; infinite distances) sets its flag and
// takes the general path, whose kernels look at the flags.
#pragma once
#include "hdb_common.cuh"
#include "hdb_distance.cuh"
#include "hdb_forward.cuh"
#include "hdb_tree_cta.cuh"
#include <cuda_bf16.h>

namespace hdb {

constexpr int kSparseRowsCta = 32;   // rows per CTA of the neighbour kernel
constexpr int kLightRows = 16;       // rows per CTA of the light-edge kernel

__device__ __forceinline__ void sparse_flag(const SparseArgs& a, int w) {
    a.flags[w] = a.stage;
    a.flags[a.n_flags + a.stage - 1] = 1;
}

// The window's float32 distance block: its own block (float32), or the first
// half of the float64 block's place (the general path overwrites it later).
template <typename Real>
__device__ __forceinline__ float* sparse_block(const SparseArgs& a, int w) {
    return reinterpret_cast<float*>(static_cast<Real*>(a.dist) + a.dist_offsets[w]);
}

// Bound between a float32 distance d~ and the float64 one, d:
// |d~ - d| <= shift + d~ * scale.  Inputs are y = RN32(x - x0), R >= |x - x0|
// for every coordinate of the window:
//   * each coordinate difference is off by at most 2^-23 R from the two
//     roundings of y, so the difference vector is off by sqrt(D) 2^-23 R;
//   * the float32 difference, its square, the D-term sum (any order, fused or
//     not) and the root add a relative (D/2 + 3) 2^-24 to first order.
// Both are taken 5% larger (plus some units) than that, which covers second
// order terms, the float64 arithmetic's own rounding and the evaluation of the
// bound itself.
//
// Products (D >= kGramMinDims): the block holds a lower bound of the squared
// distance, n_i + n_j - 2 z_i.z_j - eta (n_i + n_j) with the centred points z as
// sums of two bfloat16 parts (see sparse_eta), and the true value lies at most
// 2 eta (n_i + n_j) above it.  What decides ranks and weights is not the true
// value but the window's own arithmetic on it (sparse_exact), which adds its
// share of the square itself (sparse_chain), on both sides.  Core distances and all
// weights of the kernels below are then squares as well; exact values stay plain
// distances.
struct SparseBound {
    float up_shift, up_scale, down_shift, down_scale;
    float eta;  // products
    __device__ __forceinline__ float up(float d) const { return __fmaf_ru(d, up_scale, up_shift); }
    __device__ __forceinline__ float down(float d) const { return __fmaf_rd(d, down_scale, down_shift); }
};

// Bound of |s~ - d^2| / (n_i + n_j) for s~ = n_i + n_j - 2 g, all in float32:
//   * z = hi + lo + e; hi.hi + hi.lo + lo.hi leaves out lo.lo and the products with e:
//     (l^2 + 2 e) |z_i||z_j| with l = |lo| / |z| and e = |e| / |z|.  bfloat16 has 8
//     significant bits, so l <= 2^-8 and e <= 2^-17 (3.1e-5 in all); over the
//     coordinates of a point they average to a third of that, and the window's largest
//     of each, measured as the points are split, are taken;
//   * each matrix instruction adds 16 exact products to its accumulator; 2^-20 of
//     the running magnitude a step allows for every operand being cut off at 24
//     bits below the largest (its rounding is not specified).  The accumulator
//     starts anew every 32 coordinates, six steps, so these errors are six shares
//     of the parts' |z_i||z_j|, whose sum is at most the whole's;
//   * the parts' sum, the norms' sums, z's own rounding to float32 and the last
//     operations: (D / 8 + 32) 2^-24.
// 2 |z_i||z_j| <= n_i + n_j turns the products' shares into shares of n_i + n_j;
// 10% on top covers second order terms.
__device__ __forceinline__ float sparse_eta(const SparseArgs& a, int w) {
    const float split = __uint_as_float(a.split_share[w]) + 2.0f * sqrtf(__uint_as_float(a.split_share[a.n_flags + w]));
    return 1.1f * (split + 6.0f * 9.5367432e-7f + (float)(a.D / 8 + 32) * 5.9604645e-8f);
}

// Largest relative difference between the square of sparse_exact's value and the
// true square.  float32: two roundings of a coordinate's difference and one of its
// square in each term, one of each of the D - 1 sums, two of the root (squared), and
// the squares of core distances taken up and down: D + 8 units of 2^-24; 5% covers
// second order terms.  float64: D + 8 units of 2^-53, below a float32 unit at all
// D that take products; sparse_eta's 10% covers it.
template <typename Real>
__device__ __forceinline__ float sparse_chain(int D) {
    return sizeof(Real) == 4 ? 1.05f * (float)(D + 8) * 5.9604645e-8f : 0.0f;
}

template <typename Real>
__device__ __forceinline__ SparseBound sparse_bound(const SparseArgs& a, int w) {
    if (!a.approx) return SparseBound{0.0f, 1.0f, 0.0f, 1.0f, 0.0f};
    const float R = __uint_as_float(a.range[w]);
    if (a.gram) {
        // (4.2 instead of 4: the sums' and the chain's share of the shift itself.)
        const float chain = sparse_chain<Real>(a.D), eta = sparse_eta(a, w);
        return SparseBound{4.2f * eta * R, __fadd_ru(1.0000005f, chain), 0.0f, __fadd_rd(1.0f, -chain), eta};
    }
    const float shift = 1.05f * sqrtf((float)a.D) * 1.1920929e-7f * R;
    const float scale = 1.05f * (0.5f * (float)a.D + 8.0f) * 5.9604645e-8f;
    return SparseBound{shift, __fadd_ru(1.0f, scale), -shift, __fadd_rd(1.0f, -scale), 0.0f};
}

// Exact distance of two rows in the reference's order (k-ordered sum).
template <typename Real>
__device__ __forceinline__ Real sparse_exact(const Real* __restrict__ xa, const Real* __restrict__ xb, int D) {
    using T = RealTraits<Real>;
    Real acc = Real(0);
    int k = 0;
    for (; k + 8 <= D; k += 8) {
        Real p[8], q[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) { p[j] = xa[k + j]; q[j] = xb[k + j]; }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const Real delta = T::sub(p[j], q[j]);
            acc = T::add(acc, T::mul(delta, delta));
        }
    }
    for (; k < D; ++k) {
        const Real delta = T::sub(xa[k], xb[k]);
        acc = T::add(acc, T::mul(delta, delta));
    }
    return T::sqrt_rn(acc);
}

// ---------------------------------------------------------------------------
// float64 input -> float32 around the window's first point, with the window's
// range.  One CTA per 64 rows; non-finite values and ranges outside
// [2^-40, 2^40] (the bound assumes no overflow or underflow in float32) flag
// the window.
// ---------------------------------------------------------------------------
constexpr int kNarrowRows = 64;
// The bound's relative part is of first order in D * 2^-24 (5% on top covers the rest
// up to about 2 million dims), and a CTA's share of the input is counted in 32 bits
// (up to 2^25 dims): wider points keep the general path, far below both.
constexpr int kNarrowMaxDims = 1 << 16;

__global__ void __launch_bounds__(256) hdb_sparse_narrow_kernel(const SparseArgs a) {
    const int per = (a.nmax + kNarrowRows - 1) / kNarrowRows;
    const int item = blockIdx.x / per, r0 = (blockIdx.x - item * per) * kNarrowRows;
    const int w = a.queue[item];
    const int64_t base = a.offsets[w];
    const int n = (int)(a.offsets[w + 1] - base);
    if (r0 >= n) return;
    const int D = a.D;
    const int rows = min(kNarrowRows, n - r0);
    const double* __restrict__ X = static_cast<const double*>(a.X) + base * D;
    float* __restrict__ y = a.y + (base + r0) * D;
    const double* __restrict__ x = X + (int64_t)r0 * D;
    uint32_t top = 0;
    bool bad = false;
    for (int i = threadIdx.x; i < rows * D; i += 256) {
        const double v = x[i];
        const double c = v - X[i % D];
        const uint32_t mag = __float_as_uint(__double2float_ru(fabs(c)));  // NaN and infinity rank highest
        bad |= ((uint32_t)__double2hiint(v) & 0x7ff00000u) == 0x7ff00000u;
        top = max(top, mag & 0x7fffffffu);
        y[i] = (float)c;
    }
    top = __reduce_max_sync(0xffffffffu, top);
    const float R = __uint_as_float(top);
    if (bad || !(R <= 1.0995e12f)) sparse_flag(a, w);  // also tests NaN
    if ((threadIdx.x & 31) == 0) atomicMax(a.range + w, top);
}

// The same for products: points centred on the mean of kCentrePoints of the
// window's points (any centre is exact enough; a near one keeps the norms, and
// with them the bound, small), as bfloat16 pairs, and their squared norms.  One
// warp a row.
constexpr int kGramMinDims = 32;
constexpr int kGramMaxDims = 2048;   // the centre in shared memory
constexpr int kCentrePoints = 16;
constexpr int kSplitRows = 32;
// All shares of sparse_eta are relative to the norms, so products below float32's
// normal range must not count: with points of at least this squared norm (2^-90),
// up to 3 * 2048 products of less than 2^-126 are under 2^-22 of it even when each is
// lost.  A point at the centre itself has a norm of zero and exact products.
constexpr float kGramLeastNorm = 8.077936e-28f;

template <typename Real>
__global__ void __launch_bounds__(256) hdb_sparse_split_kernel(const SparseArgs a) {
    __shared__ Real s_centre[kGramMaxDims];
    const int per = (a.nmax + kSplitRows - 1) / kSplitRows;
    const int item = blockIdx.x / per, r0 = (blockIdx.x - item * per) * kSplitRows;
    const int w = a.queue[item];
    const int64_t base = a.offsets[w];
    const int n = (int)(a.offsets[w + 1] - base);
    if (r0 >= n) return;
    const int D = a.D, dims = a.dims;
    const Real* __restrict__ X = static_cast<const Real*>(a.X) + base * D;
    for (int k = threadIdx.x; k < D; k += 256) {
        // Summed in pairs: of sixteen copies of a point the mean is that point.
        Real sum[kCentrePoints];
#pragma unroll
        for (int j = 0; j < kCentrePoints; ++j) sum[j] = X[(int64_t)(j * n / kCentrePoints) * D + k];
#pragma unroll
        for (int h = kCentrePoints / 2; h > 0; h >>= 1)
#pragma unroll
            for (int j = 0; j < h; ++j) sum[j] += sum[j + h];
        s_centre[k] = sum[0] * Real(1.0 / kCentrePoints);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int r = warp; r < kSplitRows; r += 8) {
        const int i = r0 + r;
        if (i >= n) break;
        const Real* __restrict__ x = X + (int64_t)i * D;
        uint16_t* __restrict__ out = a.split + (base + i) * 2 * dims;
        float norm = 0.0f, low = 0.0f, rest = 0.0f;  // squared
        bool bad = false, off = false;
        for (int k = lane; k < dims; k += 32) {
            float z = 0.0f;
            if (k < D) {
                const Real v = x[k];
                bad |= !isfinite(v);
                off |= v != s_centre[k];
                z = (float)(v - s_centre[k]);
            }
            const __nv_bfloat16 hi = __float2bfloat16_rn(z);
            const float below = __fsub_rn(z, __bfloat162float(hi));  // exact, as is what is left of it
            const __nv_bfloat16 lo = __float2bfloat16_rn(below);
            const float left = __fsub_rn(below, __bfloat162float(lo));
            const int at = (k >> 5) * 64 + (k & 31);
            out[at] = __bfloat16_as_ushort(hi);
            out[at + 32] = __bfloat16_as_ushort(lo);
            norm = __fmaf_rn(z, z, norm);
            low = __fmaf_rn(__bfloat162float(lo), __bfloat162float(lo), low);
            rest = __fmaf_rn(left, left, rest);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            norm += __shfl_xor_sync(0xffffffffu, norm, o);
            low += __shfl_xor_sync(0xffffffffu, low, o);
            rest += __shfl_xor_sync(0xffffffffu, rest, o);
        }
        off = __any_sync(0xffffffffu, off);
        bad = __any_sync(0xffffffffu, bad) || !(norm <= 1.2e24f) || (off && norm < kGramLeastNorm);  // 2^80; also tests NaN
        if (lane == 0) {
            a.norm[base + i] = norm;
            if (bad) {
                sparse_flag(a, w);
            } else {
                atomicMax(a.range + w, __float_as_uint(norm));
                if (norm > 0.0f) {
                    atomicMax(a.split_share + w, __float_as_uint(low / norm));
                    atomicMax(a.split_share + a.n_flags + w, __float_as_uint(rest / norm));
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Lower bounds of the squared distances from tensor-core products: 128x128 tiles
// of the upper triangle, 8 warps of 32x64 pairs, three bfloat16 matrix products
// (high.high, high.low, low.high) accumulated in float32.  A row's 32
// coordinates are one 128-byte line of high and low parts; two stages of
// asynchronous copies, 16-byte chunks swizzled by row for ldmatrix.  Off-diagonal
// values are written to both halves from one accumulator, so the block is
// symmetric.  A finished tile goes out by way of shared memory, in whole lines, with
// the minima of 16 columns of each row and of 16 rows of each column: half of the
// instructions and store wavefronts of stores from the accumulators.  Floor: the
// block's own write (4 n^2 bytes) for small D; held back by two CTAs an SM (128
// registers a thread).  16 windows of 2048 points x 64 dims (268 MB): 112 us from
// the accumulators, 109 this way; ragged batch of 64..4096 points x 32 dims, whole
// call: 6.09 and 5.97 ms.
// ---------------------------------------------------------------------------
constexpr int kGramStage = 2 * 128 * 128;  // bytes of a stage: two operands of 128 rows x 128 bytes

__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Place of a finished tile's entry in shared memory: 16-byte chunks of a row are
// permuted by the row, such that stores of accumulator pairs (8 rows x 4), reads of
// rows and reads of 32 rows' chunks have no bank conflicts.
__device__ __forceinline__ int gram_at(int r, int c) {
    return (r << 7) + ((((c >> 2) ^ ((r << 1 | ((r >> 2) & 1)) & 7)) << 2) | (c & 3));
}

template <typename Real>
__global__ void __launch_bounds__(256, 2) hdb_sparse_gram_kernel(const SparseArgs a) {
    constexpr int TS = 128;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) float s_norm[2][TS];  // times 1 - eta
    const int tmax = (a.nmax + TS - 1) / TS;
    const int per = tmax * (tmax + 1) / 2;
    const int item = blockIdx.x / per;
    const int t = blockIdx.x - item * per;
    const int w = a.queue[item];
    const int64_t base = a.offsets[w];
    const int n = (int)(a.offsets[w + 1] - base);
    int tj = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while (tj * (tj + 1) / 2 > t) --tj;
    while ((tj + 1) * (tj + 2) / 2 <= t) ++tj;
    const int ti = t - tj * (tj + 1) / 2;
    if (tj * TS >= n || a.flags[w]) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int i0 = ti * TS, j0 = tj * TS;
    const int chunks = a.dims >> 5;
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
    const float inf = __int_as_float(0x7f800000);
    const float less = 1.0f - sparse_eta(a, w);
    for (int r = tid; r < 2 * TS; r += 256) {
        const int g = (r < TS ? i0 + r : j0 + r - TS);
        s_norm[r >> 7][r & (TS - 1)] = (g < n ? a.norm[base + g] : inf) * less;
    }
    const int row_bytes = 4 * a.dims;
    const int lr = tid >> 3;                      // 2 operands x 128 rows x 8 chunks of 16 bytes
    const uint32_t dst0 = sbase + lr * 128 + (((tid & 7) ^ (lr & 7)) << 4);
    const char* src0 = reinterpret_cast<const char*>(a.split + base * 2 * a.dims) + (tid & 7) * 16;
    auto load = [&](int c, int stage) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int g = (q < 4 ? i0 : j0) + lr + 32 * (q & 3);
            const char* src = src0 + (int64_t)min(g, n - 1) * row_bytes + c * 128;
            const int bytes = g < n ? 16 : 0;     // rows past the window are zeros
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst0 + stage * kGramStage + q * 4096),
                         "l"(src), "r"(bytes));
        }
        asm volatile("cp.async.commit_group;");
    };
    float acc[2][8][4];
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int q = 0; q < 8; ++q)
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[p][q][r] = 0.0f;
    const int wm = (warp & 3) * 32, wn = (warp >> 2) * 64;
    load(0, 0);
    for (int c = 0; c < chunks; ++c) {
        if (c + 1 < chunks) {
            load(c + 1, (c + 1) & 1);
            asm volatile("cp.async.wait_group 1;");
        } else {
            asm volatile("cp.async.wait_group 0;");
        }
        __syncthreads();
        const uint32_t A = sbase + (c & 1) * kGramStage, B = A + TS * 128;
        uint32_t hi[2][2][4], lo[2][2][4];  // [16 coordinates][16 rows]
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                const int r = wm + 16 * p + (lane & 15);
                const int ch = 2 * k + (lane >> 4);
                ldmatrix4(hi[k][p], A + r * 128 + ((ch ^ (r & 7)) << 4));
                ldmatrix4(lo[k][p], A + r * 128 + (((ch + 4) ^ (r & 7)) << 4));
            }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = wn + 16 * q + (lane & 7) + ((lane >> 4) << 3);
            float part[2][2][4];
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int e = 0; e < 4; ++e) part[p][h][e] = 0.0f;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int ch = 2 * k + ((lane >> 3) & 1);
                uint32_t bh[4], bl[4];
                ldmatrix4(bh, B + r * 128 + ((ch ^ (r & 7)) << 4));
                ldmatrix4(bl, B + r * 128 + (((ch + 4) ^ (r & 7)) << 4));
#pragma unroll
                for (int p = 0; p < 2; ++p)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        mma_bf16(part[p][h], hi[k][p], bl[2 * h], bl[2 * h + 1]);
                        mma_bf16(part[p][h], lo[k][p], bh[2 * h], bh[2 * h + 1]);
                        mma_bf16(part[p][h], hi[k][p], bh[2 * h], bh[2 * h + 1]);
                    }
            }
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[p][2 * q + h][e] += part[p][h][e];
        }
        __syncthreads();
    }
    float* __restrict__ Dw = sparse_block<Real>(a, w);
    float* __restrict__ minima = a.minima + a.dist_offsets[w] / 8;
    const int groups = (n + 15) >> 4;
    const int64_t ld = dist_ld(n);
    const bool diagonal = ti == tj;
    // Accumulators become bounds in place (the norms carry 1 - eta); points past the
    // window have infinite norms, so their entries are infinite.
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float ni = s_norm[0][wm + 16 * p + 8 * h + (lane >> 2)];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const float2 nj = *reinterpret_cast<const float2*>(&s_norm[1][wn + 8 * q + 2 * (lane & 3)]);
                acc[p][q][2 * h] = fmaxf(__fmaf_rn(-2.0f, acc[p][q][2 * h], ni + nj.x), 0.0f);
                acc[p][q][2 * h + 1] = fmaxf(__fmaf_rn(-2.0f, acc[p][q][2 * h + 1], ni + nj.y), 0.0f);
            }
        }
    // The tile in shared memory, over the stages (the loop's last barrier ended their
    // use).  In a diagonal tile both halves are in the accumulators; the products'
    // asymmetry could make them differ, so the upper one is taken for both.
    float* tile = reinterpret_cast<float*>(smem);
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = wm + 16 * p + 8 * h + (lane >> 2);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int col = wn + 8 * q + 2 * (lane & 3);
                const float v0 = acc[p][q][2 * h], v1 = acc[p][q][2 * h + 1];
                if (!diagonal) {
                    *reinterpret_cast<float2*>(tile + gram_at(r, col)) = make_float2(v0, v1);
                } else {
                    if (r <= col) tile[gram_at(r, col)] = tile[gram_at(col, r)] = v0;
                    if (r <= col + 1) tile[gram_at(r, col + 1)] = tile[gram_at(col + 1, r)] = v1;
                }
            }
        }
    __syncthreads();
    // Rows: 512 bytes a warp and store, with the minima of 16 columns (four lanes).
    // (Entries past the window, up to three in a row's padding, are infinite.)
    {
        const int gi = i0 + warp * (TS / 8), gj = j0 + 4 * lane, g = gj >> 4;
        float* out = Dw + gi * ld + gj;
        float* least = minima + (int64_t)gi * groups + g;
        const bool store = gj < n, store_min = (lane & 3) == 0 && g < groups;
#pragma unroll 8
        for (int k = 0; k < TS / 8; ++k) {
            const float4 v = *reinterpret_cast<const float4*>(tile + gram_at(warp * (TS / 8) + k, 4 * lane));
            float m = fminf(fminf(v.x, v.y), fminf(v.z, v.w));
            m = fminf(m, __shfl_xor_sync(0xffffffffu, m, 1));
            m = fminf(m, __shfl_xor_sync(0xffffffffu, m, 2));
            if (gi + k < n) {
                if (store) *reinterpret_cast<float4*>(out + k * ld) = v;
                if (store_min) least[k * groups] = m;
            }
        }
    }
    if (diagonal) return;
    // Columns: a lane reads four of one row; a warp's stores are 32 rows of one column.
    // (Rows lie above the diagonal, so inside the window.)
    for (int q = warp * 4; q < warp * 4 + 4; ++q) {
        const int gj = j0 + 4 * q;
        float* out = Dw + (int64_t)gj * ld + i0 + lane;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float4 v = *reinterpret_cast<const float4*>(tile + gram_at(32 * k + lane, 4 * q));
            if (gj < n) out[32 * k] = v.x;
            if (gj + 1 < n) out[32 * k + ld] = v.y;
            if (gj + 2 < n) out[32 * k + 2 * ld] = v.z;
            if (gj + 3 < n) out[32 * k + 3 * ld] = v.w;
        }
    }
    // The columns' minima of 16 rows: a thread takes half a column.
    const int col = tid & (TS - 1), half = tid >> 7;
    if (j0 + col < n) {
        float* least = minima + (int64_t)(j0 + col) * groups + (i0 >> 4) + 4 * half;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            float m = inf;
#pragma unroll
            for (int r = 0; r < 16; ++r) m = fminf(m, tile[gram_at(64 * half + 16 * g + r, col)]);
            least[g] = m;
        }
    }
}

// ---------------------------------------------------------------------------
// float32 distance blocks: 128x128 tiles of the upper triangle, 8x8 pairs a
// thread, mirrored, differences in packed f32x2 instructions.  float32 windows:
// the exact arithmetic of hdb_distance128_kernel (packed squares, scalar
// k-ordered sums).  float64 windows: the narrowed input, squares fused into the
// sums (one instruction a pair and coordinate, half of the exact form's).
// ---------------------------------------------------------------------------
template <typename Real>
__global__ void __launch_bounds__(256, 2) hdb_sparse_tiles_kernel(const SparseArgs a) {
    constexpr bool kExact = sizeof(Real) == 4;
    constexpr int KC = 32;
    constexpr int TS = 128;
    __shared__ __align__(16) float s_i[KC][TS];
    __shared__ __align__(16) float s_j[KC][TS];
    const int tmax = (a.nmax + TS - 1) / TS;
    const int per = tmax * (tmax + 1) / 2;
    const int item = blockIdx.x / per;
    int t = blockIdx.x - item * per;
    const int w = a.queue[item];
    const int64_t base = a.offsets[w];
    const int n = (int)(a.offsets[w + 1] - base);
    // Tile t of the lower triangle row by row: (row tj, column ti <= tj).
    int tj = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while (tj * (tj + 1) / 2 > t) --tj;
    while ((tj + 1) * (tj + 2) / 2 <= t) ++tj;
    const int ti = t - tj * (tj + 1) / 2;
    if (tj * TS >= n || a.flags[w]) return;
    const int D = a.D;
    const float* __restrict__ Y = (kExact ? static_cast<const float*>(a.X) : a.y) + base * D;
    float* __restrict__ Dw = sparse_block<Real>(a, w);
    const int64_t ld = dist_ld(n);
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int i0 = ti * TS, j0 = tj * TS;
    float2 acc[8][4];
#pragma unroll
    for (int p = 0; p < 8; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[p][q] = make_float2(0.0f, 0.0f);
    for (int k0 = 0; k0 < D; k0 += KC) {
        {
            const int r = tid & (TS - 1), kq = tid >> 7;
            const int gi = i0 + r, gj = j0 + r;
#pragma unroll
            for (int kk = 0; kk < KC / 2; ++kk) {
                const int k = kq * (KC / 2) + kk, gk = k0 + k;
                s_i[k][r] = (gi < n && gk < D) ? Y[(int64_t)gi * D + gk] : 0.0f;
                s_j[k][r] = (gj < n && gk < D) ? Y[(int64_t)gj * D + gk] : 0.0f;
            }
        }
        __syncthreads();
        const int kend = min(KC, D - k0);
        auto step = [&](int k) {
            float xi[8];
            float2 xj[4];
            DistVec<float>::load4(&s_i[k][ty * 4], xi);
            DistVec<float>::load4(&s_i[k][64 + ty * 4], xi + 4);
            const float4 u = *reinterpret_cast<const float4*>(&s_j[k][tx * 4]);
            const float4 v = *reinterpret_cast<const float4*>(&s_j[k][64 + tx * 4]);
            xj[0] = make_float2(u.x, u.y); xj[1] = make_float2(u.z, u.w);
            xj[2] = make_float2(v.x, v.y); xj[3] = make_float2(v.z, v.w);
#pragma unroll
            for (int p = 0; p < 8; ++p) {
                const float2 xa = make_float2(xi[p], xi[p]);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float2 d = __ffma2_rn(xj[q], make_float2(-1.0f, -1.0f), xa);
                    if constexpr (kExact) {
                        const float2 sq = __fmul2_rn(d, d);
                        acc[p][q].x = __fadd_rn(acc[p][q].x, sq.x);
                        acc[p][q].y = __fadd_rn(acc[p][q].y, sq.y);
                    } else {
                        acc[p][q] = __ffma2_rn(d, d, acc[p][q]);
                    }
                }
            }
        };
        if (kend == KC) {
#pragma unroll 4
            for (int k = 0; k < KC; ++k) step(k);
        } else {
            for (int k = 0; k < kend; ++k) step(k);
        }
        __syncthreads();
    }
    float out[8][8];
#pragma unroll
    for (int p = 0; p < 8; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            out[p][2 * q] = __fsqrt_rn(acc[p][q].x);
            out[p][2 * q + 1] = __fsqrt_rn(acc[p][q].y);
        }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int cj = j0 + h * 64 + tx * 4;
        if (cj < ld) {
#pragma unroll
            for (int p = 0; p < 8; ++p) {
                const int gi = i0 + (p < 4 ? ty * 4 + p : 64 + ty * 4 + p - 4);
                if (gi < n)
                    DistVec<float>::store4(Dw + gi * ld + cj, out[p][4 * h], out[p][4 * h + 1], out[p][4 * h + 2],
                                           out[p][4 * h + 3]);
            }
        }
        if (ti != tj) {
            const int ci = i0 + h * 64 + ty * 4;
            if (ci < ld) {
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int gj = j0 + (q < 4 ? tx * 4 + q : 64 + tx * 4 + q - 4);
                    if (gj < n)
                        DistVec<float>::store4(Dw + gj * ld + ci, out[4 * h][q], out[4 * h + 1][q], out[4 * h + 2][q],
                                               out[4 * h + 3][q]);
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Nearest-neighbour lists of every row, one warp a row, as hdb_core_rows_kernel
// builds them (the K smallest (distance, index), ascending, position p in lane
// p % 32).  Exact distances: position ms - 1 is the core distance.  Bounded
// ones: the rank ms - 1 is certain except among the entries whose bounds
// overlap that entry's; their positions [c, e) go to core_nbr
// for hdb_sparse_core_kernel.  A list that ends inside that range, or a
// distance that is not finite, flags the window.
// ---------------------------------------------------------------------------
// The end of a row: its list, and its core distance or the list positions where
// that is to be looked for.
template <typename Real, int E>
__device__ __forceinline__ void finish_row(const SparseArgs& a, const SparseBound& bound, int w, int64_t base, int n, int i,
                                           const uint32_t (&lk)[E], const int (&li)[E], bool wild) {
    const int lane = threadIdx.x & 31;
    const int keep = a.keep, last = keep - 1;
    auto at = [&](int p) {
        const uint32_t lo = __shfl_sync(0xffffffffu, lk[0], p & 31);
        if constexpr (E > 1) {
            const uint32_t hi = __shfl_sync(0xffffffffu, lk[1], p & 31);
            return p < 32 ? lo : hi;
        }
        return lo;
    };
    const int64_t row_at = base + i;
#pragma unroll
    for (int h = 0; h < E; ++h) {
        const int p = lane + 32 * h;
        if (p < keep) {
            a.knn_idx[row_at * a.list + p] = (uint16_t)(p < n ? li[h] : i);
            a.knn_d[row_at * a.list + p] = __uint_as_float(p < n ? lk[h] : 0x7f800000u);
        }
    }
    bool unsure = wild;
    if (!a.unit_core) {
        const int pos = a.ms - 1;
        if (!a.approx) {
#pragma unroll
            for (int h = 0; h < E; ++h)
                if (pos == lane + 32 * h) {
                    static_cast<float*>(a.core)[row_at] = __uint_as_float(lk[h]);
                    a.core_nbr[row_at] = li[h];
                }
            // Points as far as the core distance may follow the list's end.
            if (at(last) <= at(pos) && keep < n) unsure = true;
        } else {
            // The value of rank ms - 1 is at least the lower bound at that
            // position and at most the largest upper bound up to it.
            const float least = bound.down(__uint_as_float(at(pos)));
            const int inside = min(keep, n);
            float up[E], most = 0.0f;
            const float slack = 2.1f * bound.eta;
            const float norm_i = a.gram ? a.norm[row_at] : 0.0f;
#pragma unroll
            for (int h = 0; h < E; ++h) {
                const int p = lane + 32 * h;
                const float d = __uint_as_float(lk[h]);
                up[h] = bound.up(d);
                if (a.gram && p < inside) up[h] = __fmaf_ru(d, bound.up_scale, slack * (norm_i + a.norm[base + li[h]]));
                if (p <= pos) most = fmaxf(most, up[h]);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
            int c = inside, e = 0;
#pragma unroll
            for (int h = E - 1; h >= 0; --h) {
                const int p = lane + 32 * h;
                const unsigned open = __ballot_sync(0xffffffffu, p < inside && !(up[h] < least));
                if (open) c = 32 * h + __ffs(open) - 1;
                e += __popc(__ballot_sync(0xffffffffu, p < inside && bound.down(__uint_as_float(lk[h])) <= most));
            }
            if (e >= keep && keep < n) unsure = true;  // the range may go on beyond the list
            if (lane == 0) a.core_nbr[row_at] = c | (e << 8);
        }
    }
    if (unsure && lane == 0) sparse_flag(a, w);
}

template <typename Real, int K>
__global__ void __launch_bounds__(32 * kCoreRowsWarps) hdb_sparse_rows_kernel(const SparseArgs a) {
    static_assert(K <= 64, "at most two list entries per lane");
    constexpr int E = (K + 31) / 32;
    constexpr uint32_t kNone = 0xffffffffu;
    constexpr int U = 8;
    const int per = (a.nmax + kSparseRowsCta - 1) / kSparseRowsCta;
    const int item = blockIdx.x / per, r0 = (blockIdx.x - item * per) * kSparseRowsCta;
    const int w = a.queue[item];
    const int64_t base = a.offsets[w];
    const int n = (int)(a.offsets[w + 1] - base);
    // float32 core distances also serve the general path of a flagged window.
    if (r0 >= n || (a.approx && a.flags[w])) return;
    const float* __restrict__ Dw = sparse_block<Real>(a, w);
    const int64_t ld = dist_ld(n);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int keep = a.keep;
    const int last = keep - 1;
    const SparseBound bound = sparse_bound<Real>(a, w);
    for (int r = warp; r < kSparseRowsCta; r += kCoreRowsWarps) {
        const int i = r0 + r;
        if (i >= n) break;  // warp-uniform
        const float* __restrict__ row = Dw + (int64_t)i * ld;
        uint32_t lk[E], biggest = 0;
        int li[E];
        lk[0] = lane < n ? RealTraits<float>::key(__ldcg(row + lane)) : kNone;
        biggest = lane < n ? lk[0] : 0u;
        li[0] = lane;
        if constexpr (E > 1) { lk[1] = kNone; li[1] = 32 + lane; }
#pragma unroll
        for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
            for (int j = k >> 1; j > 0; j >>= 1) {
                const uint32_t pk = __shfl_xor_sync(0xffffffffu, lk[0], j);
                const int pi = __shfl_xor_sync(0xffffffffu, li[0], j);
                const bool partner_less = pk < lk[0] || (pk == lk[0] && pi < li[0]);
                const bool keep_min = ((lane & k) == 0) == ((lane & j) == 0);
                const bool take = keep_min ? partner_less : !partner_less;
                lk[0] = take ? pk : lk[0];
                li[0] = take ? pi : li[0];
            }
        }
        auto at = [&](int p) {
            const uint32_t lo = __shfl_sync(0xffffffffu, lk[0], p & 31);
            if constexpr (E > 1) {
                const uint32_t hi = __shfl_sync(0xffffffffu, lk[1], p & 31);
                return p < 32 ? lo : hi;
            }
            return lo;
        };
        uint32_t tau = at(last);
        for (int j0 = 32; j0 < n; j0 += 32 * U) {
            uint32_t v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int j = j0 + 32 * u + lane;
                v[u] = j < n ? RealTraits<float>::key(__ldcg(row + j)) : kNone;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (v[u] != kNone) biggest = max(biggest, v[u]);
                unsigned bal = __ballot_sync(0xffffffffu, v[u] < tau);
                while (bal) {
                    const int src = __ffs(bal) - 1;
                    bal &= bal - 1;
                    const uint32_t ck = __shfl_sync(0xffffffffu, v[u], src);
                    if (ck < tau) {  // warp-uniform; tau only decreases
                        const int cj = j0 + 32 * u + src;
                        uint32_t pk[E];
                        int pi[E];
                        pk[0] = __shfl_up_sync(0xffffffffu, lk[0], 1);
                        pi[0] = __shfl_up_sync(0xffffffffu, li[0], 1);
                        if constexpr (E > 1) {
                            const uint32_t upk = __shfl_up_sync(0xffffffffu, lk[1], 1);
                            const int upi = __shfl_up_sync(0xffffffffu, li[1], 1);
                            const uint32_t endk = __shfl_sync(0xffffffffu, lk[0], 31);
                            const int endi = __shfl_sync(0xffffffffu, li[0], 31);
                            pk[1] = lane == 0 ? endk : upk;
                            pi[1] = lane == 0 ? endi : upi;
                        }
#pragma unroll
                        for (int h = 0; h < E; ++h) {
                            const bool shift = (h > 0 || lane > 0) && ck < pk[h];
                            const bool place = !shift && ck < lk[h];
                            lk[h] = shift ? pk[h] : (place ? ck : lk[h]);
                            li[h] = shift ? pi[h] : (place ? cj : li[h]);
                        }
                        tau = at(last);
                    }
                }
            }
        }
        const bool wild = __any_sync(0xffffffffu, biggest >= 0x7f800000u);
        finish_row<Real, E>(a, bound, w, base, n, i, lk, li, wild);
    }
}

// One compare-exchange stage of (key, index) over the lanes, distance j.
__device__ __forceinline__ void pair_stage(uint32_t& k, int& i, int j, bool keep_min) {
    const uint32_t pk = __shfl_xor_sync(0xffffffffu, k, j);
    const int pi = __shfl_xor_sync(0xffffffffu, i, j);
    const bool partner_less = pk < k || (pk == k && pi < i);
    const bool take = keep_min ? partner_less : !partner_less;
    k = take ? pk : k;
    i = take ? pi : i;
}

// The keep-th smallest (keep <= 32) of the 64 values x0, x1 of the lanes.
__device__ __forceinline__ uint32_t smallest_of_64(uint32_t x0, uint32_t x1, int keep) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const bool keep_min = ((lane & k) == 0) == ((lane & j) == 0);
            const uint32_t p0 = __shfl_xor_sync(0xffffffffu, x0, j), p1 = __shfl_xor_sync(0xffffffffu, x1, j);
            x0 = keep_min ? min(x0, p0) : max(x0, p0);
            // The second half descends: its first 32 meet the first half's last.
            x1 = keep_min ? max(x1, p1) : min(x1, p1);
        }
    }
    // x0 ascending, x1 descending: the lane-wise minima are the 32 smallest, a bitonic sequence.
    x0 = min(x0, x1);
#pragma unroll
    for (int j = 16; j > 0; j >>= 1) {
        const uint32_t p0 = __shfl_xor_sync(0xffffffffu, x0, j);
        x0 = (lane & j) == 0 ? min(x0, p0) : max(x0, p0);
    }
    return __shfl_sync(0xffffffffu, x0, keep - 1);
}

// Merges `count` (<= 32) gathered entries into the ascending list (k, i).
__device__ __forceinline__ void merge_batch(uint32_t& k, int& i, const uint2* batch, int count) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    const uint2 e = lane < count ? batch[lane] : make_uint2(0xffffffffu, 0x7fffffffu);
    uint32_t bk = e.x;
    int bi = (int)e.y;
#pragma unroll
    for (int s = 2; s <= 32; s <<= 1)
#pragma unroll
        for (int j = s >> 1; j > 0; j >>= 1)  // descending
            pair_stage(bk, bi, j, ((lane & s) == 0) != ((lane & j) == 0));
    const bool less = bk < k || (bk == k && bi < i);
    k = less ? bk : k;
    i = less ? bi : i;
#pragma unroll
    for (int j = 16; j > 0; j >>= 1) pair_stage(k, i, j, (lane & j) == 0);
    __syncwarp();
}

// Product blocks come with the minimum of every 16 entries of a row (written by
// hdb_sparse_gram_kernel), so a row is read in two steps: its minima, whose
// keep-th smallest (of 64 partial ones, two a lane) bounds the list's end, and
// the groups that reach below it, little more than keep of them.  Entries below
// the bound gather in shared memory and join the list 32 at a time (sort,
// bitonic merge).
constexpr int kGroup = 16;

// The window's group minima, [n][ceil(n / 16)], after the distance blocks.
template <typename Real>
__device__ __forceinline__ float* sparse_minima(const SparseArgs& a, int w) {
    return a.minima + a.dist_offsets[w] / 8;
}

template <typename Real>
__global__ void __launch_bounds__(32 * kCoreRowsWarps) hdb_sparse_gram_rows_kernel(const SparseArgs a) {
    constexpr uint32_t kNone = 0xffffffffu;
    constexpr int kGroups = 4096 / kGroup;
    __shared__ uint2 s_batch[kCoreRowsWarps][64];
    __shared__ uint8_t s_group[kCoreRowsWarps][kGroups];
    const int per = (a.nmax + kSparseRowsCta - 1) / kSparseRowsCta;
    const int item = blockIdx.x / per, r0 = (blockIdx.x - item * per) * kSparseRowsCta;
    const int w = a.queue[item];
    const int64_t base = a.offsets[w];
    const int n = (int)(a.offsets[w + 1] - base);
    if (r0 >= n || a.flags[w]) return;
    const float* __restrict__ Dw = sparse_block<Real>(a, w);
    const float* __restrict__ minima = sparse_minima<Real>(a, w);
    const int64_t ld = dist_ld(n);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int keep = a.keep, last = keep - 1, groups = (n + kGroup - 1) / kGroup;
    const SparseBound bound = sparse_bound<Real>(a, w);
    uint2* batch = s_batch[warp];
    uint8_t* group = s_group[warp];
    for (int r = warp; r < kSparseRowsCta; r += kCoreRowsWarps) {
        const int i = r0 + r;
        if (i >= n) break;  // warp-uniform
        const float* __restrict__ row = Dw + (int64_t)i * ld;
        const float* __restrict__ least = minima + (int64_t)i * groups;
        uint32_t g[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) g[q] = lane + 32 * q < groups ? __float_as_uint(__ldcg(least + lane + 32 * q)) : kNone;
        const uint32_t m0 = min(min(g[0], g[2]), min(g[4], g[6])), m1 = min(min(g[1], g[3]), min(g[5], g[7]));
        uint32_t limit = smallest_of_64(m0, m1, keep);  // entries up to it pass
        int found = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const unsigned bal = __ballot_sync(0xffffffffu, g[q] <= limit && g[q] != kNone);
            if ((bal >> lane) & 1u) group[found + __popc(bal & lanemask_lt())] = (uint8_t)(lane + 32 * q);
            found += __popc(bal);
        }
        __syncwarp();
        uint32_t lk[1] = {kNone};
        int li[1] = {0x7fffffff};
        int waiting = 0;
        for (int t = 0; t < found; t += 8) {
            uint32_t v[4];
            int col[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int e = t + 2 * q + (lane >> 4);
                col[q] = e < found ? (int)group[e] * kGroup + (lane & (kGroup - 1)) : n;
                v[q] = col[q] < n ? __float_as_uint(__ldcg(row + col[q])) : kNone;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const bool pass = v[q] <= limit && v[q] != kNone;
                const unsigned bal = __ballot_sync(0xffffffffu, pass);
                if (pass) batch[waiting + __popc(bal & lanemask_lt())] = make_uint2(v[q], (uint32_t)col[q]);
                waiting += __popc(bal);
                if (waiting >= 32) {
                    merge_batch(lk[0], li[0], batch, 32);
                    waiting -= 32;
                    const uint2 rest = batch[32 + lane];
                    __syncwarp();
                    if (lane < waiting) batch[lane] = rest;
                    limit = min(limit, __shfl_sync(0xffffffffu, lk[0], last));
                }
            }
        }
        if (waiting > 0) merge_batch(lk[0], li[0], batch, waiting);
        finish_row<Real, 1>(a, bound, w, base, n, i, lk, li, false);
    }
}

// Core distances from bounded ones: the exact distances of each row's uncertain
// range (mostly one entry), the right one by (distance, index).  A warp takes 32
// rows and spreads all their entries over its lanes.
constexpr int kCoreEntries = 256;  // uncertain entries of 32 rows

template <typename Real>
__global__ void __launch_bounds__(128) hdb_sparse_core_kernel(const SparseArgs a) {
    __shared__ Real s_d[4][kCoreEntries];
    __shared__ uint16_t s_entry[4][kCoreEntries];  // row << 8 | list position
    const int per = (a.nmax + 127) / 128;
    const int item = blockIdx.x / per, i0 = (blockIdx.x - item * per) * 128;
    const int w = a.queue[item];
    const int64_t base = a.offsets[w];
    const int n = (int)(a.offsets[w + 1] - base);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int first = i0 + 32 * warp, i = first + lane;
    if (first >= n || a.flags[w]) return;  // warp-uniform
    const int D = a.D;
    const Real* __restrict__ X = static_cast<const Real*>(a.X) + base * D;
    const int64_t row = base + i;
    const int range = i < n ? a.core_nbr[row] : 0;
    const int c = range & 0xff, e = range >> 8;
    const int count = e - c;
    int at = count;  // inclusive, then exclusive prefix
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += y;
    }
    const int total = __shfl_sync(0xffffffffu, at, 31);
    at -= count;
    if (total > kCoreEntries) {  // the bound separates too little here
        if (lane == 0) sparse_flag(a, w);
        return;
    }
    for (int s = 0; s < count; ++s) s_entry[warp][at + s] = (uint16_t)((lane << 8) | (c + s));
    __syncwarp();
    for (int t = lane; t < total; t += 32) {
        const int entry = s_entry[warp][t];
        const int u = first + (entry >> 8);
        const int v = a.knn_idx[(base + u) * a.list + (entry & 0xff)];
        s_d[warp][t] = sparse_exact<Real>(X + (int64_t)u * D, X + (int64_t)v * D, D);
    }
    __syncwarp();
    if (i >= n) return;
    // The (ms - 1 - c)-th smallest of the range: repeated minimum above the last one taken.
    const uint16_t* __restrict__ list = a.knn_idx + row * a.list;
    Real value = Real(-1);
    int index = -1;
    for (int t = c; t <= a.ms - 1; ++t) {
        Real best = Real(0);
        int j_best = -1;
        for (int s = 0; s < count; ++s) {
            const Real d = s_d[warp][at + s];
            const int j = list[c + s];
            const bool above = d > value || (d == value && j > index);
            if (above && (j_best < 0 || d < best || (d == best && j < j_best))) { best = d; j_best = j; }
        }
        value = best;
        index = j_best;
    }
    static_cast<Real*>(a.core)[row] = value;
    a.core_nbr[row] = index;
    // In the block's terms: squares where it holds squares.
    if constexpr (sizeof(Real) == 4) {
        a.core_up[row] = __fmul_ru(value, value);
        a.core_down[row] = __fmul_rd(value, value);
    } else {
        a.core_up[row] = __double2float_ru(a.gram ? __dmul_ru(value, value) : value);
        a.core_down[row] = __double2float_rd(a.gram ? __dmul_rd(value, value) : value);
    }
}

// ---------------------------------------------------------------------------
// The spanning tree T' and its merge rounds, in three kernels.  Edges are
// ordered by (weight rounded up, smaller end, larger end), so all minima below
// are unique; T' is the minimum spanning tree of those weights, up to edges
// taken in forced rounds.
//
// hdb_sparse_forest_kernel (one CTA a window): rounds in which every component
// takes its least edge among the neighbour lists, as long as no edge outside
// the lists can be shorter (a list ends at a known distance).  What is left,
// typically a few percent of the points, are components whose least outgoing
// edge is longer than some member's list reaches.
//
// hdb_sparse_between_kernel (all rows): the least edge between each two of
// those components, into a table.
//
// hdb_sparse_tree_kernel (one CTA a window): the remaining rounds on the table;
// then the merge rounds (Boruvka over the n-1 edges of T') and the leaf order in
// which every component of every round is an interval.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long sparse_key(float wgt, int u, int v) {
    const uint32_t lo = (uint32_t)min(u, v), hi = (uint32_t)max(u, v);
    return ((unsigned long long)__float_as_uint(wgt) << 32) | (lo << 12) | hi;
}
__device__ __forceinline__ uint32_t key_weight(unsigned long long key) { return (uint32_t)(key >> 32); }
__device__ __forceinline__ int key_low(unsigned long long key) { return (int)((uint32_t)key >> 12) & 0xfff; }
__device__ __forceinline__ int key_high(unsigned long long key) { return (int)key & 0xfff; }

__host__ __device__ inline int sparse_round(int n) { return (n + 15) & ~15; }
__host__ __device__ inline size_t sparse_forest_smem(int n) {
    return (size_t)sparse_round(n) * (8 + 4 + 4 + 4 + 2 + 2 + 1) + 64;
}
__host__ __device__ inline size_t sparse_between_smem(int n) {
    return (size_t)sparse_round(n) * (2 + 4) + (size_t)sparse_parts_cap(n) * 8 * 8 + 64;
}
__host__ __device__ inline size_t sparse_tree_smem(int n) {
    return (size_t)sparse_round(n) * (8 + 8 + 4 + 2 + 2) + 64;
}

constexpr unsigned long long kNoChoice = ~0ull;

// Root (in `up`) that component r's chosen edge leads to.  Both ends choosing
// the same edge is the only cycle: the smaller id stays the root.
__device__ __forceinline__ int sparse_target(const unsigned long long* choice, const uint16_t* comp, int r) {
    const unsigned long long key = choice[r];
    if (key == kNoChoice) return r;
    const int lo = comp[key_low(key)], hi = comp[key_high(key)];
    const int to = lo == r ? hi : lo;
    return (choice[to] == key && r < to) ? r : to;
}
__device__ __forceinline__ int sparse_root(const uint16_t* up, int r, int n) {
    for (int guard = 0; guard < n && up[r] != r; ++guard) r = up[r];
    return r;
}

template <typename Real>
__global__ void __launch_bounds__(512) hdb_sparse_forest_kernel(const SparseArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_edges;   // tree edges found
    __shared__ int s_parts;   // components
    __shared__ int s_next;
    const int w = a.queue[blockIdx.x];
    if (a.flags[w]) return;
    const int64_t base = a.offsets[w];
    const int n = (int)(a.offsets[w + 1] - base);
    const int tid = threadIdx.x, nt = blockDim.x;
    const int cap = sparse_round(n);
    unsigned long long* choice = reinterpret_cast<unsigned long long*>(smem);
    float* core = reinterpret_cast<float*>(choice + cap);   // core distances rounded up
    uint32_t* reach_v = reinterpret_cast<uint32_t*>(core + cap);  // float bits: shortest edge a point's list can miss
    uint32_t* reach = reach_v + cap;                        // the same over a component
    uint16_t* comp = reinterpret_cast<uint16_t*>(reach + cap);
    uint16_t* up = comp + cap;
    uint8_t* at = reinterpret_cast<uint8_t*>(up + cap);
    const SparseBound bound = sparse_bound<Real>(a, w);
    if (a.approx) {
        // A range below 2^-40 (other than identical points) is outside the bound's domain.
        const float R = __uint_as_float(a.range[w]);
        if (R != 0.0f && R < (a.gram ? 8.3e-25f : 9.1e-13f)) {
            if (tid == 0) sparse_flag(a, w);
            return;
        }
    }
    const float* core_g = a.core_up;
    const int keep = min(a.keep, n);
    for (int u = tid; u < n; u += nt) {
        const float c = a.unit_core ? 0.0f : core_g[base + u];
        comp[u] = (uint16_t)u;
        core[u] = c;
        at[u] = 0;
        const float end = bound.up(a.knn_d[(base + u) * a.list + keep - 1]);
        reach_v[u] = keep == n ? 0x7f800000u : __float_as_uint(fmaxf(c, end));
    }
    if (tid == 0) s_edges = 0;
    unsigned long long* edges = a.edges + base;
    int parts = n;
    bool forced = false;
    for (int round = 0; round < 2 * kSparseLevels; ++round) {
        __syncthreads();
        for (int u = tid; u < n; u += nt) { choice[u] = kNoChoice; reach[u] = 0x7f800000u; }
        __syncthreads();
        for (int u = tid; u < n; u += nt) {
            const uint16_t* __restrict__ idx = a.knn_idx + (base + u) * a.list;
            const float* __restrict__ dd = a.knn_d + (base + u) * a.list;
            const int cu = comp[u];
            const float core_u = core[u];
            unsigned long long best = kNoChoice;
            int bv = 0;
            bool lead = true;
            int first = at[u];
            for (int t = first; t < keep; ++t) {
                const int v = idx[t];
                if (comp[v] == cu) {  // the point itself, or already joined: never looked at again
                    if (lead) first = t + 1;
                    continue;
                }
                lead = false;
                const float d = bound.up(dd[t]);
                if (__float_as_uint(d) > key_weight(best)) break;
                const unsigned long long key = sparse_key(fmaxf(fmaxf(core_u, core[v]), d), u, v);
                if (key < best) { best = key; bv = v; }
            }
            at[u] = (uint8_t)first;
            if (reach_v[u] < reach[cu]) atomicMin(&reach[cu], reach_v[u]);
            if (best != kNoChoice) {
                if (best < choice[cu]) atomicMin(&choice[cu], best);
                const int cv = comp[bv];
                if (best < choice[cv]) atomicMin(&choice[cv], best);
            }
        }
        __syncthreads();
        // An edge that the lists may have missed could be shorter: not chosen.
        if (!forced) {
            for (int r = tid; r < n; r += nt)
                if (comp[r] == r && key_weight(choice[r]) > reach[r]) choice[r] = kNoChoice;
            __syncthreads();
        }
        for (int r = tid; r < n; r += nt) {
            if (comp[r] != r) continue;
            const int to = sparse_target(choice, comp, r);
            up[r] = (uint16_t)to;
            if (to != r) edges[min(atomicAdd(&s_edges, 1), n - 1)] = choice[r];
        }
        __syncthreads();
        for (int u = tid; u < n; u += nt) comp[u] = (uint16_t)sparse_root(up, comp[u], n);
        const int now = n - s_edges;
        if (now == 1) { parts = now; break; }
        if (now == parts) {  // stalled: few enough components for the table, or joined whatever their lists say
            if (now <= sparse_parts_cap(n)) break;
            if (forced) break;
            forced = true;
        } else if (forced && now <= sparse_parts_cap(n)) {
            parts = now;
            break;
        }
        parts = now;
    }
    __syncthreads();
    const int parts_cap = sparse_parts_cap(n);
    if (parts > parts_cap) {  // unreachable: components that hold all their points' lists have 8 points or more
        if (tid == 0) sparse_flag(a, w);
        return;
    }
    // ---- components numbered, rows sorted by them, table cleared --------------
    uint32_t* number = reinterpret_cast<uint32_t*>(choice);
    uint32_t* count = number + cap;
    if (tid == 0) { s_parts = 0; s_next = 0; }
    for (int u = tid; u < n; u += nt) count[u] = 0;
    __syncthreads();
    for (int u = tid; u < n; u += nt) {
        atomicAdd(&count[comp[u]], 1u);
        if (comp[u] == u) number[u] = (uint32_t)atomicAdd(&s_parts, 1);
    }
    __syncthreads();
    for (int u = tid; u < n; u += nt)
        if (comp[u] == u) count[u] = (uint32_t)atomicAdd(&s_next, (int)count[u]);
    __syncthreads();
    for (int u = tid; u < n; u += nt) {
        const int r = comp[u];
        a.part[base + u] = (uint16_t)number[r];
        a.perm[base + atomicAdd(&count[r], 1u)] = (uint16_t)u;
    }
    unsigned long long* table = a.table + a.table_offsets[w];
    if (parts > 1)
        for (int e = tid; e < parts * parts; e += nt) table[e] = kNoChoice;
    if (tid == 0) a.parts[w] = parts;
}

// The least edge between each two components, from the upper triangle of the
// block: every row u against its columns v > u, into table row part[u].  A warp
// takes a run of rows in component order and keeps the table row of the current
// component in shared memory.  Bound by the latency of the block's read (2 n^2
// bytes): 16 bytes a lane and load, four in flight, 63 us for 16 windows of 2048
// points; 4 bytes, eight in flight, 76; two of 16 with more CTAs an SM 75.
constexpr int kBetweenRows = 32;  // rows per CTA: runs of four a warp

template <typename Real>
__global__ void __launch_bounds__(256) hdb_sparse_between_kernel(const SparseArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int kRun = kBetweenRows / 8;
    const int per = (a.nmax + kBetweenRows - 1) / kBetweenRows;
    const int item = blockIdx.x / per, p0 = (blockIdx.x - item * per) * kBetweenRows;
    const int w = a.queue[item];
    const int64_t base = a.offsets[w];
    const int n = (int)(a.offsets[w + 1] - base);
    if (p0 >= n || a.flags[w]) return;
    const int parts = a.parts[w];
    if (parts <= 1) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cap = sparse_round(n);
    float* core = reinterpret_cast<float*>(smem);
    uint16_t* part = reinterpret_cast<uint16_t*>(core + cap);
    unsigned long long* least = reinterpret_cast<unsigned long long*>(part + cap) + (size_t)warp * parts;
    const uint32_t* least_w = reinterpret_cast<const uint32_t*>(least) + 1;  // high words: weights
    for (int u = tid; u < n; u += 256) {
        core[u] = a.unit_core ? 0.0f : a.core_up[base + u];
        part[u] = a.part[base + u];
    }
    for (int u = n + tid; u < cap; u += 256) {  // (rows are read by fours)
        core[u] = 0.0f;
        part[u] = 0;
    }
    __syncthreads();
    const float* __restrict__ Dw = sparse_block<Real>(a, w);
    const int64_t ld = dist_ld(n);
    const SparseBound bound = sparse_bound<Real>(a, w);
    unsigned long long* table = a.table + a.table_offsets[w];
    int mine = -1;
    auto flush = [&]() {
        __syncwarp();
        if (mine >= 0)
            for (int c = lane; c < parts; c += 32)
                if (least[c] < table[(int64_t)mine * parts + c]) atomicMin(&table[(int64_t)mine * parts + c], least[c]);
        __syncwarp();
    };
    for (int p = p0 + kRun * warp; p < min(p0 + kRun * (warp + 1), n); ++p) {
        const int u = a.perm[base + p];
        const int cu = part[u];
        if (cu != mine) {
            flush();
            mine = cu;
            for (int c = lane; c < parts; c += 32) least[c] = table[(int64_t)mine * parts + c];
            __syncwarp();
        }
        const float* __restrict__ row = Dw + (int64_t)u * ld;
        const float core_u = core[u];
        constexpr int U = 4;
        for (int v0 = ((u + 1) & ~31) + 4 * lane; v0 < n; v0 += 128 * U) {
            float4 d4[U];
#pragma unroll
            for (int q = 0; q < U; ++q) {
                const int v = v0 + 128 * q;
                d4[q] = v < n ? __ldcg(reinterpret_cast<const float4*>(row + v)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
#pragma unroll
            for (int q = 0; q < U; ++q) {
                const int v = v0 + 128 * q;
                if (v >= n) break;
                const float4 core4 = *reinterpret_cast<const float4*>(core + v);
                const ushort4 part4 = *reinterpret_cast<const ushort4*>(part + v);
                const float d[4] = {d4[q].x, d4[q].y, d4[q].z, d4[q].w};
                const float cores[4] = {core4.x, core4.y, core4.z, core4.w};
                const int cv[4] = {part4.x, part4.y, part4.z, part4.w};
                float wgt[4];
                unsigned hit = 0;
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    wgt[b] = fmaxf(fmaxf(core_u, cores[b]), bound.up(d[b]));
                    if (cv[b] != cu && __float_as_uint(wgt[b]) <= least_w[2 * cv[b]]) hit |= 1u << b;
                }
                if (!hit) continue;
#pragma unroll
                for (int b = 0; b < 4; ++b)
                    if ((hit >> b & 1) && v + b > u && v + b < n) atomicMin(&least[cv[b]], sparse_key(wgt[b], u, v + b));
            }
        }
    }
    flush();
}

template <typename Real>
__global__ void __launch_bounds__(512) hdb_sparse_tree_kernel(const SparseArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_edges;   // tree edges found
    __shared__ int s_parts;   // components
    const int w = a.queue[blockIdx.x];
    if (a.flags[w]) return;
    const int64_t base = a.offsets[w];
    const int n = (int)(a.offsets[w + 1] - base);
    const int tid = threadIdx.x, nt = blockDim.x;
    const int cap = sparse_round(n);
    unsigned long long* choice = reinterpret_cast<unsigned long long*>(smem);
    unsigned long long* edge = choice + cap;
    float* top = reinterpret_cast<float*>(edge + cap);     // largest edge from the leaf up
    uint16_t* comp = reinterpret_cast<uint16_t*>(top + cap);
    uint16_t* up = comp + cap;
    // ---- the remaining rounds, on the table ------------------------------------
    const int parts = a.parts[w];
    const unsigned long long* __restrict__ table = a.table + a.table_offsets[w];
    for (int e = tid; e < n - parts; e += nt) edge[e] = a.edges[base + e];
    if (tid == 0) s_edges = n - parts;
    uint16_t* owner = reinterpret_cast<uint16_t*>(top);     // component of each table row, by number
    for (int c = tid; c < parts; c += nt) owner[c] = (uint16_t)c;
    // In these rounds component numbers stand for the points: comp maps a point
    // to its number's current root.
    uint16_t* part = up;
    for (int u = tid; u < n; u += nt) part[u] = a.part[base + u];
    uint16_t* next = comp;  // next[c]: root that number c's component joins
    __syncthreads();
    for (int round = 0; round < kSparseLevels && s_edges < n - 1; ++round) {
        for (int c = tid; c < parts; c += nt) choice[c] = kNoChoice;
        __syncthreads();
        for (int i = tid; i < parts * parts; i += nt) {
            const int r = i / parts, c = i - r * parts;
            const int cr = owner[r], cc = owner[c];
            if (cr == cc) continue;
            const unsigned long long key = table[i];
            if (key == kNoChoice) continue;
            if (key < choice[cr]) atomicMin(&choice[cr], key);
            if (key < choice[cc]) atomicMin(&choice[cc], key);
        }
        __syncthreads();
        for (int r = tid; r < parts; r += nt) {
            if (owner[r] != r) continue;
            const unsigned long long key = choice[r];
            int to = r;
            if (key != kNoChoice) {
                const int lo = owner[part[key_low(key)]], hi = owner[part[key_high(key)]];
                to = lo == r ? hi : lo;
                if (choice[to] == key && r < to) to = r;
                if (to != r) edge[min(atomicAdd(&s_edges, 1), n - 1)] = key;
            }
            next[r] = (uint16_t)to;
        }
        __syncthreads();
        for (int c = tid; c < parts; c += nt) owner[c] = (uint16_t)sparse_root(next, owner[c], parts);
        __syncthreads();
    }
    if (s_edges != n - 1) {  // unreachable: each round at least halves the components, 2^kSparseLevels points
        if (tid == 0) sparse_flag(a, w);
        return;
    }
    // ---- merge rounds of T' ---------------------------------------------------
    __syncthreads();
    for (int u = tid; u < n; u += nt) { comp[u] = (uint16_t)u; top[u] = 0.0f; }
    int level = 0;
    for (; level < kSparseLevels; ++level) {
        for (int u = tid; u < n; u += nt) choice[u] = kNoChoice;
        if (tid == 0) s_parts = 0;
        __syncthreads();
        for (int e = tid; e < n - 1; e += nt) {
            const unsigned long long key = edge[e];
            const int lo = comp[key_low(key)], hi = comp[key_high(key)];
            if (lo == hi) continue;
            if (key < choice[lo]) atomicMin(&choice[lo], key);
            if (key < choice[hi]) atomicMin(&choice[hi], key);
        }
        __syncthreads();
        for (int r = tid; r < n; r += nt)
            if (comp[r] == r) up[r] = (uint16_t)sparse_target(choice, comp, r);
        __syncthreads();
        for (int u = tid; u < n; u += nt) {
            const unsigned long long key = choice[comp[u]];
            if (key != kNoChoice) top[u] = fmaxf(top[u], __uint_as_float(key_weight(key)));
            const int r = sparse_root(up, comp[u], n);
            a.level_comp[(int64_t)level * a.T + base + u] = (uint16_t)r;
            a.level_max_v[(int64_t)level * a.T + base + u] = top[u];
            if (u == r) atomicAdd(&s_parts, 1);
        }
        __syncthreads();
        for (int u = tid; u < n; u += nt) comp[u] = a.level_comp[(int64_t)level * a.T + base + u];
        const int left = s_parts;
        __syncthreads();
        if (left == 1) { ++level; break; }
    }
    if (s_parts != 1) {  // unreachable, as above
        if (tid == 0) sparse_flag(a, w);
        return;
    }
    // ---- leaf order: intervals handed down the rounds ------------------------
    uint32_t* cursor = reinterpret_cast<uint32_t*>(choice);  // next free leaf of each component
    uint32_t* place = cursor + cap;                          // first leaf of each component one round down
    uint32_t* size = reinterpret_cast<uint32_t*>(top);
    for (int u = tid; u < n; u += nt) cursor[u] = 0;
    __syncthreads();
    for (int l = level; l >= 1; --l) {
        const uint16_t* parent = a.level_comp + (int64_t)(l - 1) * a.T + base;  // component after l rounds
        const uint16_t* child = l >= 2 ? a.level_comp + (int64_t)(l - 2) * a.T + base : nullptr;
        if (child) {
            for (int u = tid; u < n; u += nt) size[u] = 0;
            __syncthreads();
            for (int u = tid; u < n; u += nt) atomicAdd(&size[child[u]], 1u);
            __syncthreads();
        }
        for (int r = tid; r < n; r += nt)
            if (!child || child[r] == r) place[r] = atomicAdd(&cursor[parent[r]], child ? size[r] : 1u);
        __syncthreads();
        if (child) {
            for (int r = tid; r < n; r += nt)
                if (child[r] == r) cursor[r] = place[r];
            for (int u = tid; u < n; u += nt)
                a.level_span[(int64_t)(l - 2) * a.T + base + u] = place[child[u]] | ((place[child[u]] + size[child[u]]) << 16);
            __syncthreads();
        }
    }
    for (int u = tid; u < n; u += nt) {
        a.pos[base + u] = (uint16_t)place[u];
        a.level_span[(int64_t)(level - 1) * a.T + base + u] = (uint32_t)n << 16;
    }
    if (tid == 0) a.levels[w] = level;
}

// ---------------------------------------------------------------------------
// Light edges: all pairs (u < v) whose distance is at most the path maximum
// max(top_l(u), top_l(v)), l the first round that joins them.  Core distances
// need no test: both ends' maxima are at least their own cores.  Pairs whose
// weight is certainly a core distance are star edges and left to
// hdb_sparse_star_kernel.  A warp streams the upper triangle's part of a row in
// vertex order; pairs within the maxima at the root (mostly those inside one
// cluster) gather in shared memory and are settled 32 at a time.  A warp takes
// rows r and n - 1 - r, which together are one row long.  Bound by the instructions a pair takes and the latency
// of the block's read (2 n^2 bytes): with four columns a lane and load, and the
// maxima at the root in shared memory, 16 windows of 2048 points take 87 us (one
// column a lane and load: 102; 134 MB at the copy rate: 20).
// ---------------------------------------------------------------------------
template <typename Real>
__global__ void __launch_bounds__(256, 5) hdb_sparse_light_kernel(const SparseArgs a) {
    __shared__ uint32_t s_span[8][kSparseLevels];
    __shared__ float s_top[8][kSparseLevels];
    __shared__ uint2 s_pair[8][64];  // (distance, column) of pairs that may be light
    extern __shared__ __align__(16) unsigned char smem[];
    float* top_root = reinterpret_cast<float*>(smem);  // of every vertex; read by fours
    const int per = (a.nmax + kLightRows - 1) / kLightRows;
    const int item = blockIdx.x / per, j = blockIdx.x - item * per;
    const int w = a.queue[item];
    const int64_t base = a.offsets[w];
    const int n = (int)(a.offsets[w + 1] - base);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (j * kLightRows > n - 1) return;
    if (__syncthreads_or(threadIdx.x == 0 && a.flags[w])) return;  // (may be set meanwhile)
    const int levels = a.levels[w];
    const float* __restrict__ Dw = sparse_block<Real>(a, w);
    const int64_t ld = dist_ld(n);
    const SparseBound bound = sparse_bound<Real>(a, w);
    const uint16_t* __restrict__ pos = a.pos + base;
    for (int v = threadIdx.x; v < sparse_round(n); v += 256)
        top_root[v] = v < n ? a.level_max_v[(int64_t)(levels - 1) * a.T + base + v] : 0.0f;
    __syncthreads();
    const int limit = n * a.light_cap;
    uint32_t* light_uv = a.light_uv + base * a.light_cap;
    Real* light_w = static_cast<Real*>(a.light_w) + base * a.light_cap;
    uint32_t* span = s_span[warp];
    float* top = s_top[warp];
    uint2* pair = s_pair[warp];
    for (int turn = 0; turn < kLightRows / 8; ++turn) {
        const int r = j * (kLightRows / 2) + (turn >> 1) * 8 + warp;
        const int u = (turn & 1) == 0 ? r : n - 1 - r;
        if (2 * r > n - 1 || ((turn & 1) && u == r)) break;
        __syncwarp();
        if (lane < levels) {
            span[lane] = a.level_span[(int64_t)lane * a.T + base + u];
            top[lane] = a.level_max_v[(int64_t)lane * a.T + base + u];
        }
        __syncwarp();
        const float core_u = a.unit_core ? -1.0f : a.core_down[base + u];
        const float top_u = top[levels - 1];
        const float* __restrict__ row = Dw + (int64_t)u * ld;
        int waiting = 0;
        auto settle = [&](int count) {  // the first `count` waiting pairs, one a lane
            bool light = lane < count;
            const uint2 e = pair[lane];
            const float d = __uint_as_float(e.x);
            const int v = (int)e.y;
            if (light) {
                const uint32_t p = pos[v];
                int l = levels - 1;
                while (l > 0 && p >= (span[l - 1] & 0xffffu) && p < (span[l - 1] >> 16)) --l;
                light = bound.down(d) <= fmaxf(top[l], a.level_max_v[(int64_t)l * a.T + base + v]);
                if (light && !a.unit_core) light = !(bound.up(d) <= fmaxf(core_u, a.core_down[base + v]));
            }
            const unsigned bal = __ballot_sync(0xffffffffu, light);
            if (!bal) return;
            int at = 0;
            if (lane == 0) at = atomicAdd(a.light_count + w, __popc(bal));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(bal & lanemask_lt());
            if (light) {
                if (at >= limit) {
                    sparse_flag(a, w);
                } else {
                    light_uv[at] = (uint32_t)u | ((uint32_t)v << 16);
                    if (!a.approx) light_w[at] = (Real)d;  // above both cores
                }
            }
        };
        constexpr int U = 2;
        const float inf = __int_as_float(0x7f800000);
        for (int v0 = (u + 1) & ~31; v0 < n; v0 += 128 * U) {
            float4 d4[U];
#pragma unroll
            for (int q = 0; q < U; ++q) {
                const int v = v0 + 128 * q + 4 * lane;
                d4[q] = v < n ? __ldcs(reinterpret_cast<const float4*>(row + v)) : make_float4(inf, inf, inf, inf);
            }
#pragma unroll
            for (int q = 0; q < U; ++q) {
                const int v = v0 + 128 * q + 4 * lane;
                const float4 t = v < n ? *reinterpret_cast<const float4*>(top_root + v) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                const float d[4] = {d4[q].x, d4[q].y, d4[q].z, d4[q].w};
                unsigned may = 0;
                if (bound.down(d[0]) <= fmaxf(top_u, t.x)) may |= 1;
                if (bound.down(d[1]) <= fmaxf(top_u, t.y)) may |= 2;
                if (bound.down(d[2]) <= fmaxf(top_u, t.z)) may |= 4;
                if (bound.down(d[3]) <= fmaxf(top_u, t.w)) may |= 8;
                may &= (15u << min(max(u + 1 - v, 0), 4)) & (15u >> min(max(v + 4 - n, 0), 4));  // u < v + b < n
                if (!__any_sync(0xffffffffu, may)) continue;
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const unsigned bal = __ballot_sync(0xffffffffu, may >> b & 1);
                    if (!bal) continue;
                    if (may >> b & 1)
                        pair[waiting + __popc(bal & lanemask_lt())] = make_uint2(__float_as_uint(d[b]), v + b);
                    waiting += __popc(bal);
                    __syncwarp();
                    if (waiting >= 32) {
                        settle(32);
                        waiting -= 32;
                        const uint2 rest = pair[32 + lane];
                        __syncwarp();
                        if (lane < waiting) pair[lane] = rest;
                        __syncwarp();
                    }
                }
            }
        }
        settle(waiting);
    }
}

// ---------------------------------------------------------------------------
// Stars: of each point x, the list entries u whose edge weighs core_x
// (d <= core_x, and u's core smaller, or equal with u < x so that the edge has
// one owner).  All are kept as a mask over the list, for the sources.  The order
// needs one edge per component below core_x: x is alone below core_x, and a
// component that Prim has entered is finished before an edge of core_x is
// taken; entering from x, the lowest vertex comes first.  So of entries that T'
// joins below core_x (neighbours in leaf order, a sufficient test) only the
// lowest vertex is emitted.  One warp a point.
// ---------------------------------------------------------------------------
template <typename Real>
__global__ void __launch_bounds__(256) hdb_sparse_star_kernel(const SparseArgs a) {
    const int per = (a.nmax + kSparseRowsCta - 1) / kSparseRowsCta;
    const int item = blockIdx.x / per, r0 = (blockIdx.x - item * per) * kSparseRowsCta;
    const int w = a.queue[item];
    const int64_t base = a.offsets[w];
    const int n = (int)(a.offsets[w + 1] - base);
    if (r0 >= n || a.flags[w]) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int levels = a.levels[w];
    const int keep = min(a.keep, n);
    const SparseBound bound = sparse_bound<Real>(a, w);
    const Real* __restrict__ core = static_cast<const Real*>(a.core) + base;
    const int limit = n * a.star_cap;
    for (int r = warp; r < kSparseRowsCta; r += 8) {
        const int x = r0 + r;
        if (x >= n) break;  // warp-uniform
        const Real core_x = core[x];
        const float down_x = a.core_down[base + x];
        unsigned long long members = 0;
        for (int h = 0; h < keep; h += 32) {
            const int t = h + lane;
            uint32_t key = 0xffffffffu;
            if (t < keep) {
                const int u = a.knn_idx[(base + x) * a.list + t];
                if (u != x && bound.up(a.knn_d[(base + x) * a.list + t]) <= down_x) {
                    const Real core_u = core[u];
                    if (core_u < core_x || (core_u == core_x && u < x))
                        key = ((uint32_t)a.pos[base + u] << 12) | (uint32_t)u;
                }
            }
            const unsigned in = __ballot_sync(0xffffffffu, key != 0xffffffffu);
            members |= (unsigned long long)in << h;
            if (!in) continue;
            // Entries in leaf order.
#pragma unroll
            for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
                for (int j = k >> 1; j > 0; j >>= 1) {
                    const uint32_t other = __shfl_xor_sync(0xffffffffu, key, j);
                    const bool keep_min = ((lane & k) == 0) == ((lane & j) == 0);
                    key = keep_min ? min(key, other) : max(key, other);
                }
            }
            const uint32_t before = __shfl_up_sync(0xffffffffu, key, 1);
            const bool valid = key != 0xffffffffu;
            bool joined = false;  // to the entry before, below core_x
            if (valid && lane > 0) {
                const int64_t p = base + (before & 0xfffu), q = base + (key & 0xfffu);
                const uint32_t place = key >> 12;
                int l = 0;  // first round that joins them (the entry before lies to the left)
                while (l + 1 < levels && place >= (a.level_span[(int64_t)l * a.T + p] >> 16)) ++l;
                joined = fmaxf(a.level_max_v[(int64_t)l * a.T + p], a.level_max_v[(int64_t)l * a.T + q]) < down_x;
            }
            // Lowest vertex of each run of joined entries.
            uint32_t low = key & 0xfffu;
            const unsigned heads = __ballot_sync(0xffffffffu, valid && !joined);
            const int head = 31 - __clz(heads & ((2u << lane) - 1u));  // lane 0 is a head whenever any lane is valid
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, low, o);
                if (lane - o >= head) low = min(low, y);
            }
            const unsigned valid_mask = __ballot_sync(0xffffffffu, valid);
            const bool last = valid && (lane == 31 || !((valid_mask >> (lane + 1)) & 1u) || ((heads >> (lane + 1)) & 1u));
            const unsigned emit = __ballot_sync(0xffffffffu, last);
            int at = 0;
            if (lane == 0) at = atomicAdd(a.star_count + w, __popc(emit));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(emit & lanemask_lt());
            if (last) {
                if (at >= limit) sparse_flag(a, w);
                else a.star_uv[base * a.star_cap + at] = (uint32_t)x | (low << 16);
            }
        }
        if (lane == 0) a.star_mask[base + x] = members;
    }
}

// Exact weights of the light edges (bounded distances).
constexpr int kWeightsPerWindow = 8;  // CTAs of 128 threads sharing a window's edges

template <typename Real>
__global__ void __launch_bounds__(128) hdb_sparse_weights_kernel(const SparseArgs a) {
    using T = RealTraits<Real>;
    const int item = blockIdx.x / kWeightsPerWindow, part = blockIdx.x - item * kWeightsPerWindow;
    const int w = a.queue[item];
    if (a.flags[w]) return;
    const int64_t base = a.offsets[w];
    const int D = a.D;
    const int count = a.light_count[w];
    const Real* __restrict__ X = static_cast<const Real*>(a.X) + base * D;
    const Real* core = static_cast<const Real*>(a.core);
    Real* light_w = static_cast<Real*>(a.light_w) + base * a.light_cap;
    for (int e = part * 128 + threadIdx.x; e < count; e += 128 * kWeightsPerWindow) {
        const uint32_t uv = a.light_uv[base * a.light_cap + e];
        const int u = uv & 0xffff, v = uv >> 16;
        Real d = sparse_exact<Real>(X + (int64_t)u * D, X + (int64_t)v * D, D);
        if (!a.unit_core) d = T::vmax(T::vmax(core[base + u], core[base + v]), d);
        light_w[e] = d;
    }
}

// ---------------------------------------------------------------------------
// Prim and the hierarchy: one CTA a window.
//  1. Boruvka over the light and star edges gives the weights of the minimum
//     spanning trees; sorted, they turn weights into ranks.  An edge whose
//     weight is none of them lies in no minimum spanning tree and is dropped.
//  2. The rest become adjacency rows of packed (rank, vertex) words in shared
//     memory (in the workspace when they do not fit).
//  3. One warp runs Prim over them (sparse_prim_warp): vertices are split over
//     the lanes in 32 blocks, a lane keeps its block's least word.
//  4. Sources, then the hierarchy stages as in the dense form (the sort on all
//     warps).
// Shared memory: the arena (r0 weights, r1 sorted weights, s0 ranks then
// sources, s1 order; row starts and best words in r2, and s2/s3 for float32;
// adjacency behind them to the arena's end and on).
// ---------------------------------------------------------------------------
template <typename Real> struct SparsePrimLayout {
    // Adjacency words per point that prim_smem provides.
    static constexpr int kAdj = 5;
    __host__ __device__ static size_t adj_offset(int n) {
        const size_t cap = (size_t)Arena<Real>::round_cap(n);
        return 3 * cap * sizeof(Real) + cap * 2 * (sizeof(Real) == 4 ? 4 : 2);
    }
    __host__ __device__ static size_t bytes(int n) {
        const size_t need = adj_offset(n) + (size_t)n * kAdj * sizeof(uint32_t);
        return need > Arena<Real>::bytes(n) ? need : Arena<Real>::bytes(n);
    }
};

// A word is rank << 14 | vertex << 2 (the vertex as a byte offset).  As a
// signed number kWordIn is below every word (no update passes), as an unsigned
// one above all (no minimum).
constexpr uint32_t kWordIn = 0xffffffffu;         // in the tree
constexpr uint32_t kWordUnreached = 0x7fffffffu;  // above every word
__device__ __forceinline__ uint32_t prim_word(uint32_t rank, uint32_t vertex) { return (rank << 14) | (vertex << 2); }
__device__ __forceinline__ uint32_t word_offset(uint32_t word) { return word & 0x3ffcu; }

// Shared-memory accesses in program order, predicated instead of branched
// around: the warp never diverges inside a step.
__device__ __forceinline__ uint32_t shared_address(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ uint32_t lds32(uint32_t at) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(at));
    return v;
}
__device__ __forceinline__ uint32_t lds32_if(bool p, uint32_t at, uint32_t other) {
    uint32_t v = other;
    asm volatile("{ .reg .pred p; setp.ne.u32 p, %2, 0; @p ld.shared.u32 %0, [%1]; }" : "+r"(v) : "r"(at), "r"((uint32_t)p));
    return v;
}
__device__ __forceinline__ void sts32_if(bool p, uint32_t at, uint32_t v) {
    asm volatile("{ .reg .pred p; setp.ne.u32 p, %2, 0; @p st.shared.u32 [%0], %1; }" ::"r"(at), "r"(v), "r"((uint32_t)p));
}
__device__ __forceinline__ void sts16_if(bool p, uint32_t at, uint32_t v) {
    asm volatile("{ .reg .pred p; setp.ne.u32 p, %2, 0; @p st.shared.u16 [%0], %1; }" ::"r"(at), "h"((unsigned short)v),
                 "r"((uint32_t)p));
}
__device__ __forceinline__ void reds_min_if(bool p, uint32_t at, uint32_t v) {
    asm volatile("{ .reg .pred p; setp.ne.u32 p, %2, 0; @p red.shared.min.u32 [%0], %1; }" ::"r"(at), "r"(v),
                 "r"((uint32_t)p));
}

// A step is bound by its chain: redux -> row start -> words -> best of the
// neighbours -> redux.  The next vertex is the least of the lanes' block minima
// and of this step's own updates, so the updates need not reach their blocks
// within the step: they go to `mail` (32 words, one per block: the least update
// since the block's last rescan), read in the shadow of the next step's loads,
// as is the rescan of the block that the last vertex left.  BL: words of a
// block a lane rescans (a block is 32 * BL vertices).  Measured on synthetic
// sparse graphs of degree 4: 253 / 261 / 265 cycles a step for BL = 1 / 2 / 4;
// with the updates handed over by shuffles 633 to 655, by the mailbox within
// the step 377 to 392.
template <int BL, bool kOnChip>
__device__ __forceinline__ bool sparse_prim_warp(int n, uint32_t start, uint32_t best, uint32_t adj,
                                                 const uint32_t* adj_off, uint32_t order, uint32_t rank, uint32_t mail) {
    constexpr int kShift = (BL == 1 ? 5 : (BL == 2 ? 6 : 7)) + 2;  // of byte offsets
    static_assert((32 << kShift) == 4096 * BL, "32 blocks of 32 * BL vertices");
    const uint32_t lane = threadIdx.x & 31, end = 4u * (uint32_t)n;
    const uint32_t mine = mail + 4 * lane;
    uint32_t least = (lane << kShift) < end ? kWordUnreached : kWordIn;
    sts32_if(true, mine, 0xffffffffu);
    uint32_t cur = 0;
    bool ok = true;
    auto words_at = [&](uint32_t first, uint32_t i, uint32_t count) {
        if constexpr (kOnChip) return lds32_if(i < count, adj + 4 * (first + i), kWordUnreached);
        return i < count ? adj_off[first + i] : kWordUnreached;
    };
    for (int it = 0; it < n - 1; ++it) {
        const uint32_t own = cur >> kShift;
        const uint32_t row = lds32(start + cur);  // first word << 12 | count
        sts32_if(lane == 0, best + cur, kWordIn);
        const uint32_t post = lds32(mine);
        uint32_t block[BL];
#pragma unroll
        for (int j = 0; j < BL; ++j) {
            const uint32_t v = (own << kShift) + 128 * j + 4 * lane;
            block[j] = lds32_if(v < end, best + v, kWordIn);
        }
        const uint32_t count = row & 0xfffu, first = row >> 12;
        uint32_t word = words_at(first, lane, count);
        least = min(least, post);
        uint32_t rest = block[0];
#pragma unroll
        for (int j = 1; j < BL; ++j) rest = min(rest, block[j]);
        rest = __reduce_min_sync(0xffffffffu, rest);
        uint32_t b = lds32_if(lane < count, best + word_offset(word), 0u);
        sts32_if(lane == own, mine, 0xffffffffu);
        if (lane == own) least = rest;
        bool lower = (int)word < (int)b;  // strict: an equal older edge stays
        uint32_t update = lower ? word : 0xffffffffu;
        sts32_if(lower, best + word_offset(word), word);
        reds_min_if(lower, mail + 4 * (word_offset(word) >> kShift), word);
        for (uint32_t e = 32; e < count; e += 32) {
            word = words_at(first, e + lane, count);
            b = lds32_if(e + lane < count, best + word_offset(word), 0u);
            lower = (int)word < (int)b;
            if (lower) update = min(update, word);
            sts32_if(lower, best + word_offset(word), word);
            reds_min_if(lower, mail + 4 * (word_offset(word) >> kShift), word);
        }
        const uint32_t next = __reduce_min_sync(0xffffffffu, min(least, update));
        ok = ok && next < kWordUnreached;  // else not connected: every vertex left is unreached
        cur = word_offset(next) < end ? word_offset(next) : 0;
        sts16_if(lane == 0, order + 2 * it, cur >> 2);
        sts16_if(lane == 0, rank + 2 * it, next >> 14);
    }
    __syncwarp();
    return ok;
}

template <bool kOnChip>
__device__ __forceinline__ bool sparse_prim(int n, const uint32_t* start, const uint32_t* best, const uint32_t* adj,
                                            const uint32_t* adj_off, const int16_t* order, const int16_t* rank,
                                            const uint32_t* mail) {
    const uint32_t s = shared_address(start), b = shared_address(best), a = shared_address(adj),
                   o = shared_address(order), r = shared_address(rank), m = shared_address(mail);
    if (n <= 1024) return sparse_prim_warp<1, kOnChip>(n, s, b, a, adj_off, o, r, m);
    if (n <= 2048) return sparse_prim_warp<2, kOnChip>(n, s, b, a, adj_off, o, r, m);
    return sparse_prim_warp<4, kOnChip>(n, s, b, a, adj_off, o, r, m);
}

template <typename Real>
__global__ void __launch_bounds__(512) hdb_sparse_prim_kernel(const SparseArgs a, const __grid_constant__ ForwardArgs f) {
    using T = RealTraits<Real>;
    using Key = typename T::Bits;
    constexpr bool kWide = sizeof(Real) == 8;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t s_scan[33];
    __shared__ int s_ctr[4];
    __shared__ int s_edges;
    __shared__ int s_ok;
    const int w = a.queue[blockIdx.x];
    if (a.flags[w]) return;
    const int64_t base = a.offsets[w];
    const int n = (int)(a.offsets[w + 1] - base);
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
    Arena<Real> ar = Arena<Real>::carve(smem, n);
    const int cap = Arena<Real>::round_cap(n);
    if (f.stage_ns && tid == 0) f.stage_ns[8 * w + 0] = global_ns();
    const int n_light = a.light_count[w], n_star = a.unit_core ? 0 : a.star_count[w];
    const int m = n_light + n_star;
    const uint32_t* __restrict__ light_uv = a.light_uv + base * a.light_cap;
    const Real* __restrict__ light_w = static_cast<const Real*>(a.light_w) + base * a.light_cap;
    const uint32_t* __restrict__ star_uv = a.star_uv + base * a.star_cap;
    const Real* __restrict__ core = static_cast<const Real*>(a.core) + base;
    uint16_t* edge_rank = a.edge_rank + base * (a.light_cap + a.star_cap);
    auto edge = [&](int e, int& u, int& v, Key& key) {
        const uint32_t uv = e < n_light ? light_uv[e] : star_uv[e - n_light];
        u = (int)(uv & 0xffff);
        v = (int)(uv >> 16);
        key = T::key(e < n_light ? light_w[e] : core[u]);
    };
    // ---- 1. minimum spanning tree weights ---------------------------------------
    // Choice of a component: its least (weight, ends); float32 in one 64-bit word.
    unsigned long long* choice = reinterpret_cast<unsigned long long*>(ar.r1);
    uint32_t* choice_uv = reinterpret_cast<uint32_t*>(ar.r2);  // float64 only
    uint16_t* comp = reinterpret_cast<uint16_t*>(ar.s2);
    uint16_t* up = reinterpret_cast<uint16_t*>(ar.s3);
    for (int v = tid; v < n; v += nt) comp[v] = (uint16_t)v;
    if (tid == 0) s_edges = 0;
    for (int round = 0; round < kSparseLevels; ++round) {
        for (int v = tid; v < n; v += nt) {
            choice[v] = kNoChoice;
            if (kWide) choice_uv[v] = 0xffffffffu;
        }
        __syncthreads();
        for (int e = tid; e < m; e += nt) {
            int u, v;
            Key key;
            edge(e, u, v, key);
            const int cu = comp[u], cv = comp[v];
            if (cu == cv) continue;
            unsigned long long word = key;
            if (!kWide) word = (word << 32) | ((uint32_t)min(u, v) << 12) | (uint32_t)max(u, v);
            if (word < choice[cu]) atomicMin(&choice[cu], word);
            if (word < choice[cv]) atomicMin(&choice[cv], word);
        }
        __syncthreads();
        if (kWide) {
            for (int e = tid; e < m; e += nt) {
                int u, v;
                Key key;
                edge(e, u, v, key);
                const int cu = comp[u], cv = comp[v];
                if (cu == cv) continue;
                const uint32_t ends = ((uint32_t)min(u, v) << 12) | (uint32_t)max(u, v);
                if (choice[cu] == (unsigned long long)key) atomicMin(&choice_uv[cu], ends);
                if (choice[cv] == (unsigned long long)key) atomicMin(&choice_uv[cv], ends);
            }
            __syncthreads();
        }
        for (int r = tid; r < n; r += nt) {
            if (comp[r] != r) continue;
            const unsigned long long word = choice[r];
            int to = r;
            if (word != kNoChoice) {
                const uint32_t ends = kWide ? choice_uv[r] : (uint32_t)word;
                const int lo = comp[(ends >> 12) & 0xfff], hi = comp[ends & 0xfff];
                to = lo == r ? hi : lo;
                if (choice[to] == word && (!kWide || choice_uv[to] == ends) && r < to) to = r;
                if (to != r) ar.r0[min(atomicAdd(&s_edges, 1), n - 1)] = T::from_key((Key)(kWide ? word : word >> 32));
            }
            up[r] = (uint16_t)to;
        }
        __syncthreads();
        for (int v = tid; v < n; v += nt) comp[v] = (uint16_t)sparse_root(up, comp[v], n);
        const int found = s_edges;
        __syncthreads();
        if (found >= n - 1) break;
    }
    if (s_edges != n - 1) {  // the light and star edges hold a spanning tree: unreachable
        if (tid == 0) sparse_flag(a, w);
        return;
    }
    Key* sorted = reinterpret_cast<Key*>(ar.r1);
    __syncthreads();
    for (int i = tid; i < n - 1; i += nt) sorted[i] = T::key(ar.r0[i]);
    __syncthreads();
    bitonic_cta<Key>(sorted, n - 1);
    bool twin = false;
    for (int i = tid; i + 1 < n - 1; i += nt) twin |= key_eq(sorted[i], sorted[i + 1]);
    const bool distinct = !__syncthreads_or(twin);
    // ---- 2. adjacency -----------------------------------------------------------
    uint32_t* start = reinterpret_cast<uint32_t*>(ar.r2);
    uint32_t* best = kWide ? start + cap : reinterpret_cast<uint32_t*>(ar.s2);
    uint32_t* adj = reinterpret_cast<uint32_t*>(smem + SparsePrimLayout<Real>::adj_offset(n));
    for (int v = tid; v < n; v += nt) best[v] = 0;  // degrees
    __syncthreads();
    for (int e = tid; e < m; e += nt) {
        int u, v;
        Key key;
        edge(e, u, v, key);
        int lo = 0, hi = n - 1;  // first sorted weight not below this edge's
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (key_lt(sorted[mid], key)) lo = mid + 1; else hi = mid;
        }
        const bool in = lo < n - 1 && key_eq(sorted[lo], key);
        edge_rank[e] = in ? (uint16_t)lo : (uint16_t)0xffff;
        if (in) {
            atomicAdd(&best[u], 1u);
            atomicAdd(&best[v], 1u);
        }
    }
    __syncthreads();
    // Exclusive scan of the degrees: a contiguous run of vertices a thread.
    const int run = (n + nt - 1) / nt;
    uint32_t sum = 0;
    for (int v = tid * run; v < min(n, (tid + 1) * run); ++v) sum += best[v];
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_scan[warp] = incl;
    __syncthreads();
    uint32_t before = 0, total = 0;
    for (int j = 0; j < (nt >> 5); ++j) {
        if (j < warp) before += s_scan[j];
        total += s_scan[j];
    }
    before += incl - sum;
    for (int v = tid * run; v < min(n, (tid + 1) * run); ++v) {
        const uint32_t d = best[v];
        start[v] = (before << 12) | d;
        best[v] = before;  // next free word
        before += d;
    }
    const bool on_chip = total <= (uint32_t)(n * SparsePrimLayout<Real>::kAdj);
    uint32_t* adj_off = a.adj + 2 * base * (a.light_cap + a.star_cap);
    __syncthreads();
    for (int e = tid; e < m; e += nt) {
        const uint32_t r = edge_rank[e];
        if (r == 0xffffu) continue;
        const uint32_t uv = e < n_light ? light_uv[e] : star_uv[e - n_light];
        const uint32_t u = uv & 0xffff, v = uv >> 16;
        const uint32_t at_u = atomicAdd(&best[u], 1u), at_v = atomicAdd(&best[v], 1u);
        if (on_chip) {
            adj[at_u] = prim_word(r, v);
            adj[at_v] = prim_word(r, u);
        } else {
            adj_off[at_u] = prim_word(r, v);
            adj_off[at_v] = prim_word(r, u);
        }
    }
    __syncthreads();
    for (int v = tid; v < n; v += nt) best[v] = kWordUnreached;
    __syncthreads();
    if (f.stage_ns && tid == 0) f.stage_ns[8 * w + 1] = global_ns();
    // ---- 3. order ---------------------------------------------------------------
    if (warp == 0) {
        const bool ok = on_chip ? sparse_prim<true>(n, start, best, adj, adj_off, ar.s1, ar.s0, s_scan)
                                : sparse_prim<false>(n, start, best, adj, adj_off, ar.s1, ar.s0, s_scan);
        if (lane == 0) s_ok = ok;
    }
    __syncthreads();
    if (!s_ok) {  // unreachable, as above
        if (tid == 0) sparse_flag(a, w);
        return;
    }
    // ---- 4. sources: the first visited end of an edge of the vertex's weight --------
    uint32_t* place = best;     // position << 12 | rank of each vertex's edge
    uint32_t* source = start;   // position of its source
    for (int v = tid; v < n; v += nt) source[v] = 0xffffu;
    if (tid == 0) place[0] = 0xfffu;  // the start has no edge
    for (int i = tid; i < n - 1; i += nt)
        place[ar.s1[i]] = ((uint32_t)(i + 1) << 12) | (uint32_t)(uint16_t)ar.s0[i];
    __syncthreads();
    for (int e = tid; e < n_light; e += nt) {
        const uint32_t r = edge_rank[e];
        if (r == 0xffffu) continue;
        const uint32_t uv = light_uv[e];
        const uint32_t u = uv & 0xffff, v = uv >> 16;
        const uint32_t pu = place[u], pv = place[v];
        const bool forward = pu < pv;
        if (((forward ? pv : pu) & 0xfffu) == r) atomicMin(&source[forward ? v : u], (forward ? pu : pv) >> 12);
    }
    if (!a.unit_core) {
        for (int x = tid; x < n; x += nt) {
            unsigned long long members = a.star_mask[base + x];
            const Key key = T::key(core[x]);
            const uint32_t px = place[x];
            while (members) {
                const int t = __ffsll((long long)members) - 1;
                members &= members - 1;
                const int u = a.knn_idx[(base + x) * a.list + t];
                const uint32_t pu = place[u];
                const bool forward = px < pu;  // x first: it may be u's source
                const uint32_t r = (forward ? pu : px) & 0xfffu;
                if (r != 0xfffu && key_eq(sorted[r], key)) atomicMin(&source[forward ? u : x], (forward ? px : pu) >> 12);
            }
        }
    }
    __syncthreads();
    bool lost = false;
    for (int i = tid; i < n - 1; i += nt) {
        const uint32_t p = source[ar.s1[i]];
        lost |= p > (uint32_t)i;
        if (distinct) ar.s2[ar.s0[i]] = (int16_t)i;
        else ar.s2[i] = ar.s0[i];
        ar.r0[i] = T::from_key(sorted[ar.s0[i]]);
        ar.s0[i] = p == 0 || p > (uint32_t)i ? (int16_t)0 : ar.s1[p - 1];
    }
    if (__syncthreads_or(lost)) {  // unreachable: every vertex has a source
        if (tid == 0) sparse_flag(a, w);
        return;
    }
    if (f.stage_ns && tid == 0) f.stage_ns[8 * w + 2] = global_ns();
    tree_window_cta<Real>(f, smem, w, n, distinct ? EdgeOrder::kSorted : EdgeOrder::kRanks, s_scan, s_ctr, kBarHelp);
}

}  // namespace hdb
