// Small windows (at most kSmallMax points) from points to labels in one kernel,
// one CTA a window, everything in shared memory: exact distances, core
// distances, Prim by one warp over the distance rows, then the CTA's hierarchy
// (hdb_tree_cta.cuh).  Replaces hdbscan_gpu/_cuda.py:91-128 for such windows.
//
// A small window is a chain of short stages; as separate launches (distances,
// cores, Prim and hierarchy, or the dozen of the sparse path) their latencies and
// the launches' add up.  Bound by shared-memory latency; other windows' CTAs on
// the SM fill in.
#pragma once
#include "hdb_common.cuh"
#include "hdb_distance.cuh"
#include "hdb_forward.cuh"
#include "hdb_tree_cta.cuh"

namespace hdb {

constexpr int kSmallMax = 128;

template <typename Real> struct SmallLayout {
    static constexpr int kChunk = sizeof(Real) == 4 ? 32 : 16;  // coordinates staged at a time
    __host__ __device__ static int ld(int n) { return n | 1; }   // odd: rows and columns spread over the banks
    __host__ __device__ static size_t matrix(int n) { return ((size_t)n * ld(n) * sizeof(Real) + 127) & ~size_t(127); }
    __host__ __device__ static size_t bytes(int n) {
        const size_t stage = (size_t)n * (kChunk + 1) * sizeof(Real);
        const size_t arena = Arena<Real>::bytes(n);
        return matrix(n) + (stage > arena ? stage : arena);
    }
};

// Ascending (key, index) bitonic sort of 32 * E elements, p = lane + 32 h.
template <int E, typename Key>
__device__ __forceinline__ void sort_row(Key (&k)[E], int (&i)[E]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int size = 2; size <= 32 * E; size <<= 1) {
#pragma unroll
        for (int j = size >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
#pragma unroll
                for (int h = 0; h < E; ++h) {
                    const int o = h ^ (j >> 5);
                    if (o < h) continue;
                    const bool up = ((32 * h) & size) == 0;
                    const bool swap = (key_lt(k[o], k[h]) || (key_eq(k[o], k[h]) && i[o] < i[h])) == up;
                    const Key a = k[h], b = k[o];
                    const int x = i[h], y = i[o];
                    k[h] = key_select(swap, b, a); k[o] = key_select(swap, a, b);
                    i[h] = swap ? y : x; i[o] = swap ? x : y;
                }
            } else {
#pragma unroll
                for (int h = 0; h < E; ++h) {
                    const Key pk = shfl_key_xor(k[h], j);
                    const int pi = __shfl_xor_sync(0xffffffffu, i[h], j);
                    const bool less = key_lt(pk, k[h]) || (key_eq(pk, k[h]) && pi < i[h]);
                    const bool keep_min = (((lane + 32 * h) & size) == 0) == ((lane & j) == 0);
                    const bool take = keep_min ? less : !less;
                    k[h] = key_select(take, pk, k[h]);
                    i[h] = take ? pi : i[h];
                }
            }
        }
    }
}

// Core distances of all rows, a warp a row: the ms-th smallest (value, index), for
// few neighbours by taking minima, else from the sorted row.
constexpr int kSmallMinima = 16;

template <typename Real, int E>
__device__ __forceinline__ void small_cores(const Real* dist, int ld, int n, int ms, Real* core, Real* core_g, int32_t* nbr_g) {
    using T = RealTraits<Real>;
    using Key = typename T::Bits;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int r = warp; r < n; r += nw) {
        Key k[E];
        int i[E];
#pragma unroll
        for (int h = 0; h < E; ++h) {
            const int j = lane + 32 * h;
            k[h] = j < n ? T::key(dist[r * ld + j]) : (Key)~(Key)0;
            i[h] = j;
        }
        if (ms <= kSmallMinima) {
            Key value = 0;
            uint32_t index = 0;
            for (int t = 0; t < ms; ++t) {
                Key least = (Key)~(Key)0;
                uint32_t at = 0xffffffffu;
#pragma unroll
                for (int h = 0; h < E; ++h)
                    if (key_idx_lt(k[h], (uint32_t)i[h], least, at)) { least = k[h]; at = (uint32_t)i[h]; }
                warp_argmin(least, at);
                value = least;
                index = at;
#pragma unroll
                for (int h = 0; h < E; ++h)
                    if ((uint32_t)i[h] == at) k[h] = (Key)~(Key)0;
            }
            if (lane == 0) {
                core[r] = T::from_key(value);
                core_g[r] = T::from_key(value);
                nbr_g[r] = (int)index;
            }
            continue;
        }
        sort_row<E>(k, i);
#pragma unroll
        for (int h = 0; h < E; ++h)
            if (lane + 32 * h == ms - 1) {
                const Real v = T::from_key(k[h]);
                core[r] = v;
                core_g[r] = v;
                nbr_g[r] = i[h];
            }
    }
}

// Prim by one warp (reference _kernels.py:164-320): lane holds vertices lane + 32 h.
template <typename Real, int E>
__device__ __forceinline__ bool small_prim(const Real* dist, int ld, int n, const Real* core, const Arena<Real>& a) {
    using T = RealTraits<Real>;
    using Key = typename T::Bits;
    constexpr Key kIn = (Key)~(Key)0;
    const int lane = threadIdx.x & 31;
    Real best[E], mine[E];
    int source[E];
    bool out[E];
#pragma unroll
    for (int h = 0; h < E; ++h) {
        const int v = lane + 32 * h;
        best[h] = T::inf();
        source[h] = 1;  // reference initial source (_kernels.py:167)
        out[h] = v < n && v != 0;
        mine[h] = core && v < n ? core[v] : Real(0);
    }
    int cur = 0;
    for (int it = 0; it < n - 1; ++it) {
        const Real* row = dist + cur * ld;
        const Real core_cur = core ? core[cur] : Real(0);
        Key key = kIn;
        uint32_t index = 0xffffffffu;
#pragma unroll
        for (int h = 0; h < E; ++h) {
            const int v = lane + 32 * h;
            if (v < n) {
                const Real wgt = T::vmax(T::vmax(core_cur, mine[h]), row[v]);
                if (out[h] && T::lt(wgt, best[h])) { best[h] = wgt; source[h] = cur; }  // strict: the older source stays
                const Key k = out[h] ? T::key(best[h]) : kIn;
                if (key_lt(k, key)) { key = k; index = (uint32_t)v; }  // ascending vertices
            }
        }
        warp_argmin(key, index);
        const int next = (int)index;
        if (next < 0 || next >= n) return false;  // unreachable: a vertex outside the tree always remains
#pragma unroll
        for (int h = 0; h < E; ++h)
            if (lane + 32 * h == next) {
                a.s0[it] = (int16_t)source[h];
                a.s1[it] = (int16_t)next;
                a.r0[it] = best[h];
                out[h] = false;
            }
        cur = next;
    }
    return true;
}

template <typename Real>
__global__ void __launch_bounds__(256) hdb_small_kernel(const __grid_constant__ ForwardArgs f, const SmallArgs s) {
    using T = RealTraits<Real>;
    constexpr int KC = SmallLayout<Real>::kChunk;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ Real s_core[kSmallMax];
    __shared__ uint32_t s_scan[33];
    __shared__ int s_ctr[4];
    __shared__ int s_ok;
    const int w = f.queue[blockIdx.x];
    const int64_t base = f.offsets[w];
    const int n = (int)(f.offsets[w + 1] - base);
    const int D = f.D;
    const int tid = threadIdx.x, nt = blockDim.x, warp = tid >> 5;
    const Real* __restrict__ X = static_cast<const Real*>(f.X) + base * D;
    const int ld = SmallLayout<Real>::ld(n);
    Real* dist = reinterpret_cast<Real*>(smem);
    unsigned char* rest = smem + SmallLayout<Real>::matrix(n);
    Real* x = reinterpret_cast<Real*>(rest);  // [n][KC + 1], until the arena takes its place
    if (f.stage_ns && tid == 0) f.stage_ns[8 * w + 0] = global_ns();
    // ---- distances: 4x4 pairs a thread over the upper triangle -------------------
    const int nb = (n + 3) >> 2, blocks = nb * (nb + 1) / 2;
    int bad = 0;
    for (int k0 = 0; k0 < D; k0 += KC) {
        const int width = min(KC, D - k0);
        __syncthreads();
        for (int t = tid; t < n * width; t += nt) {
            const int i = t / width, k = t - i * width;
            const Real v = X[(int64_t)i * D + k0 + k];
            bad |= !isfinite(v);
            x[i * (KC + 1) + k] = v;
        }
        __syncthreads();
        for (int t = tid; t < blocks; t += nt) {
            int bj = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
            while (bj * (bj + 1) / 2 > t) --bj;
            while ((bj + 1) * (bj + 2) / 2 <= t) ++bj;
            const int i0 = 4 * (t - bj * (bj + 1) / 2), j0 = 4 * bj;
            Real acc[4][4];
            int pi[4], pj[4];
#pragma unroll
            for (int p = 0; p < 4; ++p) { pi[p] = min(i0 + p, n - 1); pj[p] = min(j0 + p, n - 1); }
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[p][q] = k0 > 0 ? dist[pi[p] * ld + pj[q]] : Real(0);
            for (int k = 0; k < width; ++k) {
                Real xi[4], xj[4];
#pragma unroll
                for (int p = 0; p < 4; ++p) { xi[p] = x[pi[p] * (KC + 1) + k]; xj[p] = x[pj[p] * (KC + 1) + k]; }
#pragma unroll
                for (int p = 0; p < 4; ++p)
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const Real delta = T::sub(xi[p], xj[q]);
                        acc[p][q] = T::add(acc[p][q], T::mul(delta, delta));
                    }
            }
            const bool last = k0 + KC >= D;
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (i0 + p >= n || j0 + q >= n || i0 + p > j0 + q) continue;
                    Real d = acc[p][q];
                    if (last) {
                        d = T::sqrt_rn(d);
                        bad |= (d <= T::kMax) ? 0 : 2;
                        dist[(j0 + q) * ld + i0 + p] = d;
                    }
                    dist[(i0 + p) * ld + j0 + q] = d;
                }
        }
    }
    const int nonfinite = __syncthreads_or(bad & 1), overflow = __syncthreads_or(bad & 2);
    if (nonfinite || overflow) {
        if (tid == 0) atomic_status(f.status, nonfinite ? kNonFinite : kOverflow);
        for (int j = tid; j < n; j += nt) f.labels[base + j] = -1;
        return;
    }
    // ---- cores, Prim --------------------------------------------------------------
    const Real* core = nullptr;
    if (!f.unit_core) {
        Real* core_g = static_cast<Real*>(s.core) + base;
        int32_t* nbr_g = s.core_nbr + base;
        if (n <= 32) small_cores<Real, 1>(dist, ld, n, s.ms, s_core, core_g, nbr_g);
        else if (n <= 64) small_cores<Real, 2>(dist, ld, n, s.ms, s_core, core_g, nbr_g);
        else small_cores<Real, 4>(dist, ld, n, s.ms, s_core, core_g, nbr_g);
        __syncthreads();
        core = s_core;
    }
    if (f.stage_ns && tid == 0) f.stage_ns[8 * w + 1] = global_ns();
    const Arena<Real> a = Arena<Real>::carve(rest, n);
    if (warp == 0) {
        const bool ok = n <= 32 ? small_prim<Real, 1>(dist, ld, n, core, a)
                                : (n <= 64 ? small_prim<Real, 2>(dist, ld, n, core, a)
                                           : (n <= 96 ? small_prim<Real, 3>(dist, ld, n, core, a)
                                                      : small_prim<Real, 4>(dist, ld, n, core, a)));
        if (tid == 0) s_ok = ok;
    }
    __syncthreads();
    if (f.stage_ns && tid == 0) f.stage_ns[8 * w + 2] = global_ns();
    if (!s_ok) {
        if (tid == 0) atomic_status(f.status, kInternal);
        for (int j = tid; j < n; j += nt) f.labels[base + j] = -1;
        return;
    }
    // A tree of few nodes is done by one warp before the CTA's barriers add up.
    if (n > kHelpMinEdges) tree_window_cta<Real>(f, rest, w, n, EdgeOrder::kNone, s_scan, s_ctr, kBarHelp);
    else if (warp == 0) tree_window<Real>(f, rest, w, n);
}

}  // namespace hdb
