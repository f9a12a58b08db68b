// Hierarchy stages of one window by a whole CTA (hdb_tree.cuh has the one-warp
// form; results are the same bit for bit, the arena is the same).
//
// Linkage without a union-find: at any weight the components of Prim's sequence
// are its maximal runs of smaller weights, because Prim finishes a component
// before it takes an edge of larger weight.  So the merge tree is the Cartesian
// tree of the sequence by sorted position: a node hangs in the gap between the
// nearest larger entries on both sides.  Only edges of equal weight with
// nothing larger between them (a tie run) may connect other pieces than the
// neighbouring ones; the pieces of such a run (found the same way) are joined
// by a small union-find, one thread a weight.
//
// Condensation without the level-by-level queue: depths and left-to-right
// offsets come from pointer doubling; the breadth-first order of the splits is
// their order by (depth, offset), which numbers the clusters; each cluster is a
// path, laid out by depth, whose stability one thread sums in the reference's
// order.
//
// Bound by shared-memory latency over a few hundred barriers.
#pragma once
#include "hdb_common.cuh"
#include "hdb_tree.cuh"

namespace hdb {

constexpr int kTieRunMax = 128;  // larger groups of equal weights go to the one-warp union-find

// Ascending bitonic sort of k[0..n) by the CTA.  Every comparator puts the
// smaller word at the lower index (each merge starts by mirroring its second
// half), so entries past n count as largest and stay where they are.
template <typename Key>
__device__ __forceinline__ void bitonic_cta(Key* k, int n) {
    int P = 1;
    while (P < n) P <<= 1;
    for (int size = 2; size <= P; size <<= 1) {
        for (int j = size >> 1; j > 0; j >>= 1) {
            const bool mirror = j == size >> 1;
            for (int i = threadIdx.x; i < P / 2; i += blockDim.x) {
                const int lo = 2 * i - (i & (j - 1)), hi = mirror ? lo ^ (size - 1) : lo + j;
                if (hi >= n) continue;
                const Key x = k[lo], y = k[hi];
                if (key_lt(y, x)) { k[lo] = y; k[hi] = x; }
            }
            __syncthreads();
        }
    }
}

// Exclusive scan of one value per thread over the CTA; `total` gets the sum.
__device__ __forceinline__ uint32_t cta_exclusive_scan(uint32_t value, uint32_t* s_scan, uint32_t& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t incl = value;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_scan[warp] = incl;
    __syncthreads();
    uint32_t before = 0;
    total = 0;
    for (int j = 0; j < nw; ++j) {
        if (j < warp) before += s_scan[j];
        total += s_scan[j];
    }
    __syncthreads();
    return before + incl - value;
}

// ---------------------------------------------------------------------------
// Single linkage.  In: s0 sources, s1 targets (Prim order), s2 sorted order, r0
// sorted weights.  Out: s4 left, s5 right, s6 size.  Positions 0..n-1 are the
// vertices in Prim order, edge p (1..n-1) joins position p; position 0 and n
// stand for an infinitely heavy edge.
// ---------------------------------------------------------------------------
// Bit i set: entry i of the eight 16-bit values at `eight` (16-byte aligned) exceeds `mine`.
__device__ __forceinline__ uint32_t above8(const uint16_t* eight, uint32_t mine) {
    const uint4 q = *reinterpret_cast<const uint4*>(eight);
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
    uint32_t mask = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        mask |= ((w[i] & 0xffffu) > mine ? 1u : 0u) << (2 * i);
        mask |= ((w[i] >> 16) > mine ? 1u : 0u) << (2 * i + 1);
    }
    return mask;
}

// Maxima of `at` (padded to a multiple of 8 with zeros) over 8, 64 and 512 entries.
struct PeakTree {
    const uint16_t* level[4];
    // Nearest entry left of p that exceeds `mine`, 0 if none (entry 0 is none).
    __device__ __forceinline__ int left(int p, uint32_t mine) const {
        int i = p;
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            uint32_t mask = above8(level[l] + (i & ~7), mine) & ((1u << (i & 7)) - 1u);
            if (mask) {
                i = (i & ~7) + 31 - __clz(mask);
                for (; l > 0; --l) {
                    mask = above8(level[l - 1] + 8 * i, mine);
                    i = 8 * i + 31 - __clz(mask);
                }
                return i;
            }
            i >>= 3;
        }
        return 0;
    }
    // Nearest entry right of p that exceeds `mine`, n if none.
    __device__ __forceinline__ int right(int p, uint32_t mine, int n) const {
        int i = p;
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            uint32_t mask = above8(level[l] + (i & ~7), mine) & ~((2u << (i & 7)) - 1u);
            if (mask) {
                i = (i & ~7) + __ffs(mask) - 1;
                for (; l > 0; --l) {
                    mask = above8(level[l - 1] + 8 * i, mine);
                    i = 8 * i + __ffs(mask) - 1;
                }
                return i;
            }
            i >>= 3;
        }
        return n;
    }
};

constexpr int kPeaks = 4096 / 8 + 4096 / 64 + 8;

template <typename Real>
__device__ void linkage_cta(const Arena<Real>& a, int n, bool distinct) {
    using T = RealTraits<Real>;
    const int tid = threadIdx.x, nt = blockDim.x;
    const int m = n - 1;
    const int cap = Arena<Real>::round_cap(n);
    uint16_t* at = reinterpret_cast<uint16_t*>(a.s7);   // sorted position of edge p
    uint16_t* gl = reinterpret_cast<uint16_t*>(a.s8);   // nearest later-sorted edge to the left (0: none)
    uint16_t* gr = reinterpret_cast<uint16_t*>(a.s9);   // to the right (n: none)
    uint16_t* cls = reinterpret_cast<uint16_t*>(a.s3);  // edge p's weight: first sorted position holding it
    uint16_t* pos = reinterpret_cast<uint16_t*>(a.r2);  // position of a vertex
    // Node of the gap right of edge p (entry p) and left of it (entry n + p).
    uint16_t* top = reinterpret_cast<uint16_t*>(a.r1);
    int16_t* left = a.s4;
    int16_t* right = a.s5;
    int16_t* size = a.s6;
    __shared__ __align__(16) uint16_t peaks[kPeaks];  // upper levels of the peak tree
    const int n1 = (cap / 8 + 7) & ~7, n2 = (n1 / 8 + 7) & ~7, n3 = (n2 / 8 + 7) & ~7;
    PeakTree tree;
    tree.level[0] = at;
    tree.level[1] = peaks;
    tree.level[2] = peaks + n1;
    tree.level[3] = peaks + n1 + n2;
    for (int t = tid; t < m; t += nt) {
        const int p = a.s2[t] + 1;
        at[p] = (uint16_t)t;
        pos[a.s1[t]] = (uint16_t)(t + 1);
        int c = t;
        if (!distinct) {
            const Real wgt = a.r0[t];
            while (c > 0 && !T::lt(a.r0[c - 1], wgt)) --c;
        }
        cls[p] = (uint16_t)c;
    }
    for (int p = n + tid; p < cap; p += nt) at[p] = 0;
    if (tid == 0) { at[0] = 0; pos[0] = 0; }
    __syncthreads();
    auto peak_level = [&](const uint16_t* below, int count_below, uint16_t* out, int count) {
        for (int b = tid; b < count; b += nt) {
            uint32_t best = 0;
            if (8 * b < count_below) {
                const uint4 q = *reinterpret_cast<const uint4*>(below + 8 * b);
                const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) best = max(best, max(w[i] & 0xffffu, w[i] >> 16));
            }
            out[b] = (uint16_t)best;
        }
        __syncthreads();
    };
    peak_level(at, cap, peaks, n1);
    peak_level(peaks, n1, peaks + n1, n2);
    peak_level(peaks + n1, n2, peaks + n1 + n2, n3);
    for (int p = 1 + tid; p < n; p += nt) {
        const uint32_t mine = at[p];
        gl[p] = (uint16_t)tree.left(p, mine);
        gr[p] = (uint16_t)tree.right(p, mine, n);
    }
    __syncthreads();
    // Weights of two boundary edges: -1, 0, 1 (positions 0 and n are infinite).
    auto heavier = [&](int p, int q) -> int {
        const bool ip = p <= 0, iq = q >= n;
        if (ip || iq) return (ip ? 1 : 0) - (iq ? 1 : 0);
        return (int)cls[p] - (int)cls[q];
    };
    // Every node and vertex is the top of the gap between its larger neighbours.
    auto hang = [&](int p, int q, int node) {
        const int h = heavier(p, q);
        if (h <= 0 && p > 0) top[p] = (uint16_t)node;
        if (h >= 0 && q < n) top[n + q] = (uint16_t)node;
    };
    for (int p = tid; p < n; p += nt) hang(p, p + 1, p == 0 ? 0 : (int)a.s1[p - 1]);
    uint8_t* tied = a.sel;  // edges with an equal one across a gap
    if (!distinct) {
        for (int p = tid; p < n; p += nt) tied[p] = 0;
        __syncthreads();
        for (int p = 1 + tid; p < n; p += nt) {
            const int l = gl[p], r = gr[p];
            if (l > 0 && cls[l] == cls[p]) { tied[l] = 1; tied[p] = 1; }
            if (r < n && cls[r] == cls[p]) { tied[r] = 1; tied[p] = 1; }
        }
        __syncthreads();
    }
    for (int p = 1 + tid; p < n; p += nt) {
        const int l = gl[p], r = gr[p], t = at[p];
        // Of a tie run only the last edge hangs: it stands for the whole run.
        if (!distinct && tied[p] && ((l > 0 && cls[l] == cls[p]) || (r < n && cls[r] == cls[p]))) continue;
        hang(l, r, n + t);
        size[t] = (int16_t)(r - l);
    }
    if (distinct) {
        __syncthreads();
        for (int p = 1 + tid; p < n; p += nt) {
            const int t = at[p];
            left[t] = (int16_t)top[n + p];
            right[t] = (int16_t)top[p];
        }
        __syncthreads();
        return;
    }
    // Pieces of a tie run: the one right of edge p (slot p) and the one left of
    // the run's first edge p (slot n + p).  Each tied edge's source piece: right
    // of the run's last edge at or before the source, or left of its first.
    for (int p = 1 + tid; p < n; p += nt) {
        if (!tied[p]) continue;
        const int src = pos[a.s0[p - 1]], c = cls[p];
        // Edges no lighter than this one are those sorted from c on.
        int y = src;
        if (y > 0 && at[y] < c) y = tree.left(y, (uint32_t)(c - 1));
        if (y <= 0 || cls[y] != c) y = n + (c > 0 ? tree.right(src, (uint32_t)(c - 1), n) : src + 1);
        a.s0[p - 1] = (int16_t)y;
    }
    __syncthreads();
    uint16_t* root = reinterpret_cast<uint16_t*>(a.r2);
    for (int p = 1 + tid; p < n; p += nt) {
        const int t = at[p];
        if (!tied[p]) {
            left[t] = (int16_t)top[n + p];
            right[t] = (int16_t)top[p];
        } else {
            root[p] = (uint16_t)p;
            root[n + p] = (uint16_t)(n + p);
        }
    }
    __syncthreads();
    // One thread a weight joins its runs' pieces in sorted order; the slot of the
    // larger piece stays the root and holds the merged node.
    for (int t0 = tid; t0 + 1 < m; t0 += nt) {
        if (cls[a.s2[t0] + 1] != t0 || cls[a.s2[t0 + 1] + 1] != t0) continue;  // not the first of two or more
        for (int t = t0; t < m; ++t) {
            const int p = a.s2[t] + 1;
            if (cls[p] != t0) break;
            if (!tied[p]) continue;
            int x = a.s0[p - 1], z = p;
            for (int up = root[x]; up != x; up = root[x]) x = up;
            for (int up = root[z]; up != z; up = root[z]) z = up;
            const int nx = top[x], nz = top[z];
            const int sx = nx < n ? 1 : size[nx - n], sz = nz < n ? 1 : size[nz - n];
            left[t] = (int16_t)nx;
            right[t] = (int16_t)nz;
            size[t] = (int16_t)(sx + sz);
            const int big = sx >= sz ? x : z, small = sx >= sz ? z : x;
            root[small] = (uint16_t)big;
            top[big] = (uint16_t)(n + t);
        }
    }
    __syncthreads();
}

// Largest group of equal weights in r0[0..m) is at most kTieRunMax (CTA-uniform).
template <typename Real>
__device__ __forceinline__ bool small_tie_groups(const Arena<Real>& a, int m) {
    bool wide = false;
    for (int t = threadIdx.x; t + kTieRunMax < m; t += blockDim.x)
        wide |= !RealTraits<Real>::lt(a.r0[t], a.r0[t + kTieRunMax]);
    return !__syncthreads_or(wide);
}

// ---------------------------------------------------------------------------
// Condensation: in s4 left, s5 right, s6 size, r0 weights; out as condense_warp
// (hdb_tree.cuh).  Returns next_label (CTA-uniform).  s_scan: 33 words.
// ---------------------------------------------------------------------------
template <typename Real>
__device__ int condense_cta(const Arena<Real>& a, int n, int mcs, int32_t* cl_size, uint32_t* s_scan) {
    using T = RealTraits<Real>;
    constexpr int K = 8;  // nodes a thread: 4096 over 512 threads, fewer in smaller windows
    const int tid = threadIdx.x, nt = blockDim.x;
    const int m = n - 1, root = n - 2;  // nodes by index 0..m-1
    const int16_t* left = a.s4;
    const int16_t* right = a.s5;
    const int16_t* size = a.s6;
    uint16_t* dleaf = reinterpret_cast<uint16_t*>(a.s0);  // parent node of each point
    uint16_t* dnode = reinterpret_cast<uint16_t*>(a.s1);  // of each node
    uint16_t* jump = reinterpret_cast<uint16_t*>(a.s7);   // doubling pointer, then cluster of each large node
    uint16_t* off = reinterpret_cast<uint16_t*>(a.s8);    // leaves left of the node
    uint16_t* dep = reinterpret_cast<uint16_t*>(a.s9);    // depth
    uint16_t* head = reinterpret_cast<uint16_t*>(a.s2);   // first node of the cluster
    uint16_t* first = reinterpret_cast<uint16_t*>(a.s3);  // first path slot of each cluster
    uint32_t* keys = reinterpret_cast<uint32_t*>(a.r1);   // splits
    uint32_t* count = reinterpret_cast<uint32_t*>(a.r2);  // path lengths
    Real* lam = a.r0;
    const Real inf = T::inf();
    auto size_of = [&](int c) { return c < n ? 1 : (int)size[c - n]; };
    auto is_large = [&](int t) { return t == root || (int)size[t] >= mcs; };
    auto is_split = [&](int t) { return size_of(left[t]) >= mcs && size_of(right[t]) >= mcs; };
    for (int t = tid; t < m; t += nt) {
        const Real d = lam[t];
        lam[t] = d > Real(0) ? T::recip(d) : inf;
        const int l = left[t], r = right[t];
        if (l < n) dleaf[l] = (uint16_t)t; else dnode[l - n] = (uint16_t)t;
        if (r < n) dleaf[r] = (uint16_t)t; else dnode[r - n] = (uint16_t)t;
    }
    if (tid == 0) { dnode[root] = (uint16_t)root; s_scan[32] = 0; }
    __syncthreads();
    // Pointer doubling over {jump | head << 16, off | dep << 16}: off and dep sum
    // over the ancestors below jump (all of a large node's ancestors are large;
    // the root's own terms are zero).
    uint2* state = reinterpret_cast<uint2*>(a.r1);  // over r1 and r2
    uint2 mine[K];
    uint32_t large = 0;  // bit k: this thread's k-th node is large
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int t = tid + k * nt;
        if (t >= m || !is_large(t)) continue;
        large |= 1u << k;
        const int p = dnode[t];
        const bool first_node = t == root;
        mine[k].x = (uint32_t)p | ((uint32_t)(first_node || is_split(p) ? t : p) << 16);
        mine[k].y = first_node ? 0u : ((uint32_t)(right[p] == n + t ? size_of(left[p]) : 0) | (1u << 16));
        state[t] = mine[k];
    }
    __syncthreads();
    for (int round = 0; round < 13; ++round) {
        bool open = false;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (!((large >> k) & 1u)) continue;
            const uint2 up = state[mine[k].x & 0xffffu];
            const uint32_t next = (up.x & 0xffffu) | (state[mine[k].x >> 16].x & 0xffff0000u);
            open |= next != mine[k].x;
            mine[k].x = next;
            mine[k].y += up.y;  // both halves stay below 4096
        }
        if (!__syncthreads_or(open)) break;
#pragma unroll
        for (int k = 0; k < K; ++k)
            if ((large >> k) & 1u) state[tid + k * nt] = mine[k];
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if (!((large >> k) & 1u)) continue;
        const int t = tid + k * nt;
        off[t] = (uint16_t)mine[k].y;
        dep[t] = (uint16_t)(mine[k].y >> 16);
        head[t] = (uint16_t)(mine[k].x >> 16);
    }
    __syncthreads();
    // ---- clusters: splits in breadth-first order -------------------------------
    for (int t = tid; t < m; t += nt)
        if (is_large(t) && is_split(t)) keys[atomicAdd(&s_scan[32], 1u)] = ((uint32_t)dep[t] << 12) | off[t];
    __syncthreads();
    const int splits = (int)s_scan[32];
    const int clusters = 1 + 2 * splits;
    bitonic_cta<uint32_t>(keys, splits);
    auto rank_of = [&](int t) {
        const uint32_t key = ((uint32_t)dep[t] << 12) | off[t];
        int lo = 0, hi = splits;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (keys[mid] < key) lo = mid + 1; else hi = mid;
        }
        return lo;
    };
    for (int c = tid; c < clusters; c += nt) count[c] = 0;
    __syncthreads();
    for (int t = tid; t < m; t += nt) {
        if (!is_large(t)) continue;
        const int h = head[t];
        int c = 0;
        if (h != root) {
            const int p = dnode[h];
            c = 1 + 2 * rank_of(p) + (right[p] == n + h ? 1 : 0);
        }
        jump[t] = (uint16_t)c;
        atomicAdd(&count[c], 1u);
    }
    __syncthreads();
    uint32_t paths = 0;  // slots in all: the large nodes
    {
        const int run = (clusters + nt - 1) / nt;
        uint32_t sum = 0;
        for (int c = tid * run; c < min(clusters, (tid + 1) * run); ++c) sum += count[c];
        uint32_t before = cta_exclusive_scan(sum, s_scan, paths);
        for (int c = tid * run; c < min(clusters, (tid + 1) * run); ++c) {
            first[c] = (uint16_t)before;
            before += count[c];
        }
    }
    __syncthreads();
    // Path slots and split ranks, before their arrays are reused.
    uint16_t slot[K], split_rank[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int t = tid + k * nt;
        slot[k] = split_rank[k] = 0xffff;
        if (t >= m || !is_large(t)) continue;
        slot[k] = (uint16_t)(first[jump[t]] + dep[t] - dep[head[t]]);
        if (is_split(t)) split_rank[k] = (uint16_t)rank_of(t);
    }
    __syncthreads();
    int16_t* parent = a.s2;
    Real* birth = a.r1;
    if (tid == 0) {
        parent[0] = -1;
        birth[0] = Real(0);
        a.sel[0] = 0;
        if (cl_size) cl_size[0] = n;
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int t = tid + k * nt;
        if (slot[k] == 0xffff) continue;
        if (split_rank[k] == 0xffff) continue;
        const int c = 1 + 2 * split_rank[k];
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            parent[c + b] = (int16_t)(n + jump[t]);
            birth[c + b] = lam[t];
            a.sel[c + b] = 1;
            if (cl_size) cl_size[c + b] = size_of(b == 0 ? left[t] : right[t]);
        }
    }
    // Every point was pruned at its lowest large ancestor (or the root).
    for (int i = tid; i < n; i += nt) {
        int v = dleaf[i];
        while (v != root && size[v] < mcs) v = dnode[v];
        a.s9[i] = (int16_t)(n + jump[v]);
        a.s8[i] = (int16_t)(n + v);
    }
    __syncthreads();
    uint16_t* adds = dleaf;  // points pruned at each path slot (a split prunes none)
    uint16_t* path = dnode;  // node of each path slot
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int t = tid + k * nt;
        if (slot[k] == 0xffff) continue;
        const int sl = size_of(left[t]), sr = size_of(right[t]);
        adds[slot[k]] = (uint16_t)(split_rank[k] != 0xffff ? 0 : (sl >= mcs ? 0 : sl) + (sr >= mcs ? 0 : sr));
        path[slot[k]] = (uint16_t)t;
    }
    __syncthreads();
    // Lambda of every pruned point in path order; adds becomes the first of each slot.
    Real* point_lam = a.r2;
    uint32_t pruned_in_all;
    {
        const int run = ((int)paths + nt - 1) / nt;
        const int lo = tid * run, hi = min((int)paths, lo + run);
        uint32_t sum = 0;
        for (int i = lo; i < hi; ++i) sum += adds[i];
        uint32_t at = cta_exclusive_scan(sum, s_scan, pruned_in_all);
        for (int i = lo; i < hi; ++i) {
            const Real l = lam[path[i]];
            const int points = adds[i];
            adds[i] = (uint16_t)at;
            for (int j = 0; j < points; ++j) point_lam[at++] = l;
        }
    }
    __syncthreads();
    // ---- stabilities: the reference's additions, in order, along each path --------
    Real stab[K];
    uint16_t last[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int c = tid + k * nt;
        if (c >= clusters) continue;
        const int end = c + 1 < clusters ? (int)first[c + 1] : (int)paths;
        int i = adds[first[c]];
        const int stop = c + 1 < clusters ? (int)adds[end] : (int)pruned_in_all;
        const Real cb = birth[c];
        Real st = Real(0);
        for (; i + 8 <= stop; i += 8) {
            Real l[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) l[j] = point_lam[i + j];
#pragma unroll
            for (int j = 0; j < 8; ++j) st = T::add(st, T::sub(l[j], cb));
        }
        for (; i < stop; ++i) st = T::add(st, T::sub(point_lam[i], cb));
        const int t = path[end - 1];
        const int sl = size_of(left[t]), sr = size_of(right[t]);
        if (sl >= mcs && sr >= mcs) {  // children in order
            const Real term = T::sub(lam[t], cb);
            st = T::add(st, T::mul(term, (Real)sl));
            st = T::add(st, T::mul(term, (Real)sr));
        }
        stab[k] = st;
        last[k] = (uint16_t)t;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int c = tid + k * nt;
        if (c >= clusters) continue;
        a.r2[c] = stab[k];
        a.s3[c] = (int16_t)last[k];
    }
    __syncthreads();
    return n + clusters;
}

// What tree_window_cta finds in the arena beside the Prim edges (r0, s0, s1).
enum class EdgeOrder {
    kNone,    // nothing
    kRanks,   // r1: sorted keys, s2: rank of each edge (first sorted position of its weight)
    kSorted,  // r1: sorted keys, s2: sorted order; no two weights are equal
};

// Sorted order of r0[0..m) into s2, sorted weights into r0.  With float32 and few
// ties (min_samples <= 2) a bitonic sort of (key, index) words serves first; it
// stands when no two weights are equal.  True in that case.
template <typename Real>
__device__ __forceinline__ bool order_edges_cta(const Arena<Real>& a, int m, bool try_distinct, int bar, int* s_ctr) {
    using T = RealTraits<Real>;
    const int tid = threadIdx.x, nt = blockDim.x;
    if constexpr (sizeof(Real) == 4) {
        if (try_distinct) {
            unsigned long long* word = reinterpret_cast<unsigned long long*>(a.r1);  // over r1 and r2
            for (int i = tid; i < m; i += nt) word[i] = ((unsigned long long)T::key(a.r0[i]) << 32) | (uint32_t)i;
            __syncthreads();
            bitonic_cta(word, m);
            bool twin = false;
            for (int i = tid; i + 1 < m; i += nt) twin |= (uint32_t)(word[i] >> 32) == (uint32_t)(word[i + 1] >> 32);
            if (!__syncthreads_or(twin)) {
                for (int i = tid; i < m; i += nt) {
                    a.s2[i] = (int16_t)(uint32_t)word[i];
                    a.r0[i] = T::from_key((uint32_t)(word[i] >> 32));
                }
                __syncthreads();
                return true;
            }
        }
    }
    sort_edges_cta<Real>(a, m, nt, bar, s_ctr);
    return false;
}

// The hierarchy of one window by the whole CTA (all threads call).
// s_scan: 33 words, s_ctr: 4 words of shared memory.
template <typename Real>
__device__ __noinline__ void tree_window_cta(const ForwardArgs& args, unsigned char* base_ptr, int w, int n, EdgeOrder known,
                                             uint32_t* s_scan, int* s_ctr, int bar) {
    using T = RealTraits<Real>;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int m = n - 1;
    const int64_t base = args.offsets[w];
    const int64_t ebase = base - w;
    const Arena<Real> a = Arena<Real>::carve(base_ptr, n);
    auto stamp = [&](int k) {
        if (args.stage_ns && tid == 0) {
            int64_t t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            args.stage_ns[8 * w + k] = t;
        }
    };
    stamp(3);
    if (args.edges_uv) {
        for (int i = tid; i < m; i += nt) {
            args.edges_uv[2 * (ebase + i)] = a.s0[i];
            args.edges_uv[2 * (ebase + i) + 1] = a.s1[i];
            static_cast<Real*>(args.edge_w)[ebase + i] = a.r0[i];
        }
    }
    bool distinct = known == EdgeOrder::kSorted;
    __syncthreads();
    if (known == EdgeOrder::kNone) {
        distinct = order_edges_cta<Real>(a, m, args.unit_core != 0, bar, s_ctr);
    } else {
        if (known == EdgeOrder::kRanks) {
            RankPair* p = reinterpret_cast<RankPair*>(a.r2);
            for (int i = tid; i < m; i += nt) p[i].v = ((uint32_t)(uint16_t)a.s2[i] << 16) | (uint32_t)i;
            sort_pairs_cta(p, a, m, nt, bar, s_ctr);
            for (int i = tid; i < m; i += nt) a.s2[i] = (int16_t)(p[i].v & 0xffffu);
        }
        const typename T::Bits* sorted = reinterpret_cast<const typename T::Bits*>(a.r1);
        for (int t = tid; t < m; t += nt) a.r0[t] = T::from_key(sorted[t]);
        __syncthreads();
    }
    stamp(4);
    if (args.order)
        for (int i = tid; i < m; i += nt) args.order[ebase + i] = a.s2[i];
    if (distinct || small_tie_groups<Real>(a, m)) {
        linkage_cta<Real>(a, n, distinct);
    } else {
        __syncthreads();
        for (int i = tid; i < m; i += nt) {
            const int e = a.s2[i];
            const int16_t u = a.s0[e], v = a.s1[e];
            a.s2[i] = u;
            a.s3[i] = v;
        }
        __syncthreads();
        if (warp == 0) linkage_warp<Real>(a, n);
        __syncthreads();
    }
    stamp(5);
    if (args.link_lr) {
        for (int i = tid; i < m; i += nt) {
            args.link_lr[2 * (ebase + i)] = a.s4[i];
            args.link_lr[2 * (ebase + i) + 1] = a.s5[i];
            args.link_size[ebase + i] = a.s6[i];
            static_cast<Real*>(args.link_w)[ebase + i] = a.r0[i];
        }
        __syncthreads();
    }
    const int next_label = condense_cta<Real>(a, n, args.mcs, args.cl_size ? args.cl_size + base : nullptr, s_scan);
    stamp(6);
    if (args.point_lambda) {  // s8: the linkage node each point was pruned at; r0: lambda per node
        Real* out = static_cast<Real*>(args.point_lambda) + base;
        for (int i = tid; i < n; i += nt) out[i] = a.r0[a.s8[i] - n];
    }
    if (args.cl_parent) {
        for (int c = tid; c < next_label - n; c += nt) {
            args.cl_parent[base + c] = a.s2[c];
            static_cast<Real*>(args.cl_birth)[base + c] = a.r1[c];
        }
        for (int i = tid; i < n; i += nt) args.point_parent[base + i] = a.s9[i];
    }
    __syncthreads();
    if (warp > 0) return;
    select_and_label_warp<Real>(a, n, next_label, (Real)args.eps, args.method, args.allow_single != 0, args.labels + base,
                                args.probabilities ? static_cast<Real*>(args.probabilities) + base : nullptr);
    if (args.cl_parent) {
        for (int c = lane; c < next_label - n; c += 32) {
            static_cast<Real*>(args.cl_stability)[base + c] = a.r2[c];
            args.cl_selected[base + c] = a.sel[c];
        }
        if (lane == 0) args.n_clusters[w] = next_label - n;
    }
    stamp(7);
}

}  // namespace hdb
