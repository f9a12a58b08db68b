// Plain-C++ argument blocks shared by the host plan layer and the kernels.
#pragma once
#include <cstdint>

namespace hdb {

enum Status : int32_t {
    kOk = 0,
    kOverflow = 1,     // a pairwise distance is not finite (reference: _cuda.py:112-113)
    kNonFinite = 2,    // an input coordinate is not finite (reference: _cuda.py:98-99)
    kInternal = 4,     // device-side bounds check tripped (a bug, never expected)
};

// The general path behind the sparse one does the windows of `queue` whose flag is in
// `mask` (bit f for flag f): 1 = left it by the core distances, 2 = later.  flags[n]
// and flags[n + 1] tell whether any window has either.  flags null = no such rule, all
// windows of the launch.
struct FlaggedWindows {
    const int32_t* flags;
    int n;
    int mask;
    const int32_t* queue;
    int n_windows;
};

struct ForwardArgs {
    const void* X;             // packed [T, D] Real
    const int64_t* offsets;    // [B+1] device
    const int32_t* queue;      // windows of this launch, size-sorted
    int queue_len;
    int32_t* ticket;           // persistent work counter (zeroed before launch)
    int D;
    int mcs;
    int unit_core;             // ms <= 2
    int x_in_smem;             // stage the window's coordinates in shared memory
    int n_arenas;              // 1 or 2 hierarchy arenas (2 = Prim/tree overlap)
    int arena_stride;          // bytes per arena in dynamic shared memory
    int x_off;                 // byte offset of the staged coordinates
    int core_off;              // byte offset of the staged core distances
    double eps;
    const void* core;          // [T] Real, or null when unit_core
    const void* dist;          // matrix variant: packed per-window [n, n] Real blocks
    const int64_t* dist_offsets;  // [B] element offset of each window's block
    int32_t* labels;           // [T]
    int32_t* status;           // bit-or of Status codes
    // Optional exports (null = skip).  Edge arrays are packed per window at
    // offsets[w] - w (n-1 entries each); cluster arrays at offsets[w].
    int32_t* edges_uv;         // [T-B, 2] Prim order
    void* edge_w;              // [T-B]   Prim order
    int32_t* order;            // [T-B]   argsort of edge_w (window-local indices)
    int32_t* link_lr;          // [T-B, 2] children of node n+i
    void* link_w;              // [T-B]
    int32_t* link_size;        // [T-B]
    int32_t* n_clusters;       // [B]
    int32_t* cl_parent;        // [T]
    void* cl_birth;            // [T]
    void* cl_stability;        // [T]
    uint8_t* cl_selected;      // [T]
    int32_t* point_parent;     // [T]
    int64_t* stage_ns;         // [B, 8] globaltimer at stage boundaries (diagnostics)
    void* probabilities;       // [T] membership strengths (Real)
    int32_t* cl_size;          // [T] cluster sizes at birth
    void* point_lambda;        // [T] lambda at which each point falls out (Real)
    int method;                // cluster selection: 0 excess of mass, 1 leaf
    int allow_single;          // the root may be selected
    // Cluster form only: limit of every bounded mbarrier wait (0 = the 2 s
    // default), and a test switch under which the first window ticket is never
    // broadcast, so every CTA's first wait runs out (nothing is in flight then).
    int64_t wait_limit_ns;
    int stall_first_ticket;
    FlaggedWindows flagged;
};

// Small-window kernel (hdb_small.cuh): core distances, beside ForwardArgs.
struct SmallArgs {
    int ms;
    void* core;          // [T] Real
    int32_t* core_nbr;   // [T]
};

struct DistanceArgs {
    const void* X;
    const int64_t* offsets;
    const int32_t* tiles;        // [n_tiles, 3] = (window, tile row, tile col), col >= row
    int n_tiles;
    int tile;                    // tile edge: 64, or 128 (float32 only)
    int D;
    void* dist;                  // packed blocks
    const int64_t* dist_offsets; // [B]
    int32_t* status;
    FlaggedWindows flagged;      // if set, the work is found in its windows instead of the table
};

struct CoreArgs {
    const void* X;
    const int64_t* offsets;
    const int32_t* items;        // [n_items, 2] = (window, first row)
    int n_items;
    int D;
    int ms;                      // order statistic k = ms-1 (0-based), self included
    int rows;                    // select kernel: rows per item
    const void* dist;            // matrix variant only
    const int64_t* dist_offsets;
    void* core;                  // [T]
    int32_t* core_nbr;           // [T] or null
    int32_t* status;
    FlaggedWindows flagged;      // if set, the work is found in its windows instead of the table
};

// Sparse path (hdb_sparse.cuh): one launch group covers the `n_windows` windows
// of `queue` (descending sizes, at most nmax points each).  Per-point arrays
// are indexed by packed point row, per-window ones by window.
struct SparseArgs {
    const void* X;
    const int64_t* offsets;
    const int32_t* queue;
    int n_windows;
    int nmax;
    int64_t T;                   // points of the whole batch (stride of the per-level arrays)
    int D;
    int ms;
    int unit_core;
    int32_t* flags;              // [B+2] see FlaggedWindows
    int n_flags;                 // B
    int stage;                   // flag value of the pass: 1 up to the core distances, 2 from the trees on
    int approx;                  // distances are bounded float32 ones (else exact: float32 windows of few dims)
    int gram;                    // bounded squared distances from tensor-core products (else differences)
    float* y;                    // differences: [T, D] input rounded to float32 around each window's first point
    uint16_t* split;             // products: [T, dims / 32, 64] centred input as bfloat16 pairs, 32 high then 32 low parts
    int dims;                    // D rounded up to 32
    float* minima;               // products: minimum of every 16 entries of the blocks' rows
    float* norm;                 // products: [T] squared norms of the centred points
    uint32_t* split_share;       // products: [2 B] float bits of the largest |lo|^2 / norm, then |rest|^2 / norm
    uint32_t* range;             // [B] float bits of max |x - x0| (products: of the largest norm)
    void* dist;                  // distance blocks (float32 values, see sparse_block)
    const int64_t* dist_offsets;
    uint16_t* knn_idx;           // [T, list] nearest neighbours by (distance, index), self included
    float* knn_d;                // [T, list]
    int list;                    // row stride of the lists (8, 16, 32 or 64)
    int keep;                    // valid entries of each list (<= list)
    void* core;                  // [T] Real
    int32_t* core_nbr;           // [T]
    float* core_up;              // [T] core distance rounded up (float32: core itself)
    float* core_down;            // [T] core distance rounded down (float32: core itself)
    uint16_t* part;              // [T] component number after the list rounds
    int32_t* parts;              // [B] their count
    unsigned long long* edges;   // [T] tree edges found so far
    unsigned long long* table;   // least edge between each two components, parts^2 per window
    const int64_t* table_offsets;  // [B]
    uint16_t* level_comp;        // [kSparseLevels, T] component (its representative vertex) after each merge round
    float* level_max_v;          // [kSparseLevels, T] by vertex: largest tree edge on the way up
    uint32_t* level_span;        // [kSparseLevels, T] by vertex: its component's leaf interval, begin | end << 16
    uint16_t* perm;              // [T] vertices in component order
    int32_t* levels;             // [B] merge rounds
    uint16_t* pos;               // [T] vertex -> leaf position
    int32_t* light_count;        // [B] light edges other than star edges
    uint32_t* light_uv;          // [T * light_cap] u | v << 16
    void* light_w;               // [T * light_cap] Real
    int light_cap;               // kept per point
    int32_t* star_count;         // [B] star edges the order needs
    uint32_t* star_uv;           // [T * star_cap] x | u << 16, of weight core_x
    unsigned long long* star_mask;  // [T] list positions of each point's star
    int star_cap;
    uint16_t* edge_rank;         // [T * (light_cap + star_cap)]
    uint32_t* adj;               // [T * (light_cap + star_cap) * 2] adjacency that shared memory does not hold
};
// Components that the list rounds may leave.
#ifdef __CUDACC__
__host__ __device__
#endif
inline int sparse_parts_cap(int n) { return n < 256 ? 32 : n / 8; }
constexpr int kSparseLevels = 12;  // every merge round at least halves the components: 2^12 points

constexpr int kBackwardWarps = 8;  // backward kernel: warps (32 linkage rows each) per CTA

struct BackwardArgs {
    const void* X;               // [T, D]
    const int64_t* offsets;      // [B+1]
    int windows;                 // B
    int n_edges;                 // T - B
    int D;
    int unit_core;
    const int32_t* edges_uv;     // [T-B, 2] Prim order (window-local vertex ids)
    const int32_t* order;        // [T-B] Prim-edge index (window-local) of linkage row i
    const void* link_w;          // [T-B] merge weights in linkage order
    const void* grad;            // [T-B] dL/dmerge_weight in linkage order
    const void* core;            // [T] or null
    const int32_t* core_nbr;     // [T] or null
    void* dX;                    // [T, D] accumulated (caller zeroes)
};

}  // namespace hdb
