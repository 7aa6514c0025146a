// mm_common.cuh -- shared device helpers and the mm_graph object.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "mm_match.h"

namespace mm {

// Round caps of the reference (src/matchcpu.h:24-25): fixed types run
// NR_MATCH_ROUNDS = 20 rounds, maximal types loop while ++count < 256.
constexpr int kFixedRounds = 20;
constexpr int kMaxRounds = 255;

// Per-vertex colour state.  It carries what a neighbour's request/respond test
// needs from the reference's match value (src/matchgpu.cu:303-316, 380-386,
// 346, 431): kBlue (match 0), kRed (match 1), kDead (match 2), kMatched (match >= 4).
enum : uint8_t { kBlue = 0, kRed = 1, kDead = 2, kMatched = 3 };

// Colouring hash of src/matchgpu.cu:196-217: 16 MD5-style steps over
// (vertex id, round seed) with the first 16 SHA-256 constants, the MD5
// round-1 rotations and the MD5 initial words.  The reference adds up
// h0 + h1 + h2 + h3 before the first step and after each.  A step moves the
// four words along (h0 <- h3 <- h2 <- h1) and makes one new one, so with B_k
// the word that step k makes, the sum is a constant plus 4 (B_1 + .. + B_13)
// + 3 B_14 + 2 B_15 + B_16: one addition a step in place of four.  Set-up and
// commit passes over millions of vertices are bound by these instructions.
__device__ __forceinline__ uint32_t colour_hash(uint32_t v, uint32_t seed)
{
    constexpr uint32_t K[16] = {0x428a2f98u, 0x71374491u, 0xb5c0fbcfu, 0xe9b5dba5u,
                                0x3956c25bu, 0x59f111f1u, 0x923f82a4u, 0xab1c5ed5u,
                                0xd807aa98u, 0x12835b01u, 0x243185beu, 0x550c7dc3u,
                                0x72be5d74u, 0x80deb1feu, 0x9bdc06a7u, 0xc19bf174u};
    constexpr int R[4] = {7, 12, 17, 22};
    constexpr uint32_t A = 0x67452301u, B = 0xefcdab89u, C = 0x98badcfeu, D = 0x10325476u;
    uint32_t a = A, b = B, c = C, d = D;
    uint32_t g = v, run = 0u, sum = A + 2u * D + 3u * C + 4u * B;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const uint32_t f = (b & c) | (~b & d);
        const uint32_t x = a + f + (K[k] + g);
        a = d;
        d = c;
        c = b;
        b = b + __funnelshift_l(x, x, R[k & 3]);
        run += b;
        if (k >= 12) sum += run;
        g *= seed;
    }
    return sum;
}

// Blue iff the hash is below the select barrier (src/matchgpu.cu:217).
__device__ __forceinline__ uint8_t colour_of(uint32_t v, uint32_t seed, uint32_t barrier)
{
    return colour_hash(v, seed) < barrier ? kBlue : kRed;
}

// Order-preserving map of a float to uint32 for the weighted argmax.  Only
// weights the reference can pick reach it (w > -1, so never NaN); -0.0 is
// folded onto +0.0 because the reference's `nw > maxWeight` treats them as
// equal (src/matchgpu.cu:391, 437).
__device__ __forceinline__ uint32_t weight_order(float w)
{
    uint32_t u = __float_as_uint(w);
    if (u == 0x80000000u) u = 0u;
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

}  // namespace mm

// Device-resident graph plus per-graph scratch.  Everything lives on `device`.
struct mm_graph {
    int device = 0;
    int n = 0;
    long long nnz = 0;
    bool has_weights = false;
    bool contiguous = false;  // ranges tile [0, nnz) in vertex order
    // Set at upload: ranges tile [0, nnz), every list is strictly increasing and
    // the entries (v, u) are those (u, v) transposed -- with the weights too for
    // sym_weights.  Then a red vertex's order of preference over its proposers is
    // (weight, smaller proposer id) and the push path needs no reverse index.
    bool sym_pairs = false;   // the ranges tile [0, nnz) and every entry has a reverse entry, in any order
    bool no_self = false;     // the ranges tile [0, nnz) and no list names its own vertex
    bool sym_struct = false;
    bool sym_weights = false;
    int2 *d_ranges = nullptr;
    int *d_nbrs = nullptr;
    float *d_w = nullptr;     // unit weights when the graph came without any
    long long max_degree = 0;
    long long sum_degree = 0;
    bool scanned = false;          // degree classes below are valid
    long long long_count = 0;      // vertices with more than 32 neighbour entries
    long long long_entries = 0;    // entries in those longer lists
    long long win_groups = 0;      // groups of 4 entries of all preference windows
    long long win_even = 0;        // windows' lengths rounded up to even numbers, in all (limited, windows_begin)

    // device buffer for host-output calls (mm_match)
    int *d_out = nullptr;

    // scratch shared by the paths, grown on demand
    void *scratch = nullptr;
    size_t scratch_bytes = 0;

    // push path: reverse proposal keys, one per adjacency slot, per weighting
    unsigned long long *d_revkey[2] = {nullptr, nullptr};  // [0] random, [1] weighted
    long long *d_slot_off = nullptr;  // non-contiguous CSR: slot index of vertex v's first entry
    int2 *d_pwin = nullptr;           // weighted types: preference windows {neighbour, position | flag}
    int *d_pwin_off = nullptr;        // weighted types, [n + 1]: first group of 4 window entries, bit 31: list longer than 32
    bool pwin_weights = false;        // d_pwin's second words hold weights (symmetric weighted path)
    int2 *win_build = nullptr;        // windows while being built (d_pwin once complete)
    int *win_big = nullptr;           // while being built: queued lists longer than a window chunk
    void *win_tmp[3] = {};            // while being built: scratch, the first of win_tmp_bytes
    size_t win_tmp_bytes = 0;

    // push path: per-call state of the round kernel
    void *push_exec = nullptr;  // internal (mm::PushState *)
    // launch options (mm_graph_tune; 0 = the library's default)
    int opt_fin_div = 0;        // finish phase from the round whose active set is <= 1/opt of round 0's; -1 never
    int opt_blocks_per_sm = 0;  // blocks per SM of the matching kernel

    // a batch of independent graphs (mm_graph_set_batch): graph i holds
    // vertices [goff[i], goff[i + 1]); vbase[v] = goff of v's graph; last[v]
    // = last round at whose colouring v was unmatched
    int ngraphs = 0;
    int *d_goff = nullptr;
    int *d_vbase = nullptr;
    uint8_t *d_last = nullptr;
    int *d_glast = nullptr;  // last active round of each graph
};

namespace mm {

void set_error(const std::string &msg);
mm_status cuda_fail(cudaError_t e, const char *what);
#define MM_CUDA_TRY(expr, what)                              \
    do {                                                     \
        cudaError_t mm_e_ = (expr);                          \
        if (mm_e_ != cudaSuccess) return mm::cuda_fail(mm_e_, what); \
    } while (0)

// Pooled device memory (one stream-ordered pool per device, never trimmed
// unless mm_release_cached_memory asks): allocation and free are ordered on
// `stream`; a buffer used on other streams needs that stream synchronised first.
cudaError_t dev_alloc(void **p, size_t bytes, cudaStream_t stream);
void dev_free(void *p, cudaStream_t stream);
// Small page-locked host blocks, recycled process-wide.
cudaError_t pinned_get(void **p, size_t bytes);
void pinned_put(void *p, size_t bytes);
mm_status release_cached(int device);

// Polls a grid-barrier wait makes before it gives up (the kernel then returns
// an error status instead of waiting on).
constexpr long long kSpinLimitDefault = 1ll << 22;
// Testing hooks (mm_debug): the grid barriers' poll limit and the barrier mark
// at which block 0 does not arrive (-1: none).
long long debug_spin_limit();
int debug_skip_mark();

// Entries that neighbour and weight arrays are allocated for: a multiple of 4
// plus 4, so that 16-byte vector loads starting at any in-range, 4-aligned slot
// stay inside.
inline size_t padded_entries(long long nnz) { return ((size_t)nnz + 3) / 4 * 4 + 4; }

// A graph from device arrays of the pool, which it takes over: valid lists that
// tile [0, nnz) in vertex order, strictly increasing, arrays padded with zeros.
mm_status adopt_arrays(int device, int n, long long nnz, int2 *ranges, int *nbrs, float *w, bool sym_struct, bool sym_w,
                       mm_graph **out);

// Symmetry of a graph's entries: the multiset of entries (v, u) equals that of
// (u, v), and with weights, of (v, u, w) and (u, v, w).  Each entry below the
// diagonal adds a 64-bit hash of its ordered pair (and weight), each above takes
// it away; a symmetric multiset leaves 0, another one only by a 64-bit
// coincidence.  (splitmix64's finalizer; one hash a pair and one more for its
// weight, where sums of both orders took five.)
__device__ __forceinline__ unsigned long long mix64(unsigned long long z)
{
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__device__ __forceinline__ void add_skew(unsigned v, unsigned u, unsigned wbits, bool weights, unsigned long long &skew_s,
                                         unsigned long long &skew_w)
{
    if (v == u) return;
    const unsigned lo = v < u ? v : u, hi = v < u ? u : v;
    const unsigned long long h = mix64((((unsigned long long)lo << 32) | hi) + 0x9E3779B97F4A7C15ull);
    skew_s += v < u ? h : 0ull - h;
    if (weights) {
        const unsigned long long x = mix64(h ^ ((unsigned long long)wbits * 0xD1B54A32D192ED03ull + 0x2545F4914F6CDD1Dull));
        skew_w += v < u ? x : 0ull - x;
    }
}

// Add the block's sum of v to *dst with one atomic (called by all threads of a
// block of at most 1024, any number of times): atomics of all warps on one
// word took longer than the passes that made them (k_pairs over 2^20 vertices:
// 45 us with two a warp).
__device__ __forceinline__ void block_add(unsigned long long *dst, unsigned long long v)
{
    __shared__ unsigned long long part[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();  // part[] may still be read
    if (lane == 0) part[warp] = v;
    __syncthreads();
    if (warp == 0) {
        v = lane < (int)(blockDim.x + 31) / 32 ? part[lane] : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0 && v) atomicAdd(dst, v);
    }
}

// What one pass over the ranges tells (zero before it).
struct RangeInfo {
    unsigned long long sum_deg;
    unsigned long long max_deg;
    unsigned long long long_count;    // lists of more than 32 entries
    unsigned long long long_entries;  // entries in those
    unsigned long long win_groups;    // preference windows: groups of 4 entries
    unsigned long long win_even;      // preference windows: lengths rounded up to even numbers
    int noncontig;                    // ranges do not tile [0, nnz) in vertex order
    int bad;                          // a range outside [0, nnz)
};
cudaError_t scan_ranges(const int2 *ranges, int n, long long nnz, RangeInfo *d_info, long long *deg_out, cudaStream_t stream);
void apply_ranges(mm_graph *g, const RangeInfo &info);

// Ensure g->scratch holds at least `bytes`; returns MM_OK or an error.
mm_status ensure_scratch(mm_graph *g, size_t bytes);

// Paths.
mm_status pull_match(mm_graph *g, int type, uint32_t barrier, const uint32_t *seeds, int nseeds,
                     int *d_match, int *rounds_out, long long *stats, int stats_rounds,
                     cudaStream_t stream, uint32_t (*draw)(void *) = nullptr, void *draw_ctx = nullptr);
mm_status push_prepare(mm_graph *g, int weighted, cudaStream_t stream);
mm_status push_match(mm_graph *g, int type, uint32_t barrier, const uint32_t *seeds, int nseeds,
                     int *d_match, int *rounds_out, long long *stats, int stats_rounds,
                     cudaStream_t stream);
mm_status push_profile(mm_graph *g, int type, uint32_t barrier, const uint32_t *seeds, int nseeds, int *d_match,
                       int *rounds_out, float *ms_kernels, int cap_rounds, int *launched, cudaStream_t stream);
void push_release(mm_graph *g);
mm_status push_batch_rounds(mm_graph *g, int type, int *rounds_host, cudaStream_t stream);
mm_status push_match_policy(mm_graph *g, int type, uint32_t barrier, const uint32_t *seeds, int nseeds,
                            const float *mlp_host, float level, int *d_match, int *rounds_out, float *trace,
                            int trace_rounds, cudaStream_t stream);
// Preference windows of the weighted types, in steps (see mm_push.cu).
mm_status windows_begin(mm_graph *g, cudaStream_t stream, cudaStream_t mem);
mm_status windows_range(mm_graph *g, int va, int vb, cudaStream_t stream);
mm_status windows_end(mm_graph *g, cudaStream_t stream, cudaStream_t mem);
void windows_settle(mm_graph *g, cudaStream_t mem);
void windows_discard(mm_graph *g);

inline int max_rounds_of(int type)
{
    if (type == MM_TYPE_RANDOM || type == MM_TYPE_WEIGHTED) return kFixedRounds;
    if (type == MM_TYPE_RANDOM_MAXIMAL || type == MM_TYPE_WEIGHTED_MAXIMAL) return kMaxRounds;
    return -1;
}
inline bool is_weighted(int type) { return type == MM_TYPE_WEIGHTED || type == MM_TYPE_WEIGHTED_MAXIMAL; }
inline bool is_maximal(int type) { return type == MM_TYPE_RANDOM_MAXIMAL || type == MM_TYPE_WEIGHTED_MAXIMAL; }

inline int grid_for(long long items, int block, int cap = 148 * 32)
{
    long long g = (items + block - 1) / block;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (int)g;
}

}  // namespace mm
