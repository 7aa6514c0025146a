// mm_check.cu -- GPU validation and weight of a matching.
//
// Device counterparts of the reference's host-side checks, so that a matching
// of a large graph can be judged without copying it back and sorting it on
// the host:
//   mm_matching_weight  GraphMatching::getWeight   (src/matchcpu.cu:64-97)
//   mm_matching_check   GraphMatching::testMatching (src/matchcpu.cu:127-246)
// Both read the graph's device CSR and a device match array, and report
// through their outputs; nothing is printed.
//
// A matching whose every value is held by exactly two vertices, one of them
// the vertex that the value names, needs neither a sort nor a gather of match
// values: k_pairs finds each vertex's partner (and whether the matching is of
// that kind), and one pass over the lists looks for the partner's id, a group
// of lanes per list (of symmetric graphs, one list a pair).  That is every
// matching the matchers write; on RGG 2^20 weight and check together take 147 us
// so, 371 us by the general kernels (a thread a vertex and its list, a radix
// sort of the values, three synchronisations).
// Anything else takes the general kernels, which follow the reference's walk.
#include <cuda_runtime.h>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_reduce.cuh>
#include <cub/device/device_scan.cuh>

#include "mm_common.cuh"

#define MM_API extern "C" __attribute__((visibility("default")))

namespace mm {
namespace {

__device__ __forceinline__ bool is_matched(int m) { return m >= 4; }  // matchcpu.h:41

// ---- matchings made of clean pairs ----

// Scratch of the pair passes, cleared before them.
struct PairState {
    unsigned long long nmin;       // vertices that their own value names
    unsigned long long nother;     // vertices whose value names another
    unsigned long long counts[5];  // as mm_matching_check's
    unsigned long long size;       // as mm_matching_weight's
    unsigned long long size_general;  // the same by the general kernel
    double weight;
    int broken;                    // a value that names no vertex, or one that does not hold it (k_pairs)
    int clash;                     // a vertex that is not the only other one with its value (k_pair_lists)
    int nlong;                     // lists left to the block scans
};

// other[a]: 1 + the partner of the vertex a that a value names (0: none).  The matching is
// clean iff nothing is broken, nmin == nother and every other vertex is the
// only one to claim its named vertex (which holds the value too; no clash).
__global__ void k_pairs(const int *match, int n, int *other, PairState *st)
{
    int nmin = 0, nother = 0, broken = 0;
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const int m = match[v];
        if (!is_matched(m)) continue;
        const long long a = (long long)m - 4;
        if (a == v) {
            ++nmin;
        } else if (a >= n || match[a] != m) {
            broken = 1;
        } else {
            other[a] = v + 1;  // the last of several stays; the others find that out (k_pair_lists)
            ++nother;
        }
    }
    block_add(&st->nmin, (unsigned long long)nmin);
    block_add(&st->nother, (unsigned long long)nother);
    if (__any_sync(0xffffffffu, broken) && (threadIdx.x & 31) == 0) atomicOr(&st->broken, 1);
}

// What k_pairs found.  The list pass looks at nothing else before it starts: a
// word that its own blocks write would let warps of one block part ways ahead of
// the block's barriers.
__host__ __device__ __forceinline__ bool paired(const PairState *st) { return !st->broken && st->nmin == st->nother; }
// The matching is clean (after the list pass).
__host__ __device__ __forceinline__ bool clean(const PairState *st) { return paired(st) && !st->clash; }

// Whether an entry naming u is what a pass looks for at vertex v:
//   partner >= 0  the partner (kSelf: or the vertex itself, whose match value
//                 is the same)
//   partner < 0   (unmatched, the check only) an unmatched neighbour
template <bool kSelf>
__device__ __forceinline__ bool entry_hit(const int *match, int v, int partner, int u)
{
    if (partner >= 0) return u == partner || (kSelf && u == v);
    return u != v && !is_matched(match[u]);
}

// What one list adds: kWeight the matched entry's weight and 1, else the
// check's counts (cnt: invalid, matchable, unmatched).  kHalf: a pair's lists
// name each other or neither does, with the same weight, so the list of the
// vertex that the value names speaks for both.  Otherwise a pair is invalid if
// either list misses the other vertex: the first of the two to say so (bad[],
// at the vertex that the value names) counts it.
template <bool kWeight, bool kHalf>
__device__ __forceinline__ void pair_result(const float *w, int v, int partner, int at, double *contrib,
                                            unsigned (&cnt)[3], int *bad)
{
    if (kWeight) {
        const double x = at >= 0 ? (double)w[at] : 0.0;
        contrib[v] = x;
        if (kHalf && partner >= 0) contrib[partner] = x;  // (< 0: named by no other's value, so not clean)
        cnt[0] += at >= 0 ? (kHalf ? 2u : 1u) : 0u;
    } else if (partner >= 0) {
        if (at < 0 && (kHalf || atomicExch(bad + min(v, partner), 1) == 0)) ++cnt[0];
    } else {
        ++cnt[2];
        cnt[1] += at >= 0;
    }
}

template <bool kWeight>
__device__ __forceinline__ void add_counts(const unsigned (&cnt)[3], PairState *st)
{
    if (kWeight) {
        if (cnt[0]) atomicAdd(&st->size, (unsigned long long)cnt[0]);
    } else {
        for (int k = 0; k < 3; ++k)
            if (cnt[k]) atomicAdd(&st->counts[2 + k], (unsigned long long)cnt[k]);
    }
}

// One pass over all vertices, 32 a warp at a time: a lane reads a vertex's
// match value, range and partner, then the lists that have to be searched are
// dealt to groups of G lanes, kSlots a group, 4 G entries of each a step.  The
// pass waits on the chain vertex -> list -> entries, so what counts is how many
// lists a warp has in flight, and on its instructions.  RGG 2^20: weight 30 us,
// check 31 us with one list a pair and 16 of them in flight; 50 us each with a
// group for every vertex, 8 in flight and a ballot for each entry of a step.
// Longer lists than kPairList are queued for a block each.
constexpr int kPairList = 1024;
constexpr int kSlots = 2;
constexpr int kPairBlocks = 6;  // a multiprocessor (at 60 registers, 4 of them, the check took 54 us)

template <int G, bool kWeight, bool kHalf>
__global__ void __launch_bounds__(256, kPairBlocks) k_pair_lists(const int2 *ranges, const int *nbrs, const float *w, const int *match,
                                                    int n, const int *other, int *bad, int *queue, double *contrib,
                                                    PairState *st)
{
    if (!paired(st)) return;
    __shared__ uint8_t s_from[8][32];
    constexpr int kGroups = 32 / G;
    const int lane = threadIdx.x & 31, l = lane & (G - 1);
    uint8_t *from = s_from[threadIdx.x >> 5];
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long stride = ((long long)gridDim.x * blockDim.x >> 5) * 32;
    unsigned cnt[3] = {0u, 0u, 0u};
    bool clash = false;
    for (long long base = warp * 32; base < n; base += stride) {  // warp-uniform
        const bool in = base + lane < n;
        const int v = in ? (int)base + lane : -1, mv = in ? match[v] : 0;
        const int2 r = in ? ranges[v] : make_int2(0, 0);
        const bool matched = is_matched(mv);
        const int a = mv - 4, o = matched ? other[a] : 0;
        const int partner = !matched ? -1 : (a == v ? o - 1 : a);
        clash |= matched && a != v && o != v + 1;
        if (kWeight && in && !matched) contrib[v] = 0.0;
        bool want = in && (matched ? !kHalf || a == v : !kWeight);
        if (want && r.y > r.x && r.y - r.x > kPairList) {
            queue[atomicAdd(&st->nlong, 1)] = v;
            want = false;
        }
        const unsigned wants = __ballot_sync(0xffffffffu, want);
        const int nw = __popc(wants);
        __syncwarp();
        if (want) from[__popc(wants & ((1u << lane) - 1u))] = (uint8_t)lane;
        __syncwarp();
        for (int b = 0; b < nw; b += kSlots * kGroups) {
            int vs[kSlots], ps[kSlots], js[kSlots], je[kSlots], at[kSlots];
            bool mine[kSlots], go[kSlots], any = false;
#pragma unroll
            for (int q = 0; q < kSlots; ++q) {
                const int slot = b + q * kGroups + lane / G;
                mine[q] = slot < nw;
                const int src = mine[q] ? from[slot] : 0;
                vs[q] = __shfl_sync(0xffffffffu, v, src);
                ps[q] = __shfl_sync(0xffffffffu, partner, src);
                js[q] = __shfl_sync(0xffffffffu, r.x, src);
                je[q] = __shfl_sync(0xffffffffu, r.y, src);
                at[q] = -1;
                go[q] = mine[q] && js[q] < je[q];
                any |= go[q];
            }
            while (__any_sync(0xffffffffu, any)) {
                int u[kSlots][4];
#pragma unroll
                for (int q = 0; q < kSlots; ++q)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        u[q][k] = go[q] && k * G + l < je[q] - js[q] ? __ldg(nbrs + js[q] + k * G + l) : -1;
                any = false;
#pragma unroll
                for (int q = 0; q < kSlots; ++q) {
                    // the group's first hit of the step, counted from js
                    int first = 4 * G;
#pragma unroll
                    for (int k = 3; k >= 0; --k)
                        if (u[q][k] >= 0 && entry_hit<kWeight>(match, vs[q], ps[q], u[q][k])) first = k * G + l;
#pragma unroll
                    for (int o = G / 2; o > 0; o >>= 1) first = min(first, __shfl_xor_sync(0xffffffffu, first, o));
                    if (go[q] && first < 4 * G) at[q] = js[q] + first;
                    go[q] = go[q] && first == 4 * G && je[q] - js[q] > 4 * G;
                    js[q] += go[q] ? 4 * G : 0;
                    any |= go[q];
                }
            }
#pragma unroll
            for (int q = 0; q < kSlots; ++q)
                if (mine[q] && l == 0) pair_result<kWeight, kHalf>(w, vs[q], ps[q], at[q], contrib, cnt, bad);
        }
    }
    if (__any_sync(0xffffffffu, clash) && lane == 0) atomicOr(&st->clash, 1);
    if (kWeight) {
        block_add(&st->size, cnt[0]);
    } else {
        for (int k = 0; k < 3; ++k) block_add(&st->counts[2 + k], cnt[k]);
    }
}

// The queued long lists, a block each (the lowest hit of a step is the first).
template <bool kWeight, bool kHalf>
__global__ void __launch_bounds__(256) k_pair_long(const int2 *ranges, const int *nbrs, const float *w, const int *match,
                                                   const int *other, int *bad, const int *queue, double *contrib,
                                                   PairState *st)
{
    if (!clean(st)) return;
    __shared__ int s_at;
    const int nlong = st->nlong;
    for (int i = blockIdx.x; i < nlong; i += gridDim.x) {
        const int v = queue[i], mv = match[v];
        const int a = mv - 4, partner = !is_matched(mv) ? -1 : (a == v ? other[v] - 1 : a);
        const int2 r = ranges[v];
        if (threadIdx.x == 0) s_at = 0x7fffffff;
        __syncthreads();
        // unsigned: a list may end at 2^31 - 1, and a step beyond it must not wrap
        for (unsigned j = r.x; j < (unsigned)r.y; j += 4 * 256) {
            int first = 0x7fffffff;
#pragma unroll
            for (int k = 3; k >= 0; --k) {
                const unsigned q = j + k * 256 + threadIdx.x;
                if (q < (unsigned)r.y && entry_hit<kWeight>(match, v, partner, __ldg(nbrs + q))) first = (int)q;
            }
            if (first != 0x7fffffff) atomicMin(&s_at, first);
            __syncthreads();
            const bool done = s_at != 0x7fffffff;
            __syncthreads();
            if (done) break;
        }
        if (threadIdx.x == 0) {
            unsigned cnt[3] = {0u, 0u, 0u};
            pair_result<kWeight, kHalf>(w, v, partner, s_at == 0x7fffffff ? -1 : s_at, contrib, cnt, bad);
            add_counts<kWeight>(cnt, st);
        }
        __syncthreads();
    }
}

// Host side: the pair passes of one call.  st is followed by other[n], bad[n]
// (the check only) and queue[n]; all but the queue is cleared at once.
size_t pair_bytes(int n) { return 128 + sizeof(int) * 3 * (size_t)n; }
static_assert(sizeof(PairState) <= 128, "the arrays follow it");

template <bool kWeight, bool kHalf>
cudaError_t launch_pairs(const mm_graph *g, const int *d_match, double *contrib, PairState *st, cudaStream_t s)
{
    const int n = g->n;
    int *other = reinterpret_cast<int *>(reinterpret_cast<char *>(st) + 128), *bad = other + n, *queue = bad + n;
    const cudaError_t e = cudaMemsetAsync(st, 0, 128 + sizeof(int) * (kWeight || kHalf ? 1 : 2) * (size_t)n, s);
    if (e != cudaSuccess) return e;
    k_pairs<<<grid_for(n, 256, 148 * 8), 256, 0, s>>>(d_match, n, other, st);
    const long long per = n > 0 ? g->nnz / n : 0;
    auto run = [&](auto kernel) {
        kernel<<<grid_for(n, 256, 148 * kPairBlocks), 256, 0, s>>>(g->d_ranges, g->d_nbrs, g->d_w, d_match, n, other, bad, queue,
                                                                   contrib, st);
    };
    if (per <= 20) run(k_pair_lists<4, kWeight, kHalf>);
    else if (per <= 80) run(k_pair_lists<8, kWeight, kHalf>);
    else run(k_pair_lists<32, kWeight, kHalf>);
    if (g->nnz > kPairList && !(g->scanned && g->max_degree <= kPairList))
        k_pair_long<kWeight, kHalf><<<148 * 4, 256, 0, s>>>(g->d_ranges, g->d_nbrs, g->d_w, d_match, other, bad, queue, contrib, st);
    return cudaGetLastError();
}

// getWeight: a matched vertex i adds the weight of the first entry of its list
// whose neighbour carries the same match value, and counts 1.  contrib[i]
// holds that weight (0 otherwise); size is counted alongside.
__global__ void k_weight(const int2 *ranges, const int *nbrs, const float *w, const int *match, int n,
                         double *contrib, PairState *st)
{
    if (clean(st)) return;
    unsigned long long cnt = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int m = match[i];
        double x = 0.0;
        if (is_matched(m)) {
            const int2 r = ranges[i];
            for (int j = r.x; j < r.y; ++j) {
                if (match[nbrs[j]] == m) {
                    x = (double)w[j];
                    ++cnt;
                    break;
                }
            }
        }
        contrib[i] = x;
    }
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(&st->size_general, cnt);
}

// Sort keys for testMatching's order: unmatched vertices first, then by match
// value; the sort is stable, so a value's vertices follow in increasing id.
__global__ void k_check_keys(const int *match, int n, unsigned *keys, int *ids)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int m = match[i];
        keys[i] = is_matched(m) ? (unsigned)m : 0u;
        ids[i] = i;
    }
}

// Is b in a's list?  Binary search when the graph's lists are sorted.
__device__ bool in_list(const int2 *ranges, const int *nbrs, int a, int b, bool sorted)
{
    const int2 r = ranges[a];
    if (r.y <= r.x) return false;
    if (sorted) {
        int lo = r.x, hi = r.y;
        while (lo < hi) {
            const int mid = (int)(((long long)lo + hi) >> 1);
            if (nbrs[mid] < b) lo = mid + 1;
            else hi = mid;
        }
        return lo < r.y && nbrs[lo] == b;
    }
    for (int j = r.x; j < r.y; ++j)
        if (nbrs[j] == b) return true;
    return false;
}

// testMatching walks the matched vertices in sorted order two at a time: i1,
// then i2.  A pair of equal values is checked (both must be in each other's
// lists, else "invalidly matched") and further vertices of that value are
// "multi-matched"; if i2's value differs, i1 is "under-matched" and i2 is
// consumed with it, so the walk enters i2's group at its second vertex.
// Per group of equal value (size s), the walk is a map of one bit: whether
// the group's first vertex was already consumed (c).  Entering with c:
//   s - c >= 2   pair (c, c + 1) checked, s - c - 2 multi-matched, leave 0
//   s - c == 1   one under-matched, leave 1 (the next group's first is consumed)
//   s - c == 0   nothing (the group was that consumed vertex), leave 0
// A prefix scan of the composed maps gives each group its c, exactly as the
// sequential walk would.
__global__ void k_group_flags(const unsigned *keys, int n, int *flag)
{
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x)
        flag[p] = keys[p] != 0u && (p == 0 || keys[p - 1] != keys[p]) ? 1 : 0;
}

__global__ void k_group_starts(const int *flag, const int *gidx, int n, int *starts)
{
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x)
        if (flag[p]) starts[gidx[p]] = p;
}

// bit c of a map: the bit it leaves for the next group when entered with c
__global__ void k_group_maps(const int *starts, int ngroups, uint8_t *maps)
{
    for (int gi = blockIdx.x * blockDim.x + threadIdx.x; gi < ngroups; gi += gridDim.x * blockDim.x) {
        const int s = starts[gi + 1] - starts[gi];
        const int out0 = s == 1 ? 1 : 0, out1 = s == 2 ? 1 : 0;
        maps[gi] = (uint8_t)(out0 | (out1 << 1));
    }
}

struct ComposeMaps {
    // a applies first, then b
    __host__ __device__ uint8_t operator()(uint8_t a, uint8_t b) const
    {
        const int r0 = (b >> (a & 1)) & 1, r1 = (b >> ((a >> 1) & 1)) & 1;
        return (uint8_t)(r0 | (r1 << 1));
    }
};

// counts: [0] under, [1] multi, [2] invalid
__global__ void k_group_eval(const int *starts, const uint8_t *prefix, int ngroups, const int *ids, const int2 *ranges,
                             const int *nbrs, int sorted, unsigned long long *counts)
{
    unsigned long long under = 0, multi = 0, invalid = 0;
    for (int gi = blockIdx.x * blockDim.x + threadIdx.x; gi < ngroups; gi += gridDim.x * blockDim.x) {
        const int c = prefix[gi] & 1;  // the composed maps of all earlier groups, entered with 0
        const int p = starts[gi], s = starts[gi + 1] - p, r = s - c;
        if (r >= 2) {
            const int i1 = ids[p + c], i2 = ids[p + c + 1];
            if (!in_list(ranges, nbrs, i1, i2, sorted != 0) || !in_list(ranges, nbrs, i2, i1, sorted != 0)) ++invalid;
            multi += (unsigned long long)(r - 2);
        } else if (r == 1) {
            ++under;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        under += __shfl_down_sync(0xffffffffu, under, o);
        multi += __shfl_down_sync(0xffffffffu, multi, o);
        invalid += __shfl_down_sync(0xffffffffu, invalid, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (under) atomicAdd(counts + 0, under);
        if (multi) atomicAdd(counts + 1, multi);
        if (invalid) atomicAdd(counts + 2, invalid);
    }
}

// Vertices that can still be matched: unmatched with an unmatched neighbour
// other than themselves.  counts[3] matchable, counts[4] unmatched.
__global__ void k_check_matchable(const int2 *ranges, const int *nbrs, const int *match, int n,
                                  unsigned long long *counts)
{
    unsigned long long matchable = 0, unmatched = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (is_matched(match[i])) continue;
        ++unmatched;
        const int2 r = ranges[i];
        for (int j = r.x; j < r.y; ++j) {
            const int u = nbrs[j];
            if (u != i && !is_matched(match[u])) {
                ++matchable;
                break;
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        matchable += __shfl_down_sync(0xffffffffu, matchable, o);
        unmatched += __shfl_down_sync(0xffffffffu, unmatched, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (matchable) atomicAdd(counts + 3, matchable);
        if (unmatched) atomicAdd(counts + 4, unmatched);
    }
}

struct DeviceScope {
    int prev = -1;
    explicit DeviceScope(int dev)
    {
        cudaGetDevice(&prev);
        if (prev != dev) cudaSetDevice(dev);
    }
    ~DeviceScope()
    {
        int cur = -1;
        cudaGetDevice(&cur);
        if (prev >= 0 && cur != prev) cudaSetDevice(prev);
    }
};

}  // namespace
}  // namespace mm

using namespace mm;

MM_API mm_status mm_matching_weight(mm_graph *g, const int *d_match, double *weight, long long *size, void *stream)
{
    if (!g || !weight || !size || (!d_match && g->n > 0)) {
        set_error("mm_matching_weight: null argument");
        return MM_ERR_ARG;
    }
    *weight = 0.0;
    *size = 0;
    if (g->n == 0) return MM_OK;
    DeviceScope scope(g->device);
    cudaStream_t st = (cudaStream_t)stream;
    const int n = g->n;
    double *contrib = nullptr;
    PairState *ps = nullptr;
    void *tmp = nullptr;
    size_t tmp_bytes = 0;
    cudaError_t e = dev_alloc((void **)&contrib, sizeof(double) * (size_t)n, st);
    if (e == cudaSuccess) e = dev_alloc((void **)&ps, pair_bytes(n), st);
    if (e == cudaSuccess) e = (g->sym_weights && g->no_self ? launch_pairs<true, true> : launch_pairs<true, false>)(g, d_match, contrib, ps, st);
    if (e == cudaSuccess) {
        k_weight<<<grid_for(n, 256, 148 * 8), 256, 0, st>>>(g->d_ranges, g->d_nbrs, g->d_w, d_match, n, contrib, ps);
        e = cudaGetLastError();
    }
    // a fixed reduction tree: the same sum on every run
    if (e == cudaSuccess) e = cub::DeviceReduce::Sum(nullptr, tmp_bytes, contrib, &ps->weight, n, st);
    if (e == cudaSuccess) e = dev_alloc(&tmp, tmp_bytes, st);
    if (e == cudaSuccess) e = cub::DeviceReduce::Sum(tmp, tmp_bytes, contrib, &ps->weight, n, st);
    PairState h = {};
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, ps, sizeof h, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    dev_free(tmp, st);
    dev_free(contrib, st);
    dev_free(ps, st);
    if (e != cudaSuccess) return cuda_fail(e, "mm_matching_weight");
    *weight = h.weight / 2.0;  // every matched edge is counted from both ends
    *size = (long long)(clean(&h) ? h.size : h.size_general);
    return MM_OK;
}

MM_API mm_status mm_matching_check(mm_graph *g, const int *d_match, long long *counts, int *valid, void *stream)
{
    if (!g || !counts || !valid || (!d_match && g->n > 0)) {
        set_error("mm_matching_check: null argument");
        return MM_ERR_ARG;
    }
    for (int k = 0; k < 5; ++k) counts[k] = 0;
    *valid = 1;
    if (g->n == 0) return MM_OK;
    DeviceScope scope(g->device);
    cudaStream_t st = (cudaStream_t)stream;
    const int n = g->n;
    cudaError_t e = cudaSuccess;
    {
        PairState *ps = nullptr;
        e = dev_alloc((void **)&ps, pair_bytes(n), st);
        if (e == cudaSuccess) e = (g->sym_struct ? launch_pairs<false, true> : launch_pairs<false, false>)(g, d_match, nullptr, ps, st);
        PairState h = {};
        if (e == cudaSuccess) e = cudaMemcpyAsync(&h, ps, sizeof h, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        dev_free(ps, st);
        if (e != cudaSuccess) return cuda_fail(e, "mm_matching_check");
        if (clean(&h)) {
            for (int k = 2; k < 5; ++k) counts[k] = (long long)h.counts[k];
            *valid = counts[2] == 0 ? 1 : 0;
            return MM_OK;
        }
    }
    // the reference's walk
    unsigned *k0 = nullptr, *k1 = nullptr;
    int *v0 = nullptr, *v1 = nullptr;
    unsigned long long *c = nullptr;
    void *tmp = nullptr;
    size_t tmp_bytes = 0;
    e = dev_alloc((void **)&k0, sizeof(unsigned) * (size_t)n, st);
    if (e == cudaSuccess) e = dev_alloc((void **)&k1, sizeof(unsigned) * (size_t)n, st);
    if (e == cudaSuccess) e = dev_alloc((void **)&v0, sizeof(int) * (size_t)n, st);
    if (e == cudaSuccess) e = dev_alloc((void **)&v1, sizeof(int) * (size_t)n, st);
    if (e == cudaSuccess) e = dev_alloc((void **)&c, sizeof(unsigned long long) * 5, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(c, 0, sizeof(unsigned long long) * 5, st);
    if (e == cudaSuccess) {
        k_check_keys<<<grid_for(n, 256, 148 * 8), 256, 0, st>>>(d_match, n, k0, v0);
        e = cudaGetLastError();
    }
    cub::DoubleBuffer<unsigned> kb(k0, k1);
    cub::DoubleBuffer<int> vb(v0, v1);
    if (e == cudaSuccess) e = cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, kb, vb, n, 0, 32, st);
    if (e == cudaSuccess) e = dev_alloc(&tmp, tmp_bytes, st);
    if (e == cudaSuccess) e = cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, kb, vb, n, 0, 32, st);
    // groups of equal value: starts, per-group maps, their prefix composition, counts
    int *flag = nullptr, *gidx = nullptr, *starts = nullptr;
    uint8_t *maps = nullptr, *prefix = nullptr;
    void *tmp2 = nullptr;
    size_t tmp2_bytes = 0;
    int ngroups = 0;
    if (e == cudaSuccess) e = dev_alloc((void **)&flag, sizeof(int) * (size_t)n, st);
    if (e == cudaSuccess) e = dev_alloc((void **)&gidx, sizeof(int) * (size_t)n, st);
    if (e == cudaSuccess) {
        k_group_flags<<<grid_for(n, 256, 148 * 8), 256, 0, st>>>(kb.Current(), n, flag);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(nullptr, tmp2_bytes, flag, gidx, n, st);
    if (e == cudaSuccess) e = dev_alloc(&tmp2, tmp2_bytes, st);
    if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(tmp2, tmp2_bytes, flag, gidx, n, st);
    int last[2] = {0, 0};
    if (e == cudaSuccess) e = cudaMemcpyAsync(&last[0], gidx + n - 1, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&last[1], flag + n - 1, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    dev_free(tmp2, st);
    tmp2 = nullptr;
    if (e == cudaSuccess) ngroups = last[0] + last[1];
    if (e == cudaSuccess && ngroups > 0) {
        e = dev_alloc((void **)&starts, sizeof(int) * ((size_t)ngroups + 1), st);
        if (e == cudaSuccess) e = dev_alloc((void **)&maps, (size_t)ngroups, st);
        if (e == cudaSuccess) e = dev_alloc((void **)&prefix, (size_t)ngroups, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(starts + ngroups, &n, sizeof(int), cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) {
            k_group_starts<<<grid_for(n, 256, 148 * 8), 256, 0, st>>>(flag, gidx, n, starts);
            k_group_maps<<<grid_for(ngroups, 256, 148 * 8), 256, 0, st>>>(starts, ngroups, maps);
            e = cudaGetLastError();
        }
        tmp2_bytes = 0;
        if (e == cudaSuccess)
            e = cub::DeviceScan::ExclusiveScan(nullptr, tmp2_bytes, maps, prefix, ComposeMaps(), (uint8_t)2, ngroups, st);
        if (e == cudaSuccess) e = dev_alloc(&tmp2, tmp2_bytes, st);
        if (e == cudaSuccess)
            e = cub::DeviceScan::ExclusiveScan(tmp2, tmp2_bytes, maps, prefix, ComposeMaps(), (uint8_t)2, ngroups, st);
        if (e == cudaSuccess) {
            k_group_eval<<<grid_for(ngroups, 256, 148 * 8), 256, 0, st>>>(starts, prefix, ngroups, vb.Current(),
                                                                          g->d_ranges, g->d_nbrs,
                                                                          g->sym_struct ? 1 : 0, c);
            e = cudaGetLastError();
        }
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);  // n above is a host value copied asynchronously
    dev_free(tmp2, st);
    dev_free(flag, st);
    dev_free(gidx, st);
    dev_free(starts, st);
    dev_free(maps, st);
    dev_free(prefix, st);
    if (e == cudaSuccess) {
        k_check_matchable<<<grid_for(n, 256, 148 * 8), 256, 0, st>>>(g->d_ranges, g->d_nbrs, d_match, n, c);
        e = cudaGetLastError();
    }
    unsigned long long h[5] = {0, 0, 0, 0, 0};
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, c, sizeof h, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    dev_free(tmp, st);
    dev_free(k0, st);
    dev_free(k1, st);
    dev_free(v0, st);
    dev_free(v1, st);
    dev_free(c, st);
    if (e != cudaSuccess) return cuda_fail(e, "mm_matching_check");
    for (int k = 0; k < 5; ++k) counts[k] = (long long)h[k];
    *valid = (h[0] == 0 && h[1] == 0 && h[2] == 0) ? 1 : 0;
    return MM_OK;
}
