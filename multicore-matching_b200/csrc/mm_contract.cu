// mm_contract.cu -- contraction of a matched graph (one level of multilevel coarsening).
//
// No counterpart in the reference, which stops at the matching; this is the
// step that multilevel partitioners put after it.  Each matched pair becomes
// one coarse vertex and every unmatched vertex stays one; the coarse lists
// hold the members' entries mapped to coarse ids, in increasing id, without
// self-loops, and an edge that several fine entries map to carries the sum of
// their weights.  The sum is taken in double, in the members' list order, and
// rounded once: the coarse graph of a symmetric graph is symmetric again,
// weights included (exactly so while the weights' sum fits a double's
// mantissa, as for weights on a common 2^-k grid).
//
// A coarse list is the union of at most two short lists, so it is gathered,
// sorted and merged where it is: by the lanes of a warp up to 64 entries, in a
// warp's shared memory up to 128, in a block's up to 2048; only longer ones go
// through a segmented sort in global memory.  Nothing returns to the host
// before the merged sizes are known (one synchronisation), and the arrays that
// the last pass writes become the coarse graph's own.  On RGG 2^20 this takes
// the place of a segmented sort of all entries, seven passes over them, four
// synchronisations and a copy and a re-validation of the result (1430 us).
#include <cuda_runtime.h>
#include <cub/device/device_scan.cuh>
#include <cub/device/device_segmented_sort.cuh>

#include <climits>

#include "mm_common.cuh"

#define MM_API extern "C" __attribute__((visibility("default")))

namespace mm {
namespace {

constexpr unsigned kAll = 0xffffffffu;
constexpr int kWarpSort = 32, kSmemSort = 128, kBlockSort = 2048;  // longest list of each way
constexpr int kSmemWarps = 8;

__device__ __forceinline__ int degree_of(int2 r) { return r.y > r.x ? r.y - r.x : 0; }

// What a contraction reports, and the lists left to the later ways.
struct ContractState {
    int bad;                   // the match array is not a matching
    int nsmem, nblock, nlong;  // queued lists
    long long long_entries;    // entries of the long ones
    unsigned long long skew_s, skew_w;  // symmetry sums of the coarse graph (0: symmetric)
};

// The representative of v: the smaller vertex of its pair (the match value
// minus 4), or v.  A value naming no vertex, or a vertex that does not name it
// back, is an invalid matching.
__device__ __forceinline__ int rep_of(const int *match, int n, int v, bool &bad)
{
    const int m = match[v];
    if (m < 4) return v;
    const long long a = (long long)m - 4;
    if (a >= n || match[a] != m) {
        bad = true;
        return v;
    }
    return (int)a;
}

__global__ void k_reps(const int *match, int n, int *flag, ContractState *st)
{
    bool bad = false;
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v <= n; v += gridDim.x * blockDim.x)
        flag[v] = v < n && rep_of(match, n, v, bad) == v ? 1 : 0;
    if (bad) atomicOr(&st->bad, 1);
}

// cmap[v] = coarse id of v's representative; mem[c] = the members of c (-1:
// none), cleared to -1 before.  A second vertex without entries adds nothing and
// needs no place; a third one with entries is no matching.
__global__ void k_members(const int *match, const int2 *ranges, const int *cid, int n, int *cmap, int2 *mem, ContractState *st)
{
    bool bad = false;
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const int r = rep_of(match, n, v, bad), c = cid[r];
        cmap[v] = c;
        if (r == v) mem[c].x = v;
        else if (degree_of(ranges[v]) > 0 && atomicExch(&mem[c].y, v) != -1) bad = true;
    }
    if (bad) atomicOr(&st->bad, 1);
}

// Upper bounds of the coarse lists' lengths (0 past the last one).
__global__ void k_lengths(const int2 *ranges, const int2 *mem, const int *cid, int n, long long *len)
{
    const int nc = cid[n];
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c <= n; c += gridDim.x * blockDim.x) {
        long long l = 0;
        if (c < nc) {
            const int2 m = mem[c];
            l = degree_of(ranges[m.x]) + (m.y >= 0 ? (long long)degree_of(ranges[m.y]) : 0ll);
        }
        len[c] = l;
    }
}

// Members' entries of coarse vertex c: entry i of the first list, then of the second.
struct Entries {
    int2 a, b;
    int da, db;
    __device__ __forceinline__ Entries(const int2 *ranges, int2 m)
    {
        a = ranges[m.x];
        b = m.y >= 0 ? ranges[m.y] : make_int2(0, 0);
        da = degree_of(a);
        db = degree_of(b);
    }
    __device__ __forceinline__ int pos(long long i) const { return (int)(i < da ? a.x + i : b.x + (i - da)); }
    __device__ __forceinline__ long long total() const { return (long long)da + db; }
};

// Sort keys across groups of S lanes, ascending (a bitonic network).
template <int S, class K>
__device__ __forceinline__ void group_sort(K &k, int lane)
{
#pragma unroll
    for (int size = 2; size <= S; size <<= 1)
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            const K o = __shfl_xor_sync(kAll, k, stride);
            const bool up = (lane & size) == 0 || size == S, low = (lane & stride) == 0;
            k = low == up ? min(k, o) : max(k, o);
        }
}

// One lane's entry of coarse vertex c's lists (c < 0: none): its key holds the
// coarse neighbour and the entry's place (B bits), so equal neighbours keep the
// members' list order; self-loops are dropped.
template <int B, class K>
__device__ __forceinline__ void load_entry(const int *nbrs, const float *w, const int *cmap, const Entries &e, int c, int i,
                                           int place, K &key, float &wt)
{
    key = ~(K)0;
    wt = 0.0f;
    if (i < e.total()) {
        const int j = e.pos(i), cu = cmap[__ldg(nbrs + j)];
        wt = __ldg(w + j);
        if (cu != c) key = ((K)(unsigned)cu << B) | (K)place;
    }
}

// Coarse list of at most S entries from its group's loaded entries.
template <int S, class K>
__device__ __forceinline__ void merge_group(const long long *off, int c, K key, float wt, int *tkey, float *tw, int *cnt)
{
    const int lane = threadIdx.x & 31, l = lane & (S - 1), g0 = lane & ~(S - 1);
    const unsigned gmask = S == 32 ? kAll : ((1u << (S & 31)) - 1u) << g0;
    const long long o = c >= 0 ? off[c] : 0;
    group_sort<S, K>(key, lane);
    const bool in = key != ~(K)0;
    const K nb = key >> 5;
    wt = __shfl_sync(kAll, wt, in ? (int)(key & 31) : lane);
    const K before = __shfl_up_sync(kAll, nb, 1);
    const bool head = in && (l == 0 || before != nb);
    double sum = 0.0 + (double)wt;  // as every way sums: from 0, so a -0 alone becomes 0
    for (int d = 1; d < S; ++d) {
        const K other = __shfl_down_sync(kAll, nb, d);  // (a dropped entry's differs from every id)
        const float x = __shfl_down_sync(kAll, wt, d);
        const bool same = in && l + d < S && other == nb;
        if (same) sum += (double)x;  // a head's own run, in order
        if (!__any_sync(kAll, same)) break;
    }
    const unsigned heads = __ballot_sync(kAll, head) & gmask;
    if (head) {
        const int at = __popc(heads & ((1u << lane) - 1u));
        tkey[o + at] = (int)nb;
        tw[o + at] = (float)sum;
    }
    if (c >= 0 && l == 0) cnt[c] = __popc(heads);
}

// N coarse lists after one another, a group of S lanes each: the entries of
// all of them are loaded before the first is sorted (the loads are a chain of
// four, members, ranges, neighbours and their coarse ids).
template <int S, int N, class K>
__device__ __forceinline__ void sort_groups(const int2 *ranges, const int *nbrs, const float *w, const int *cmap,
                                            const int2 *mem, const long long *off, int here, int *tkey, float *tw, int *cnt)
{
    const int lane = threadIdx.x & 31, l = lane & (S - 1);
    K key[N];
    float wt[N];
    int c[N];
#pragma unroll
    for (int h = 0; h < N; ++h) {
        c[h] = N == 1 && S > 8 ? here : __shfl_sync(kAll, here, h * (32 / S) + lane / S);
        key[h] = ~(K)0;
        wt[h] = 0.0f;
        if (c[h] >= 0) load_entry<5, K>(nbrs, w, cmap, Entries(ranges, mem[c[h]]), c[h], l, lane, key[h], wt[h]);
    }
#pragma unroll
    for (int h = 0; h < N; ++h) merge_group<S, K>(off, c[h], key[h], wt[h], tkey, tw, cnt);
}

// A list of 33 to 64 entries by a warp, two a lane (places lane and lane + 32).
template <class K>
__device__ __forceinline__ void sort_pairs(const int2 *ranges, const int *nbrs, const float *w, const int *cmap,
                                           const int2 *mem, const long long *off, int c, int *tkey, float *tw, int *cnt,
                                           float *wt)
{
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const Entries e(ranges, mem[c]);
    K k0, k1;
    float w0, w1;
    load_entry<6, K>(nbrs, w, cmap, e, c, lane, lane, k0, w0);
    load_entry<6, K>(nbrs, w, cmap, e, c, lane + 32, lane + 32, k1, w1);
    wt[lane] = w0;
    wt[lane + 32] = w1;
    // bitonic network over 64 places: place lane in k0, lane + 32 in k1
#pragma unroll
    for (int size = 2; size <= 64; size <<= 1)
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride == 32) {
                const K lo = k0 < k1 ? k0 : k1, hi = k0 < k1 ? k1 : k0;
                k0 = lo;
                k1 = hi;
            } else {
                const K o0 = __shfl_xor_sync(kAll, k0, stride), o1 = __shfl_xor_sync(kAll, k1, stride);
                const bool low = (lane & stride) == 0;
                const bool up0 = size == 64 || (lane & size) == 0;
                const bool up1 = size == 64 || ((lane + 32) & size) == 0;
                k0 = low == up0 ? min(k0, o0) : max(k0, o0);
                k1 = low == up1 ? min(k1, o1) : max(k1, o1);
            }
        }
    __syncwarp();  // wt is complete
    const bool in0 = k0 != ~(K)0, in1 = k1 != ~(K)0;
    const K n0 = k0 >> 6, n1 = k1 >> 6;
    const K before0 = __shfl_up_sync(kAll, n0, 1), before1 = __shfl_up_sync(kAll, n1, 1), last0 = __shfl_sync(kAll, n0, 31);
    const bool h0 = in0 && (lane == 0 || before0 != n0), h1 = in1 && (lane == 0 ? last0 : before1) != n1;
    double s0 = 0.0 + (in0 ? (double)wt[(int)(k0 & 63)] : 0.0), s1 = 0.0 + (in1 ? (double)wt[(int)(k1 & 63)] : 0.0);
    for (int d = 1; d < 64; ++d) {  // runs, in order
        const int q0 = lane + d, q1 = lane + 32 + d;
        const K a0 = __shfl_sync(kAll, k0, q0 & 31), a1 = __shfl_sync(kAll, k1, q0 & 31);
        const K x0 = q0 < 32 ? a0 : a1;
        const bool m0 = h0 && q0 < 64 && x0 != ~(K)0 && (x0 >> 6) == n0;
        const bool m1 = h1 && q1 < 64 && a1 != ~(K)0 && (a1 >> 6) == n1;
        if (m0) s0 += (double)wt[(int)(x0 & 63)];
        if (m1) s1 += (double)wt[(int)(a1 & 63)];
        if (!__any_sync(kAll, m0 || m1)) break;
    }
    const unsigned b0 = __ballot_sync(kAll, h0), b1 = __ballot_sync(kAll, h1);
    const long long o = off[c];
    if (h0) {
        tkey[o + __popc(b0 & below)] = (int)n0;
        tw[o + __popc(b0 & below)] = (float)s0;
    }
    if (h1) {
        tkey[o + __popc(b0) + __popc(b1 & below)] = (int)n1;
        tw[o + __popc(b0) + __popc(b1 & below)] = (float)s1;
    }
    if (lane == 0) cnt[c] = __popc(b0) + __popc(b1);
    __syncwarp();  // wt is refilled by the next list
}

// All coarse vertices, a warp for four at a time: groups of 8 lanes if their
// lists are that short, else of 16, else the whole warp.  Longer lists are queued.
template <class K>
__global__ void __launch_bounds__(256) k_sort_warp(const int2 *ranges, const int *nbrs, const float *w, const int *cmap,
                                                   const int2 *mem, const long long *off, const int *cid, int n, int *tkey,
                                                   float *tw, int *cnt, int *qsmem, int *qblock, int *qlong, ContractState *st)
{
    const int nc = cid[n], lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    if (warp == 0 && lane == 0) cnt[nc] = 0;
    for (long long c0 = warp * 4; c0 < nc; c0 += nwarps * 4) {
        const int mine = c0 + (lane & 3) < nc ? (int)c0 + (lane & 3) : -1;
        const long long len = mine >= 0 ? off[mine + 1] - off[mine] : 0;
        if (lane < 4 && len > kWarpSort) {
            if (len <= kSmemSort) qsmem[atomicAdd(&st->nsmem, 1)] = mine;
            else if (len <= kBlockSort) qblock[atomicAdd(&st->nblock, 1)] = mine;
            else {
                qlong[atomicAdd(&st->nlong, 1)] = mine;
                atomicAdd((unsigned long long *)&st->long_entries, (unsigned long long)len);
            }
        }
        const int here = len <= kWarpSort ? mine : -1;
        const int most = __reduce_max_sync(kAll, here >= 0 ? (int)len : 0);
        if (most <= 8) {
            sort_groups<8, 1, K>(ranges, nbrs, w, cmap, mem, off, here, tkey, tw, cnt);
        } else if (most <= 16) {
            for (int h = 0; h < 2; ++h)
                sort_groups<16, 1, K>(ranges, nbrs, w, cmap, mem, off, __shfl_sync(kAll, here, 2 * h + (lane >> 4)), tkey, tw, cnt);
        } else {
            for (int h = 0; h < 4; ++h)
                sort_groups<32, 1, K>(ranges, nbrs, w, cmap, mem, off, __shfl_sync(kAll, here, h), tkey, tw, cnt);
        }
    }
}

// Queued lists, sorted in shared memory by T threads each (a warp or a block).
// Keys are {coarse neighbour, entry}: equal neighbours keep list order.
template <int T>
__device__ __forceinline__ void group_sync()
{
    if (T == 32) __syncwarp();
    else __syncthreads();
}

template <int T, int kCap>
__device__ __forceinline__ void sort_smem(const int2 *ranges, const int *nbrs, const float *w, const int *cmap,
                                          const int2 *mem, const long long *off, int c, int *tkey, float *tw, int *cnt,
                                          unsigned long long *key, float *wt, int *scan)
{
    const int tid = T == 32 ? threadIdx.x & 31 : threadIdx.x;
    const Entries e(ranges, mem[c]);
    const int len = (int)e.total();
    int size = 2;
    while (size < len) size <<= 1;
    for (int i = tid; i < size; i += T) {
        unsigned long long k = ~0ull;
        if (i < len) {
            const int j = e.pos(i), cu = cmap[__ldg(nbrs + j)];
            wt[i] = __ldg(w + j);
            if (cu != c) k = ((unsigned long long)(unsigned)cu << 32) | (unsigned)i;
        }
        key[i] = k;
    }
    group_sync<T>();
    for (int s = 2; s <= size; s <<= 1)
        for (int d = s >> 1; d > 0; d >>= 1) {
            for (int i = tid; i < size / 2; i += T) {
                const int lo = 2 * i - (i & (d - 1)), hi = lo + d;
                const unsigned long long x = key[lo], y = key[hi];
                if ((x > y) == ((lo & s) == 0)) {
                    key[lo] = y;
                    key[hi] = x;
                }
            }
            group_sync<T>();
        }
    // heads of runs, T at a time in order
    const long long o = off[c];
    int done = 0;
    for (int i0 = 0; i0 < size; i0 += T) {
        const int i = i0 + tid;
        const unsigned nb = i < size ? (unsigned)(key[i] >> 32) : 0xffffffffu;
        const bool head = nb != 0xffffffffu && (i == 0 || (unsigned)(key[i - 1] >> 32) != nb);
        const unsigned m = __ballot_sync(kAll, head);
        int at = __popc(m & ((1u << (threadIdx.x & 31)) - 1u)), all = __popc(m);
        if (T > 32) {
            __syncthreads();  // scan[] is reused
            if ((threadIdx.x & 31) == 0) scan[threadIdx.x >> 5] = all;
            __syncthreads();
            all = 0;
            for (int q = 0; q < T / 32; ++q) {
                if (q < (int)(threadIdx.x >> 5)) at += scan[q];
                all += scan[q];
            }
        }
        if (head) {
            double sum = 0.0;
            for (int q = i; q < size && (unsigned)(key[q] >> 32) == nb; ++q) sum += (double)wt[(unsigned)key[q]];
            tkey[o + done + at] = (int)nb;
            tw[o + done + at] = (float)sum;
        }
        done += all;
    }
    if (tid == 0) cnt[c] = done;
    group_sync<T>();  // the arrays are reused by the next list
}

template <class K>
__global__ void __launch_bounds__(32 * kSmemWarps) k_sort_smem(const int2 *ranges, const int *nbrs, const float *w,
                                                               const int *cmap, const int2 *mem, const long long *off,
                                                               int *tkey, float *tw, int *cnt, const int *q,
                                                               const ContractState *st)
{
    __shared__ unsigned long long key[kSmemWarps][kSmemSort];
    __shared__ float wt[kSmemWarps][kSmemSort];
    const int wi = threadIdx.x >> 5, count = st->nsmem;
    for (int i = blockIdx.x * kSmemWarps + wi; i < count; i += gridDim.x * kSmemWarps) {
        const int c = q[i];
        if (off[c + 1] - off[c] <= 64) sort_pairs<K>(ranges, nbrs, w, cmap, mem, off, c, tkey, tw, cnt, wt[wi]);
        else sort_smem<32, kSmemSort>(ranges, nbrs, w, cmap, mem, off, c, tkey, tw, cnt, key[wi], wt[wi], nullptr);
    }
}

__global__ void __launch_bounds__(256) k_sort_block(const int2 *ranges, const int *nbrs, const float *w, const int *cmap,
                                                    const int2 *mem, const long long *off, int *tkey, float *tw, int *cnt,
                                                    const int *q, const ContractState *st)
{
    __shared__ unsigned long long key[kBlockSort];
    __shared__ float wt[kBlockSort];
    __shared__ int scan[8];
    const int count = st->nblock;
    for (int i = blockIdx.x; i < count; i += gridDim.x)
        sort_smem<256, kBlockSort>(ranges, nbrs, w, cmap, mem, off, q[i], tkey, tw, cnt, key, wt, scan);
}

// Long lists: their lengths, their entries (INT_MAX for a self-loop, sorted
// last and dropped), and after the stable segmented sort their merged runs, a
// block each.
__global__ void k_long_lengths(const long long *off, const int *q, int count, long long *len)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= count; i += gridDim.x * blockDim.x)
        len[i] = i < count ? off[q[i] + 1] - off[q[i]] : 0;
}

__global__ void k_long_gather(const int2 *ranges, const int *nbrs, const float *w, const int *cmap, const int2 *mem,
                              const int *q, int count, const long long *loff, int *key, float *val)
{
    for (int i = blockIdx.x; i < count; i += gridDim.x) {
        const int c = q[i];
        const Entries e(ranges, mem[c]);
        const long long total = e.total(), o = loff[i];
        for (long long k = threadIdx.x; k < total; k += blockDim.x) {
            const int j = e.pos(k), cu = cmap[__ldg(nbrs + j)];
            key[o + k] = cu == c ? INT_MAX : cu;
            val[o + k] = __ldg(w + j);
        }
    }
}

__global__ void __launch_bounds__(256) k_long_merge(const long long *off, const int *q, int count, const long long *loff,
                                                    const int *key, const float *val, int *tkey, float *tw, int *cnt)
{
    __shared__ int scan[8];
    for (int i = blockIdx.x; i < count; i += gridDim.x) {
        const int c = q[i];
        const long long b = loff[i], e = loff[i + 1], o = off[c];
        long long done = 0;
        for (long long k0 = b; k0 < e; k0 += 256) {
            const long long k = k0 + threadIdx.x;
            const int nb = k < e ? key[k] : INT_MAX;
            const bool head = nb != INT_MAX && (k == b || key[k - 1] != nb);
            const unsigned m = __ballot_sync(kAll, head);
            int at = __popc(m & ((1u << (threadIdx.x & 31)) - 1u)), all = 0;
            __syncthreads();  // scan[] is reused
            if ((threadIdx.x & 31) == 0) scan[threadIdx.x >> 5] = __popc(m);
            __syncthreads();
            for (int x = 0; x < 8; ++x) {
                if (x < (int)(threadIdx.x >> 5)) at += scan[x];
                all += scan[x];
            }
            if (head) {
                double sum = 0.0;
                for (long long x = k; x < e && key[x] == nb; ++x) sum += (double)val[x];
                tkey[o + done + at] = nb;
                tw[o + done + at] = (float)sum;
            }
            done += all;
        }
        if (threadIdx.x == 0) cnt[c] = (int)done;
    }
}

// The coarse graph from the merged lists (8 lanes a list): ranges, entries,
// and the symmetry sums of what they hold; and the caller's copy of the coarse
// map (null: none), which is written here, last, as it may be the match array
// itself and a refused call leaves it as it is.
__global__ void __launch_bounds__(256) k_emit(const int *tkey, const float *tw, const long long *off, const int *cnt,
                                              const long long *roff, int nc, int2 *ranges, int *out_nbr,
                                              float *out_w, const int *cmap, int *map_out, int n, ContractState *st)
{
    constexpr int G = 8;
    if (map_out)
        for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x)
            map_out[v] = cmap[v];
    const int l = threadIdx.x & (G - 1);
    const long long stride = (long long)gridDim.x * blockDim.x / G;
    unsigned long long ss = 0, sw = 0;
    for (long long c = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / G; c < nc; c += stride) {
        const long long o = off[c], r = roff[c];
        const int k = cnt[c];
        if (l == 0) ranges[c] = make_int2((int)r, (int)(r + k));
        for (int i0 = l; i0 < k; i0 += 4 * G) {
            int u[4];
            float x[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int i = i0 + q * G;
                u[q] = i < k ? tkey[o + i] : (int)c;
                x[q] = i < k ? tw[o + i] : 0.0f;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int i = i0 + q * G;
                if (i < k) {
                    out_nbr[r + i] = u[q];
                    out_w[r + i] = x[q];
                }
                add_skew((unsigned)c, (unsigned)u[q], __float_as_uint(x[q]), true, ss, sw);  // (c, c) adds nothing
            }
        }
    }
    block_add(&st->skew_s, ss);
    block_add(&st->skew_w, sw);
}

struct Scratch {
    static constexpr int kMax = 32;
    void *p[kMax] = {};
    int k = 0;
    cudaStream_t st;
    explicit Scratch(cudaStream_t s) : st(s) {}
    template <class T>
    cudaError_t get(T **out, size_t count)
    {
        if (k == kMax) return cudaErrorMemoryAllocation;
        cudaError_t e = dev_alloc((void **)out, sizeof(T) * (count ? count : 1), st);
        if (e == cudaSuccess) p[k++] = *out;
        return e;
    }
    template <class T>
    void keep(T *x)  // not freed here any more
    {
        for (int i = 0; i < k; ++i)
            if (p[i] == (void *)x) p[i] = nullptr;
    }
    ~Scratch()
    {
        for (int i = 0; i < k; ++i) dev_free(p[i], st);
        cudaStreamSynchronize(st);
    }
    template <class In, class Out>
    cudaError_t sums(const In *in, Out *out, size_t count)
    {
        void *tmp = nullptr;
        size_t tb = 0;
        cudaError_t e = cub::DeviceScan::ExclusiveSum(nullptr, tb, in, out, count, st);
        if (e == cudaSuccess) e = get((char **)&tmp, tb);
        if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(tmp, tb, in, out, count, st);
        return e;
    }
};

template <class T>
cudaError_t read_back(T *host, const T *dev, cudaStream_t st)
{
    return cudaMemcpyAsync(host, dev, sizeof(T), cudaMemcpyDeviceToHost, st);
}

__global__ void k_widen(const int *cnt, const int *cid, int n, long long *out)
{
    const int nc = cid[n];
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c <= n; c += gridDim.x * blockDim.x) out[c] = c < nc ? cnt[c] : 0;
}

mm_status contract(mm_graph *g, const int *d_match, mm_graph **coarse, int *d_cmap)
{
    const int n = g->n;
    cudaStream_t st = 0;
    Scratch sc(st);
    ContractState *cs = nullptr, h = {};
    int *flag = nullptr, *cid = nullptr, *cmap = nullptr, *cnt = nullptr, *q = nullptr;
    int2 *mem = nullptr;
    long long *len = nullptr, *off = nullptr, *roff = nullptr;
    const size_t nv = (size_t)n + 1;
    cudaError_t e = sc.get(&cs, 1);
    if (e == cudaSuccess) e = sc.get(&flag, nv);
    if (e == cudaSuccess) e = sc.get(&cid, nv);
    if (e == cudaSuccess) e = sc.get(&mem, nv);
    if (e == cudaSuccess) e = sc.get(&len, nv);
    if (e == cudaSuccess) e = sc.get(&off, nv);
    if (e == cudaSuccess) e = sc.get(&roff, nv);
    if (e == cudaSuccess) e = sc.get(&cnt, nv);
    if (e == cudaSuccess) e = sc.get(&q, 3 * nv);
    if (e == cudaSuccess) e = sc.get(&cmap, nv);
    if (e == cudaSuccess) e = cudaMemsetAsync(cs, 0, sizeof(ContractState), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(mem, 0xff, sizeof(int2) * nv, st);
    const int gv = grid_for(n + 1ll, 256, 148 * 64);  // a vertex a thread: the passes are chains of gathers
    if (e == cudaSuccess) {
        k_reps<<<gv, 256, 0, st>>>(d_match, n, flag, cs);
        e = sc.sums(flag, cid, nv);
    }
    if (e == cudaSuccess) {
        k_members<<<gv, 256, 0, st>>>(d_match, g->d_ranges, cid, n, cmap, mem, cs);
        k_lengths<<<gv, 256, 0, st>>>(g->d_ranges, mem, cid, n, len);
        e = sc.sums(len, off, nv);
    }
    // entries before merging: known for lists that tile the arrays
    long long total = g->nnz;
    if (e == cudaSuccess && !g->sym_struct) {
        e = read_back(&total, off + n, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    }
    int *tkey = nullptr;
    float *tw = nullptr;
    if (e == cudaSuccess) e = sc.get(&tkey, (size_t)total);
    if (e == cudaSuccess) e = sc.get(&tw, (size_t)total);
    int *qsmem = q, *qblock = q + nv, *qlong = q + 2 * nv;
    if (e == cudaSuccess && n > 0) {
        const int gw = grid_for((nv + 3) / 4 * 32, 256, 148 * 16);
        // a 32-bit key holds the coarse id and one of 64 places
        auto sorts = [&](auto key) {
            typedef decltype(key) K;
            k_sort_warp<K><<<gw, 256, 0, st>>>(g->d_ranges, g->d_nbrs, g->d_w, cmap, mem, off, cid, n, tkey, tw, cnt, qsmem,
                                               qblock, qlong, cs);
            k_sort_smem<K><<<148 * 8, 32 * kSmemWarps, 0, st>>>(g->d_ranges, g->d_nbrs, g->d_w, cmap, mem, off, tkey, tw, cnt,
                                                                qsmem, cs);
        };
        if (n < (1 << 26) - 1) sorts(0u);
        else sorts(0ull);
        k_sort_block<<<148 * 4, 256, 0, st>>>(g->d_ranges, g->d_nbrs, g->d_w, cmap, mem, off, tkey, tw, cnt, qblock, cs);
        e = cudaGetLastError();
    }
    long long ne = 0;
    int nc = 0;
    auto sizes = [&]() {
        k_widen<<<gv, 256, 0, st>>>(cnt, cid, n, len);
        cudaError_t x = sc.sums(len, roff, nv);
        if (x == cudaSuccess) x = read_back(&ne, roff + n, st);
        if (x == cudaSuccess) x = read_back(&nc, cid + n, st);
        if (x == cudaSuccess) x = read_back(&h, cs, st);
        if (x == cudaSuccess) x = cudaStreamSynchronize(st);
        return x;
    };
    if (e == cudaSuccess) e = sizes();
    if (e == cudaSuccess && h.bad) {
        set_error("mm_graph_contract: the match array is not a matching (a value names no partner that names it back)");
        return MM_ERR_ARG;
    }
    if (e == cudaSuccess && h.nlong > 0) {
        long long *llen = nullptr, *loff = nullptr;
        int *k0 = nullptr, *k1 = nullptr;
        float *v0 = nullptr, *v1 = nullptr;
        const size_t lt = (size_t)h.long_entries;
        e = sc.get(&llen, (size_t)h.nlong + 1);
        if (e == cudaSuccess) e = sc.get(&loff, (size_t)h.nlong + 1);
        if (e == cudaSuccess) e = sc.get(&k0, lt);
        if (e == cudaSuccess) e = sc.get(&k1, lt);
        if (e == cudaSuccess) e = sc.get(&v0, lt);
        if (e == cudaSuccess) e = sc.get(&v1, lt);
        if (e == cudaSuccess) {
            k_long_lengths<<<grid_for(h.nlong + 1, 256), 256, 0, st>>>(off, qlong, h.nlong, llen);
            e = sc.sums(llen, loff, (size_t)h.nlong + 1);
        }
        if (e == cudaSuccess) {
            k_long_gather<<<min(h.nlong, 148 * 8), 256, 0, st>>>(g->d_ranges, g->d_nbrs, g->d_w, cmap, mem, qlong, h.nlong, loff,
                                                                 k0, v0);
            size_t tb = 0;
            void *tmp = nullptr;
            // stable: equal neighbours keep the members' list order
            e = cub::DeviceSegmentedSort::StableSortPairs(nullptr, tb, k0, k1, v0, v1, h.long_entries, h.nlong, loff, loff + 1, st);
            if (e == cudaSuccess) e = sc.get((char **)&tmp, tb);
            if (e == cudaSuccess)
                e = cub::DeviceSegmentedSort::StableSortPairs(tmp, tb, k0, k1, v0, v1, h.long_entries, h.nlong, loff, loff + 1, st);
        }
        if (e == cudaSuccess) {
            k_long_merge<<<min(h.nlong, 148 * 8), 256, 0, st>>>(off, qlong, h.nlong, loff, k1, v1, tkey, tw, cnt);
            e = sizes();
        }
    }
    if (e != cudaSuccess) return cuda_fail(e, "mm_graph_contract");
    if (ne >= (1ll << 31)) {
        set_error("mm_graph_create: nnz must fit the reference's int indices (< 2^31)");
        return MM_ERR_UNSUPPORTED;
    }
    // the last pass writes the coarse graph's own arrays (padded as an upload's)
    int2 *cranges = nullptr;
    int *out_nbr = nullptr;
    float *out_w = nullptr;
    const size_t pad = padded_entries(ne);
    e = sc.get(&cranges, (size_t)nc);
    if (e == cudaSuccess) e = sc.get(&out_nbr, pad);
    if (e == cudaSuccess) e = sc.get(&out_w, pad);
    if (e == cudaSuccess) e = cudaMemsetAsync(out_nbr + ne, 0, (pad - (size_t)ne) * sizeof(int), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(out_w + ne, 0, (pad - (size_t)ne) * sizeof(float), st);
    if (e == cudaSuccess && nc > 0) {
        k_emit<<<grid_for(nc * 8ll, 256, 148 * 8), 256, 0, st>>>(tkey, tw, off, cnt, roff, nc, cranges, out_nbr, out_w, cmap, d_cmap, n,
                                                               cs);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = read_back(&h, cs, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_fail(e, "mm_graph_contract");
    mm_status s = adopt_arrays(g->device, nc, ne, cranges, out_nbr, out_w, nc > 0 && h.skew_s == 0, h.skew_w == 0, coarse);
    if (s == MM_OK) {
        sc.keep(cranges);
        sc.keep(out_nbr);
        sc.keep(out_w);
    }
    return s;
}

}  // namespace
}  // namespace mm

using namespace mm;

MM_API mm_status mm_graph_contract(mm_graph *g, const int *d_match, mm_graph **coarse, int *d_cmap)
{
    if (!g || !coarse || (!d_match && g->n > 0)) {
        set_error("mm_graph_contract: null argument");
        return MM_ERR_ARG;
    }
    *coarse = nullptr;
    int prev = -1;
    cudaGetDevice(&prev);
    if (prev != g->device) MM_CUDA_TRY(cudaSetDevice(g->device), "set device");
    const mm_status result = contract(g, d_match, coarse, d_cmap);
    if (prev >= 0 && prev != g->device) cudaSetDevice(prev);
    return result;
}
