// mm_push.cu -- the B200 round loop ("push" path).
//
// Same matching as the reference's GPU round (src/matchgpu.cu:184-451), with
// the work re-cut so that each round streams only the adjacency lists of BLUE
// vertices, and the whole loop runs in one cooperative kernel launch.
//
// Reformulation (exact, for any CSR the reference accepts):
//   * Respond (grRespond / gwRespond, matchgpu.cu:329-357, 411-451) lets red r
//     pick, among its blue neighbours u with requests[u] == r, the entry of its
//     own list with the largest weight (strict >, starting from -1), earliest
//     position first; in random mode the earliest position.  That is the
//     maximum over r's list of a 64-bit key (weight order << 32 | ~position),
//     restricted to entries pointing at proposers.  For every adjacency slot
//     (v -> r) the preparation step stores revkey = the best such key among
//     r's entries pointing back at v (0 if none can ever be picked).  A blue
//     proposer then atomicMax-es its revkey into best[r]; the maximum over
//     proposers equals the maximum over r's list.  Red vertices never scan.
//   * Commit (gMatch, matchgpu.cu:260-283): red r is matched iff best[r] is
//     non-zero (its partner is neighbours[~low32(key)]); blue u is matched iff
//     the low 32 bits of best[its target] equal the low 32 bits of its own
//     revkey (positions in r's list are unique).
//   * Select (gaSelect, matchgpu.cu:220-258) of round t+1 is fused into the
//     commit pass of round t: a survivor recolours itself with seed t+1.
//   * Dead marking (requests == n+1) happens as soon as the blue scan finds no
//     unmatched neighbour; readers of its colour see "unmatched, not red"
//     either way, so their outcome is unchanged.
//
// Work layout.  Every vertex belongs to one block for the whole matching: the
// vertices are dealt to the blocks in chunks of 64, and a block keeps the ones
// that can still be matched in lists of its own (4 bytes an item: the vertex).
// So no counter, list or request is shared between blocks: all that crosses
// them are the colours, the proposals' atomic maxima and the barriers.
//   windows        a blue vertex's choice is the first red candidate among its
//                  best min(deg, 32) entries in order of preference (weight,
//                  then position; list order for random types), stored at
//                  preparation.  A lane holds one vertex and reads eight
//                  window entries a step, refilled from a prefetched item as
//                  soon as its vertex is decided (scan_window).
//   fallback       a list longer than its window with no red candidate in it
//                  is scanned whole, by a warp or by the block that owns it;
//                  the longest lists (hubs), and on dense graphs all of a block
//                  that has many, go to a list of the round that all blocks
//                  share, cut into 2048-entry pieces (scan_shared).
//   finish phase   once the active set is small its components are tiny, and
//                  the remaining rounds of each component are played on their
//                  own, with two more grid barriers in all (finish_scan,
//                  finish_roots).
// A list's best entry is kept as a 64-bit key (weight order << 32 | ~position),
// which orders ties by position exactly as the reference's strict ">" scan in
// list order does.
//
// Loop.  k_match is launched cooperatively (all blocks resident) and runs
// set-up, then per round the window scan (A1, with the owner's fallback
// scans), the shared fallback scan (A2, only in rounds that have such lists)
// and the commit phase (B: commit + recolour + worklist compaction), with
// bounded grid barriers in between.  A barrier carries a sum (the vertices
// still active, the blocks with shared fallback lists), so nothing else has to
// be read to decide what comes next.  A graph that fits one block runs
// without grid barriers at all.  Nothing returns to the host until the
// matching is maximal (the reference copies a flag back every round,
// matchgpu.cu:607-614): the call is one launch, its arguments (seeds among
// them) travel as launch parameters and its result is written to host memory.
#include <cuda_runtime.h>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <climits>
#include <cstddef>
#include <cmath>
#include <cstring>
#include <mutex>
#include <new>

#include "mm_common.cuh"

namespace mm {
namespace {

constexpr int kThreads = 512;            // threads per block of the round kernel
constexpr int kWarps = kThreads / 32;
constexpr unsigned kFull = 0xffffffffu;
constexpr int kWin = 32;                 // preference window: the first min(deg, 32) choices
constexpr int kChunk = 64;               // vertices dealt to the blocks at a time
constexpr int kPiece = 2048;             // shared fallback lists: entries a warp scans

// Request codes of a blue item (a target vertex otherwise).
enum : int { kReqDead = -1, kReqNone = -2, kReqShared = -3 };

// Control block of one call, zero at launch.  A graph has two, used by
// alternate calls: each call clears the other one, so no call pays for a
// memory operation ahead of its launch.
constexpr int kRing = 4;        // barrier words in use by turns
constexpr int kRingStride = 16; // words of 8 bytes per barrier line (128 bytes)
struct Ctl {
    unsigned long long ring[kRing * kRingStride];  // (sum << 32) | blocks arrived
    unsigned long long staged_pack;  // shared fallback list of the round: (items << 32) | pieces
    int fin_abort;         // finish phase: t + 1 if the attempt in round t was called off
    int fin_last;          // finish phase: last round in which any of its vertices was active
    int iso_last;          // 1 + the last round in which a vertex without neighbours was active (0: none)
    int pad;
};

// What a call returns, in page-locked host memory that the kernel writes.
struct Result {
    int rounds;            // rounds the reference executes (-1: the kernel did not end its loop)
    int status;            // 0 ok, 1 seeds exhausted, 2 a bounded grid-barrier wait gave up
};

struct Params {
    int n;
    int contiguous;
    int sym;                        // proposal keys computed from the proposer's entry (no reverse index)
    int region;                     // list slots of a block
    int share_from;                 // fallback lists of a block from which it leaves them to all blocks
    uint32_t turn_magic;            // floor(2^32 / blocks) + 1
    const int2 *ranges;
    const int *nbrs;
    const float *w;
    const unsigned long long *revkey;
    const long long *slot_off;
    // weighted: preference windows in groups of four entries (32 bytes, one
    // load), {neighbour, weight} on the symmetric path, else {neighbour,
    // position | flag}; the last group is filled up with {-1, flag}
    const int2 *pwin;
    const int *pwin_off;            // weighted, [n + 1]: first group, bit 31: list longer than the window
    uint32_t *col;                  // colours, two bits a vertex
    int2 *req;                      // per vertex: proposal of a shared fallback list {target or code, key low half};
                                    // finish phase: a vertex's record
    int *lists[2];                  // items (vertices) by round parity: block b's region starts at b * region,
                                    // blue items from its front, red items from its back
    int *prop;                      // per blue item: target or code
    uint32_t *prop_key;             // per blue item, off the symmetric path: the proposal key's low half
    unsigned long long *best;       // per red vertex: max proposal key this round
    unsigned long long *part_key;   // per cut fallback list: max over finished pieces
    int *part_cnt;                  // per cut fallback list: finished pieces
    int4 *staged;                   // shared fallback items {v, begin, end, first piece}
    int *piece_item;                // per piece of the shared fallback lists: its item
    int fin;                        // the finish phase applies: lists symmetric in structure
    int4 *rec;                      // finish phase: records, rec_region of them for a block
    int rec_region;
    int rec_stride;                 // int4 a record: 3 on the symmetric path, else 4
    int *match;                     // output array of this call
    uint32_t barrier;
    int cap;                        // 20 or 255
    int maximal;
    int nseeds;
    Ctl *ctl;
    Ctl *ctl_next;                  // the next call's control block, cleared by this call
    Result *result;                 // host memory
    unsigned long long *stats;      // [kMaxRounds][MM_STATS_COLS] or null
    unsigned long long *tstamp;     // [3 * kMaxRounds + 1] barrier times (ns) or null
    int zero_parts;                 // set-up clears part_key and part_cnt (not known to be zero)
    int fin_div;                    // finish phase from the round whose active set is <= 1/fin_div of round 0's (0: never)
    // testing hooks (mm_debug): polls before a barrier wait gives up, and the
    // mark of a barrier at which block 0 does not arrive (-1: none)
    long long spin_limit;
    int skip_mark;
    // A batch of independent graphs (a disjoint union, edges never cross): each
    // vertex's graph starts at vbase[v], and the graph's own numbering (v -
    // vbase[v]) drives the colouring and the match values, so every graph gets
    // the matching a call on it alone would give.  last[v] is the last round
    // at whose colouring v was still unmatched, written once, when v leaves.
    // Both null for one graph.
    const int *vbase;
    uint8_t *last;
    // Learned colouring (k_match<..., kPolicy>): blue iff hash < p_v * 2^32 with
    // p_v from a per-vertex MLP over local features.  wfeat[v]: (max, mean)
    // incident weight; trace: per round and vertex, the features, colour and
    // outcome (for training), or null.
    float level;
    const float2 *wfeat;
    float *trace;
    int trace_rounds;
    // A policy whose output weights are all zero ignores the features: its
    // threshold, computed once on the host, is policy_bar (policy_const = 1).
    int policy_const;
    uint32_t policy_bar;
    // Learned colouring with a constant policy: the finish phase plays the
    // remaining rounds under the policy's threshold and its retirement rule.
    int fin_retire;
    // The policy's weights and the colouring seeds travel by value in the
    // launch parameters: every thread reads the same one, so they come straight
    // from the constant bank, and no copy precedes the launch.
    float mlp[MM_POLICY_FLOATS];
    uint32_t seeds[256];
};
static_assert(sizeof(Params) <= 4096, "launch parameters stay within the classic 4 KB limit");

__device__ __forceinline__ int base_of(const Params &p, int v) { return p.vbase ? __ldg(p.vbase + v) : 0; }

__device__ __forceinline__ int degree_of(int2 r) { return r.y > r.x ? r.y - r.x : 0; }
__device__ __forceinline__ int degree_of(int4 it) { return it.z > it.y ? it.z - it.y : 0; }
__device__ __forceinline__ int win_len(int deg) { return deg < kWin ? deg : kWin; }

// Positions in scans.  A list may end at 2^31 - 1, where a step of up to kThreads
// * kRows entries beyond its end would wrap a signed position to a place before
// the list.  So a scan counts down what is left of its list, or a position that
// may lie beyond the end is unsigned (Pos; not for empty ranges, whose ends may
// be anything).
typedef unsigned Pos;

template <class P>
__device__ __forceinline__ void stat_add(const P &p, int round, int col, unsigned long long v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(kFull, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&p.stats[(size_t)round * MM_STATS_COLS + col], v);
}

// The vertex at slot k of this block's share, or -1: chunk q of block b is
// chunk q * gridDim.x + (b + 61 q) % gridDim.x of the vertex range.  The turn
// by 61 keeps a block off one residue: ids cluster by degree (R-MAT hubs have
// ids with low bits zero), and a plain stride of a multiple of 8 blocks would
// give every eighth block the hubs.  The remainder comes from a multiplication
// (exact: b + 61 q < 61 n / (64 blocks) + blocks, times blocks, stays below 2^32).
__device__ __forceinline__ int own_vertex(const Params &p, int k)
{
    const unsigned nb = gridDim.x, q = (unsigned)k / kChunk;
    const unsigned x = blockIdx.x + 61u * q;
    const unsigned c = nb == 1u ? q : q * nb + (x - __umulhi(x, p.turn_magic) * nb);
    const unsigned v = c * kChunk + (unsigned)k % kChunk;
    return v < (unsigned)p.n ? (int)v : -1;
}

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Colours are packed two bits a vertex, 16 to a word: the scans' gathers are
// bound by the sectors they request from L2, and a matching's colours then fit
// L1 (up to half a million vertices) or mostly hit it.  A chunk's words belong
// to one block, which changes them by atomic XOR.  What scans need to tell
// apart is red, matched and neither: a vertex that becomes unmatchable keeps
// its colour's bits (blue, or red where no unmatched vertex lists it).
__device__ __forceinline__ unsigned colour_bits(uint32_t word, int u)
{
    return __funnelshift_r(word, word, 2u * (unsigned)u) & 3u;  // the shift is taken modulo 32
}

// A matching's working arrays: in global memory, or (kSolo, a graph that one
// block matches) in that block's shared memory.
template <bool kSolo>
struct Mem {
    uint32_t *col_;
    unsigned long long *best_;
    __device__ __forceinline__ uint32_t word(int u) const { return col_[(unsigned)u >> 4]; }
    __device__ __forceinline__ unsigned col(int u) const { return colour_bits(word(u), u); }
    __device__ __forceinline__ void flip(int v, unsigned delta) const
    {
        atomicXor(col_ + ((unsigned)v >> 4), delta << (2u * ((unsigned)v & 15u)));
    }
    __device__ __forceinline__ unsigned long long best(int v) const { return kSolo ? best_[v] : __ldcg(best_ + v); }
    __device__ __forceinline__ void propose(int v, unsigned long long key) const { atomicMax(best_ + v, key); }
    // list items, streamed
    static __device__ __forceinline__ int item(const int *a) { return kSolo ? *a : __ldcs(a); }
    static __device__ __forceinline__ void put(int *a, int v)
    {
        if (kSolo) *a = v;
        else __stcs(a, v);
    }
};

// Key under which a blue vertex ranks a red neighbour at position j
// (gwRequest: strict > from -1, earliest j on ties; grRequest: earliest j).
// Every candidate key is >= 2^31, so the value 1 can stand for "an unmatched
// neighbour that is not a candidate" and a single max-reduction carries both
// the choice and the dead flag (0 = nothing unmatched seen).
template <bool kW>
__device__ __forceinline__ unsigned long long cand_key(int j, float w)
{
    if (kW) return w > -1.0f ? (((unsigned long long)weight_order(w) << 32) | (uint32_t)~j) : 1ull;
    return (unsigned long long)(uint32_t)~j;
}

// Key of a scan's best entry: weight order and position of its best red
// neighbour (the reference's rule: strict > from -1 in list order), else 1 if
// an unmatched neighbour was seen, else 0.
template <bool kW>
__device__ __forceinline__ unsigned long long strip_key(float bw, int bj, bool alive)
{
    if (bw > -1.0f) return kW ? (((unsigned long long)weight_order(bw) << 32) | (uint32_t)~bj)
                              : (unsigned long long)(uint32_t)~bj;
    return alive ? 1ull : 0ull;
}

// Fold one scanned entry (neighbour colour c, weight w, position j) into a
// lane's running best: strict > from -1 over increasing positions, so ties
// keep the earliest entry; in random mode the first red entry.
template <bool kW>
__device__ __forceinline__ void fold_entry(unsigned c, float w, int j, float &bw, int &bj, bool &alive)
{
    alive |= c != kMatched;
    if (c == kRed) {
        const float x = kW ? w : 0.0f;
        if (x > bw) {
            bw = x;
            bj = j;
        }
    }
}

constexpr int kRows = 4;    // fallback scans: rows of 32 entries per iteration

// Window scan: the block's lists that go to a fallback scan.
constexpr int kStageCap = 1024;
struct FallbackStage {
    int2 item[kStageCap];          // {vertex, list slot}
    unsigned short big[kStageCap]; // the ones the whole block scans
};

// Requests of the block's first kPropCap blue items, from the window scan to
// the commit (the rest are in global memory): a request is a 4-byte store of
// its own, which cost the scan of RGG 2^20's round 0 a fifth of its time.
constexpr int kPropCap = 4800;
struct Requests {
    int target[kPropCap];
};

constexpr int kPer = 4;  // items a lane handles at a time in the set-up and commit passes

// Set-up: a warp's stack of vertices without neighbours, {vertex, next round}.
constexpr int kIsoCap = 31 + 32 * kPer;
struct IsoStack {
    int2 item[kWarps][kIsoCap];
    uint32_t seeds[256];
};

// ---- finish phase: a warp's component ----
constexpr int kFinMembers = 32;    // members of a component played by one warp (one per lane)
constexpr int kFinEntries = 128;   // entries between members of one component

// One warp's component: members' first entry, the entries between members
// (preference key and the target's member slot), the members' colours of the
// round being played and the best proposal each received.
struct FinWarp {
    unsigned long long pref[kFinEntries];
    unsigned long long best[kFinMembers];
    int mem[kFinMembers];
    int eoff[kFinMembers + 1];
    uint8_t tgt[kFinEntries];
    uint8_t st[kFinMembers];
};

// Shared memory of the round kernel (dynamic); the phases' working areas share
// it.  Two blocks fit the 64 KB configuration, which leaves the rest to L1.
struct Smem {
    union {
        IsoStack iso;
        struct {
            FallbackStage fb;
            Requests req;
        };
        FinWarp fin[kWarps];
    };
    unsigned long long red_key[kWarps];   // block-wide list scan: the warps' best keys
    int count[2][2];                      // the block's items by round parity and colour
    unsigned sync_sum;                    // grid barrier: the sum it carried
    int sync_ok;
    int wnext;                            // window scan: next item of the block
    int stage_n;                          // window scan: fallback lists collected by the block
    int big_n;                            // window scan: of those, lists for the whole block
    int flag;                             // window scan: lists appended to the shared list; finish phase: called off
    int zero;                             // 0
};
static_assert(sizeof(Smem) <= 31 * 1024, "two blocks a multiprocessor in the 64 KB configuration");
constexpr size_t kSmemBytes = (sizeof(Smem) + 127) / 128 * 128;

// Graphs of at most this many vertices are matched by one block (unless their
// long lists are many, launch_match): its rounds need no grid barrier, and its
// working arrays follow in its shared memory.
constexpr int kSoloVertices = 4096;
struct SoloMem {
    unsigned long long best[kSoloVertices];
    int lists[2][kSoloVertices];
    uint32_t col[kSoloVertices / 16];
};
static_assert(kSoloVertices <= kPropCap, "its requests stay in shared memory too");

// Where a blue vertex's request goes: the item's slot (in shared memory, or
// past its capacity in global memory), or for shared fallback lists the
// vertex's own word.
struct ItemReq {
    const Params &p;
    Smem &sm;
    long long rbase;
    int i;
    __device__ __forceinline__ void put(int target, uint32_t low) const
    {
        if (i < kPropCap) sm.req.target[i] = target;
        else __stcs(p.prop + rbase + i, target);
        if (!p.sym) __stcs(p.prop_key + rbase + i, low);
    }
};
struct VertexReq {
    const Params &p;
    int v;
    __device__ __forceinline__ void put(int target, uint32_t low) const { __stcs(p.req + v, make_int2(target, (int)low)); }
};

// Blue vertex v proposes to `target`, the neighbour at position j of its list
// (begin = first position): the reverse key of that slot goes to best[target].
template <bool kW, bool kSolo, class Req>
__device__ __forceinline__ void propose_to(const Params &p, const Mem<kSolo> &m, Req rq, int v, int begin, int j, int target)
{
    unsigned long long rk;
    if (p.sym) {
        // target's entry for v has v's weight, and earlier positions in its
        // strictly increasing list hold smaller ids
        if (kW) {
            const float x = __ldg(p.w + j);
            rk = x > -1.0f ? (((unsigned long long)weight_order(x) << 32) | (uint32_t)~v) : 0ull;
        } else {
            rk = (unsigned long long)(uint32_t)~v;
        }
    } else {
        const long long slot = p.contiguous ? (long long)j : __ldg(p.slot_off + v) + (j - begin);
        rk = __ldg(p.revkey + slot);
    }
    if (rk) m.propose(target, rk);
    rq.put(target, (uint32_t)rk);
}

// Symmetric weighted path: blue v proposes to `target` through an entry of
// weight w (w > -1); the target's entry for v has the same weight, and v's id
// breaks ties (smaller first).
template <bool kSolo, class Req>
__device__ __forceinline__ void propose_weight(const Mem<kSolo> &m, Req rq, int v, float w, int target)
{
    const unsigned long long rk = ((unsigned long long)weight_order(w) << 32) | (uint32_t)~v;
    m.propose(target, rk);
    rq.put(target, (uint32_t)rk);
}

// Blue vertex v without a red choice: unmatchable if no neighbour is
// unmatched (requests == n + 1), else no proposal this round.
template <class Req>
__device__ __forceinline__ void no_proposal(const Params &p, Req rq, int v, bool alive, int t)
{
    if (!alive) {
        p.match[v] = 2;
        if (p.last) p.last[v] = (uint8_t)t;
        rq.put(kReqDead, 0u);
    } else {
        rq.put(kReqNone, 0u);
    }
}

// Adjacency entries the reference's request loop inspects for this vertex
// (random mode stops at the first red neighbour, at position j).
template <bool kW>
__device__ __forceinline__ unsigned long long request_seen(int begin, int deg, int j)
{
    if (kW || j < 0) return (unsigned long long)deg;
    return (unsigned long long)(j - begin + 1);
}

// Finish blue vertex v (entries from `begin`, deg of them) after a full scan whose result is `key`.
template <bool kW, bool kStats, bool kSolo, class Req>
__device__ __forceinline__ void propose_key(const Params &p, const Mem<kSolo> &m, Req rq, int v, int begin, int deg, unsigned long long key,
                                            int t)
{
    if (kStats) {
        const int j = key >= 2 ? (int)~(uint32_t)key : -1;
        atomicAdd(&p.stats[(size_t)t * MM_STATS_COLS + MM_ST_REQ_ENTRIES], request_seen<kW>(begin, deg, j));
        atomicAdd(&p.stats[(size_t)t * MM_STATS_COLS + MM_ST_BLUE_DEG], (unsigned long long)deg);
    }
    if (key < 2) {
        no_proposal(p, rq, v, key == 1, t);
        return;
    }
    const int j = (int)~(uint32_t)key;
    propose_to<kW>(p, m, rq, v, begin, j, __ldg(p.nbrs + j));
}

// ---- grid barrier ----
//
// The kernel is launched cooperatively, so all its blocks are resident at once
// and a barrier over them cannot deadlock on scheduling.  Each block adds
// (its summand, part[0] + part[1] in shared memory, << 32) | 1 to the barrier's word and polls until all blocks
// have: one release-add and one round trip after the last arrival (2500
// cycles over 148 blocks, where a two-level tree of counters took 3800), and
// the sum of the summands comes with it.  The words are used by turns; block 0
// clears the word after next, which every block has left behind since the
// barrier before.  A single block needs no word.  Each wait is bounded: after
// spin_limit polls (a testing hook, mm_debug, can set fewer) the block records
// status 2 and the kernel returns; the other blocks then give up at their next
// barrier.  Thread 0's release and acquire, with the block barriers around
// them, make every block's writes of the phase visible to every thread of
// every block afterwards.
__device__ __noinline__ bool grid_sync(Smem &sm, Ctl *ctl, unsigned &turn, const int *part, unsigned *sum, Result *result,
                                       unsigned long long *tstamp, int mark, long long spin_limit, int skip_mark)
{
    const unsigned nb = gridDim.x, w = turn & (kRing - 1);
    turn += 1;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        const unsigned add = (unsigned)(part[0] + part[1]);
        unsigned total = add;
        // testing hook: block 0 leaves this barrier out, so every wait on it runs out
        const bool skip = blockIdx.x == 0 && mark >= 0 && mark == skip_mark;
        if (nb > 1) {
            unsigned long long *word = ctl->ring + w * kRingStride;
            if (blockIdx.x == 0) ctl->ring[((w + 2) & (kRing - 1)) * kRingStride] = 0ull;
            if (!skip)
                asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(word),
                             "l"(((unsigned long long)add << 32) | 1ull)
                             : "memory");
            unsigned long long got;
            long long it = 0;
            for (;;) {
                asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(got) : "l"(word) : "memory");
                if ((unsigned)got == nb) break;
                if (++it > spin_limit) {
                    ok = 0;
                    break;
                }
                if (it > 4096) __nanosleep(100);
            }
            total = (unsigned)(got >> 32);
        } else if (skip) {
            ok = 0;
        }
        if (!ok) *(volatile int *)&result->status = 2;
        sm.sync_ok = ok;
        sm.sync_sum = total;
        if (tstamp && blockIdx.x == 0 && mark >= 0) tstamp[mark] = global_ns();
    }
    __syncthreads();
    *sum = sm.sync_sum;
    return sm.sync_ok != 0;
}

// ---- learned colouring ----
//
// The policy is a 6 -> 16 -> 1 MLP (ReLU, sigmoid output) evaluated per vertex
// when it is coloured; its weights are a launch parameter, laid out as
// W1[16][6], b1[16], W2[16], b2.  Features: log2(1 + deg), the vertex's role
// in the previous round (0 red or first round, 0.5 blue without a proposal, 1
// blue whose proposal lost), max and mean incident weight, min(round, 32) /
// 32, level / 16.  The blue probability is clamped
// to [1/16, 15/16] and compared with the colouring hash like the select
// barrier: an unmatched edge then splits blue/red in at least 11.7% of the
// rounds, so the maximal types finish well inside the 255-round cap whatever
// the weights (a pair left alone survives 255 rounds with p < 1e-13).
constexpr int kFeat = 6, kHid = 16;
static_assert(kHid * kFeat + kHid + kHid + 1 == MM_POLICY_FLOATS, "policy layout");
constexpr int kTraceCols = 8;  // features, colour (1 blue, 0 red), left the active set in that round
constexpr int kRetireFrom = 3;      // learned colouring: first round in which red vertices retire
constexpr int kRetireMaxDeg = 128;  // learned colouring: longest list a red vertex checks

// Trace: vertex v left the active set in round t (matched, or blue with no
// unmatched neighbour and so retired).
template <bool kPolicy>
__device__ __forceinline__ void trace_left(const Params &p, int t, int v)
{
    if (kPolicy && p.trace && t < p.trace_rounds) p.trace[((size_t)t * p.n + v) * kTraceCols + kFeat + 1] = 1.0f;
}

__device__ __forceinline__ void policy_features(const Params &p, float2 wf, int deg, float role, int t,
                                                float (&x)[kFeat])
{
    x[0] = __log2f(1.0f + (float)deg);
    x[1] = role;
    x[2] = wf.x;
    x[3] = wf.y;
    x[4] = (float)min(t, 32) * (1.0f / 32.0f);
    x[5] = p.level * (1.0f / 16.0f);
}

__device__ __forceinline__ uint32_t policy_barrier(const Params &p, const float (&x)[kFeat])
{
    constexpr int kB1 = kHid * kFeat, kW2 = kB1 + kHid, kB2 = kW2 + kHid;
    float out = p.mlp[kB2];
#pragma unroll
    for (int j = 0; j < kHid; ++j) {
        float a = p.mlp[kB1 + j];
#pragma unroll
        for (int i = 0; i < kFeat; ++i) a = fmaf(p.mlp[j * kFeat + i], x[i], a);
        out = fmaf(p.mlp[kW2 + j], fmaxf(a, 0.0f), out);
    }
    float prob = 1.0f / (1.0f + __expf(-out));
    prob = fminf(fmaxf(prob, 1.0f / 16.0f), 15.0f / 16.0f);
    return (uint32_t)(prob * 4294967296.0f);
}

// Whether colouring round t needs the features: a policy that ignores them
// needs them only for the trace.
__device__ __forceinline__ bool policy_needs_features(const Params &p, int t)
{
    return !p.policy_const || (p.trace && t < p.trace_rounds);
}

// Colour of vertex v for round t: the select barrier, or the policy's.
template <bool kPolicy>
__device__ __forceinline__ bool colour_blue(const Params &p, int v, int base, float role, int t, uint32_t seed)
{
    uint32_t bar = p.barrier;
    if (kPolicy) {
        float x[kFeat];
        if (policy_needs_features(p, t))
            policy_features(p, __ldg(p.wfeat + v), degree_of(__ldg(p.ranges + v)), role, t, x);
        bar = p.policy_const ? p.policy_bar : policy_barrier(p, x);
        const bool blue = colour_of((uint32_t)(v - base), seed, bar) == kBlue;
        if (p.trace && t < p.trace_rounds) {
            float *row = p.trace + ((size_t)t * p.n + v) * kTraceCols;
#pragma unroll
            for (int i = 0; i < kFeat; ++i) row[i] = x[i];
            row[kFeat] = blue ? 1.0f : 0.0f;
            row[kFeat + 1] = 0.0f;
        }
        return blue;
    }
    return colour_of((uint32_t)(v - base), seed, bar) == kBlue;
}

// ---- worklist compaction for the set-up and commit passes ----
//
// A warp handles tiles of 32 W consecutive items (lane l items l, l + 32, ..;
// W = 4 where the block has enough for all its warps, so that four items'
// loads and hashes overlap, else 1) and takes its places in the block's lists with one shared
// atomic a tile and colour, so no warp waits for another: with block-wide
// prefix sums, three block barriers a tile left the set-up of R-MAT 2^22 at
// half the instruction rate its pipes allow.
enum : int { kDrop = -1, kToBlue = 0, kToRed = 1 };

constexpr int kWideItems = 2 * kThreads;  // items from which a block takes tiles of W = 4

template <bool kSolo, int W>
__device__ __forceinline__ void compact_tile(int *count, int *list, int region, const int (&dest)[W],
                                             const int (&item)[W])
{
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    unsigned mb[W], mr[W];
    int nb = 0, nr = 0;
#pragma unroll
    for (int k = 0; k < W; ++k) {
        mb[k] = __ballot_sync(kFull, dest[k] == kToBlue);
        mr[k] = __ballot_sync(kFull, dest[k] == kToRed);
        nb += __popc(mb[k]);
        nr += __popc(mr[k]);
    }
    int at = 0;
    if (lane < 2) at = atomicAdd(count + lane, lane == 0 ? nb : nr);
    int *blue = list + __shfl_sync(kFull, at, 0), *red = list + (region - 1 - __shfl_sync(kFull, at, 1));
#pragma unroll
    for (int k = 0; k < W; ++k) {
        if (dest[k] == kToBlue) Mem<kSolo>::put(blue + __popc(mb[k] & below), item[k]);
        if (dest[k] == kToRed) Mem<kSolo>::put(red - __popc(mr[k] & below), item[k]);
        blue += __popc(mb[k]);
        red -= __popc(mr[k]);
    }
}

// Vertices without neighbours on the symmetric path: no list names them, so
// nothing depends on them but their own match value and the round count.  One
// leaves (match value 2) in the first round in which it is blue, or stays red
// to the cap (match value 1).  The set-up keeps the ones red in round 0 on a
// stack of their warp in shared memory and hashes the top 32 of them for
// their next round each, as long as there are 32, so every lane works (a walk
// per vertex would cost every lane its warp's longest one); the few that are
// left stay in the rounds, as red items, with the same fate.  iso_last: the
// last round in which one was active (the cap's last round if it stays red to
// it, nseeds if the seeds run out first: the reference would draw more, and
// the round count then exceeds nseeds).
__device__ __forceinline__ void resolve_isolated(const Params &p, Smem &sm, int &n, int &iso_last)
{
    const int lane = threadIdx.x & 31;
    int2 *stack = sm.iso.item[threadIdx.x >> 5];
    const int lim = min(p.cap, p.nseeds);
    while (n >= 32) {
        n -= 32;
        const int2 e = stack[n + lane];
        __syncwarp();  // the places above n are free
        const int v = e.x, r = e.y;
        bool stays = false;
        if (r >= lim) {
            // red in every round up to the limit
            p.match[v] = 1;
            if (p.last) p.last[v] = (uint8_t)(p.cap - 1);
            iso_last = max(iso_last, lim == p.cap ? p.cap - 1 : lim);
        } else if (colour_of((uint32_t)(v - base_of(p, v)), sm.iso.seeds[r], p.barrier) == kBlue) {
            p.match[v] = 2;
            if (p.last) p.last[v] = (uint8_t)r;
            iso_last = max(iso_last, r);
        } else {
            stays = true;
        }
        const unsigned m = __ballot_sync(kFull, stays);
        if (stays) stack[n + __popc(m & ((1u << lane) - 1u))] = make_int2(v, r + 1);
        n += __popc(m);
        __syncwarp();
    }
}

// Set-up: colour every vertex with seeds[0] and fill the first worklists.
// best[] starts at 0 and stays 0 for every vertex that is not matched: a red
// vertex that receives a proposal is matched in the same round.  On the
// symmetric path the vertices without neighbours are resolved here, whatever
// their colour (resolve_isolated); the instrumented kernel keeps them in the
// rounds, whose per-round counters count them as the reference does.  A list
// is known to be empty, or longer than its window, from its window's offsets
// (weighted types) or from its range.
template <bool kW, bool kStats, bool kPolicy, bool kSolo, int W>
__device__ __forceinline__ void init_tiles(const Params &p, const Mem<kSolo> &m, Smem &sm, int *list, int &iso_n,
                                           int &iso_last)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t seed = p.seeds[0];
    constexpr int tsize = 32 * W;
    const int ntiles = (p.region + tsize - 1) / tsize;
    // each tile's ranges are loaded while the tile before it is coloured and compacted
    int vv[W];
    int2 rr[W];
    auto fetch = [&](int tile) {
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const int s = tile * tsize + k * 32 + lane;
            vv[k] = s < p.region ? own_vertex(p, s) : -1;
            rr[k] = make_int2(0, 0);
            if (vv[k] >= 0) {
                if (kW) rr[k] = make_int2(__ldg(p.pwin_off + vv[k]), __ldg(p.pwin_off + vv[k] + 1));
                else rr[k] = __ldg(p.ranges + vv[k]);
            }
        }
    };
    fetch(warp);
    for (int tile = warp; tile < ntiles; tile += kWarps) {
        int dest[W], item[W], base_v[W];
        bool none[W], longer[W], blue_k[W];
#pragma unroll
        for (int k = 0; k < W; ++k) {
            item[k] = vv[k];
            base_v[k] = p.vbase && vv[k] >= 0 ? __ldg(p.vbase + vv[k]) : 0;
            none[k] = kW ? ((rr[k].y ^ rr[k].x) & 0x7fffffff) == 0 : degree_of(rr[k]) == 0;
            longer[k] = kW ? rr[k].x < 0 : degree_of(rr[k]) > kWin;
        }
        if (tile + kWarps < ntiles) fetch(tile + kWarps);
        // straight-line hashes, the four items' instructions interleaved
#pragma unroll
        for (int k = 0; k < W; ++k)
            blue_k[k] = kPolicy ? false : colour_of((uint32_t)(item[k] - base_v[k]), seed, p.barrier) == kBlue;
        unsigned long long act = 0, blue_n = 0;
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const int v = item[k];
            dest[k] = kDrop;
            bool queue = false;
            if (v >= 0) {
                const bool blue = kPolicy ? colour_blue<kPolicy>(p, v, base_v[k], 0.0f, 0, seed) : blue_k[k];
                // (every completed round leaves them zero: a cut list's last piece clears them)
                if (p.zero_parts && longer[k]) {
                    p.part_key[v] = 0ull;
                    p.part_cnt[v] = 0;
                }
                ++act;
                blue_n += blue;
                if (!kStats && p.sym && none[k] && (kPolicy || blue)) {
                    // no neighbours: unmatchable as soon as it is blue (learned
                    // colouring: at once, whatever its colour)
                    p.match[v] = 2;
                    if (p.last) p.last[v] = 0;
                    if (!kPolicy) iso_last = max(iso_last, 0);
                    trace_left<kPolicy>(p, 0, v);
                } else if (!kStats && !kPolicy && p.sym && none[k]) {
                    queue = true;
                } else {
                    m.best_[v] = 0ull;
                    dest[k] = blue ? kToBlue : kToRed;
                }
            }
            if (!kStats && !kPolicy && p.sym) {
                const unsigned mq = __ballot_sync(kFull, queue);
                if (queue) sm.iso.item[warp][iso_n + __popc(mq & ((1u << lane) - 1u))] = make_int2(v, 1);
                iso_n += __popc(mq);
            }
            // the colours of 32 consecutive vertices: two words, written whole
            {
                const unsigned bits = dest[k] == kToRed ? (unsigned)kRed << (2 * (lane & 15)) : 0u;
                const unsigned w0 = __reduce_or_sync(kFull, lane < 16 ? bits : 0u);
                const unsigned w1 = __reduce_or_sync(kFull, lane < 16 ? 0u : bits);
                if (v >= 0 && (lane & 15) == 0) m.col_[(unsigned)v >> 4] = lane < 16 ? w0 : w1;
            }
        }
        if (kStats) {
            stat_add(p, 0, MM_ST_ACTIVE, act);
            stat_add(p, 0, MM_ST_BLUE, blue_n);
            stat_add(p, 0, MM_ST_RED, act - blue_n);
        }
        compact_tile<kSolo>(sm.count[0], list, p.region, dest, item);
        if (!kStats && !kPolicy && p.sym) {
            __syncwarp();
            resolve_isolated(p, sm, iso_n, iso_last);
        }
    }
}

template <bool kW, bool kStats, bool kPolicy, bool kSolo>
__device__ __forceinline__ void init_phase(const Params &p, const Mem<kSolo> &m, Smem &sm, int *list)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        sm.count[0][0] = sm.count[0][1] = sm.count[1][0] = sm.count[1][1] = 0;
        sm.wnext = 3 * kThreads;
        sm.stage_n = sm.big_n = sm.flag = sm.zero = 0;
    }
    for (int i = threadIdx.x; i < 256; i += kThreads) sm.iso.seeds[i] = p.seeds[i];
    __syncthreads();
    int iso_n = 0, iso_last = -1;
    if (p.region > kWideItems) init_tiles<kW, kStats, kPolicy, kSolo, kPer>(p, m, sm, list, iso_n, iso_last);
    else init_tiles<kW, kStats, kPolicy, kSolo, 1>(p, m, sm, list, iso_n, iso_last);
    if (!kPolicy && !kStats && p.sym) {
        // the ones left on the stack stay in the rounds: red, as in round 0
        int dest[1] = {kDrop}, item[1] = {-1};
        if (lane < iso_n) {
            item[0] = sm.iso.item[warp][lane].x;
            dest[0] = kToRed;
            m.best_[item[0]] = 0ull;
        }
        compact_tile<kSolo>(sm.count[0], list, p.region, dest, item);
        iso_last = __reduce_max_sync(kFull, iso_last);
        if (lane == 0 && iso_last >= 0) atomicMax(&p.ctl->iso_last, iso_last + 1);
    }
}

// ---- phase A1: preference windows ----
//
// A blue vertex picks the entry the reference's request loop would pick
// (gwRequest: the heaviest red neighbour, strict > from -1, earliest position
// on ties; grRequest: the first red neighbour in list order).  Its candidates
// in that order of preference are its window: for weighted types the
// preparation step sorts each list's best min(deg, 32) entries by (weight,
// earlier position) into pwin, with entries whose weight can never be picked
// (<= -1 or NaN) flagged and last; for random types the window is simply the
// first min(deg, 32) entries of the list.  So the first red candidate in the
// window is the reference's choice, and the scan stops there.  A list that
// fits in its window and has no red candidate is decided too (unmatchable iff
// no entry is unmatched).  A longer list with no red candidate in its window
// falls back to a full scan.

// Learned colouring, graphs with symmetric structure: a red vertex of at most
// kRetireMaxDeg entries whose neighbours are all matched leaves in phase A of
// this round, while the blue vertices scan (the reference waits until it is
// coloured blue and scans).  Colours do not change during phase A, so the
// check is exact, and no vertex reads the retired one's colour: every vertex
// that lists it is its neighbour, hence matched, and matched vertices do not
// scan.  (Without symmetry an unmatched blue vertex could list it, and its
// choice would depend on the timing of the retirement.)  Red items are taken
// from the top of the thread range down, so on small rounds they run on
// threads that have no blue item.  Each list is read 16 entries at a time,
// each batch's colour loads in flight together, stopping after the first batch
// with an unmatched neighbour (most lists fit the first batch).  A limit of
// 128 entries cut R-MAT rounds further than 32 did; 512 cut no more and cost
// time.  A retired vertex's worklist item is marked with its id complemented,
// so the commit phase sees the retirement in the item it loads anyway.
template <bool kPolicy, bool kSolo>
__device__ __forceinline__ void retire_red(const Params &p, const Mem<kSolo> &m, int t, int *list, int cr)
{
    for (int i = kThreads - 1 - (int)threadIdx.x; i < cr; i += kThreads) {
        int *slot = list + (p.region - 1 - i);
        const int v = *slot;
        const int2 r = __ldg(p.ranges + v);
        if (degree_of(r) > kRetireMaxDeg) continue;
        bool gone = true;
        for (Pos j0 = r.x; gone && j0 < (Pos)r.y; j0 += 16) {  // (no reversed ranges on the symmetric path)
            int nb[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) nb[u] = j0 + u < (Pos)r.y ? __ldg(p.nbrs + (j0 + u)) : -1;
#pragma unroll
            for (int u = 0; u < 16; ++u)
                if (nb[u] >= 0 && m.col(nb[u]) != kMatched) gone = false;
        }
        if (gone) {
            p.match[v] = 2;
            if (p.last) p.last[v] = (uint8_t)t;
            *slot = ~v;
            trace_left<kPolicy>(p, t, v);
        }
    }
}

// Blue vertex v (list r) as item idx of the round's shared fallback list, its
// pieces from `first` on.
__device__ __forceinline__ int pieces_of(int deg) { return (deg + kPiece - 1) / kPiece; }
__device__ __forceinline__ void put_shared(const Params &p, int v, const ItemReq &rq, int2 r, int idx, int first, int pieces)
{
    p.staged[idx] = make_int4(v, r.x, r.y, first);
    for (int s = 0; s < pieces; ++s) p.piece_item[first + s] = idx;
    rq.put(kReqShared, 0u);  // it proposes through req[v]
}

// Append blue vertex v to the shared list: one 64-bit atomic hands out the item
// and its pieces.
__device__ __forceinline__ void stage_shared(const Params &p, Smem &sm, int v, const ItemReq &rq, int2 r)
{
    const int pieces = pieces_of(degree_of(r));
    const unsigned long long old = atomicAdd(&p.ctl->staged_pack, (1ull << 32) | (unsigned long long)(unsigned)pieces);
    put_shared(p, v, rq, r, (int)(old >> 32), (int)(unsigned)old, pieces);
    sm.flag = 1;
}

// Group g of a blue vertex's window: four neighbours and their second words
// (weight, position | flag, or position); -1 for entries outside the window.
template <bool kW>
__device__ __forceinline__ void window_group(const Params &p, int g, int lo, int hi, int *nb, int *jv)
{
    if (kW) {
        const int2 *a = p.pwin + 4ll * g;
        asm volatile("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(nb[0]), "=r"(jv[0]), "=r"(nb[1]), "=r"(jv[1]), "=r"(nb[2]), "=r"(jv[2]), "=r"(nb[3]),
                       "=r"(jv[3])
                     : "l"(a));
    } else {
        const int4 x = __ldg(reinterpret_cast<const int4 *>(p.nbrs) + g);
        const int v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            jv[k] = (int)(4u * (unsigned)g + k);
            nb[k] = jv[k] >= lo && jv[k] < hi ? v[k] : -1;
        }
    }
}

// Whether a window entry's neighbour colour c and second word j make it the
// vertex's choice (a red candidate): on the symmetric weighted path j is the
// weight; elsewhere for weighted types the position, bit 31 set for a weight
// that can never be picked; random types: the position.
template <bool kW>
__device__ __forceinline__ bool window_choice(const Params &p, unsigned c, int j)
{
    return c == kRed && (!kW || (p.sym ? __int_as_float(j) > -1.0f : j >= 0));
}

// A window's place: its groups [g, gend), for the random types the entries
// [lo, hi) of the list (groups are aligned, so the first and last may be
// partial), and whether the list is longer.  raw is the pair of window offsets
// (weighted) or the range.
template <bool kW>
__device__ __forceinline__ int2 window_raw(const Params &p, int v)
{
    return kW ? make_int2(__ldg(p.pwin_off + v), __ldg(p.pwin_off + v + 1)) : __ldg(p.ranges + v);
}
template <bool kW>
__device__ __forceinline__ void window_place(int2 raw, int &g, int &gend, int &lo, int &hi, bool &longer)
{
    if (kW) {
        g = raw.x & 0x7fffffff;
        gend = raw.y & 0x7fffffff;
        longer = raw.x < 0;
    } else {
        const int deg = degree_of(raw);
        lo = raw.x;
        hi = lo + win_len(deg);
        g = lo >> 2;
        gend = deg > 0 ? (int)(((Pos)hi + 3u) >> 2) : g;
        longer = deg > kWin;
    }
}

// Full scan of a list by the lanes of one or more warps: entries b + first,
// b + first + step, ... in rows of 32 * kRows per warp; the lanes' best keys.
// Random types stop at the first row with a red entry.
template <bool kW, bool kSolo>
__device__ __forceinline__ unsigned long long scan_rows(const Params &p, const Mem<kSolo> &m, int b, int e, int first, int step)
{
    const int lane = threadIdx.x & 31;
    float bw = -1.0f;
    int bj = 0;
    bool alive = false;
    Pos j0 = (Pos)b + first + lane;
    const int *a = p.nbrs + b + first + lane;
    const float *wa = p.w + b + first + lane;
    for (int left = e - b - first; left > 0; left -= step, a += step, wa += step, j0 += step) {
        int nb[kRows];
        float wv[kRows];
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            const bool in = r * 32 + lane < left;
            nb[r] = in ? __ldg(a + r * 32) : -1;
            wv[r] = kW && in ? __ldg(wa + r * 32) : 0.0f;
        }
        unsigned c[kRows];
#pragma unroll
        for (int r = 0; r < kRows; ++r) c[r] = nb[r] >= 0 ? m.word(nb[r]) : 0xffffffffu;
#pragma unroll
        for (int r = 0; r < kRows; ++r) fold_entry<kW>(colour_bits(c[r], nb[r]), wv[r], (int)(j0 + r * 32), bw, bj, alive);
        if (!kW && __any_sync(kFull, bw > -1.0f)) break;
    }
    return strip_key<kW>(bw, bj, alive);
}

__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long k)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long y = __shfl_xor_sync(kFull, k, o);
        k = y > k ? y : k;
    }
    return k;
}

template <bool kStats>
__device__ __forceinline__ void count_fallback(const Params &p, int t, int deg)
{
    if (kStats) {
        atomicAdd(&p.stats[(size_t)t * MM_STATS_COLS + MM_ST_STAGED_DEG], (unsigned long long)deg);
        atomicAdd(&p.stats[(size_t)t * MM_STATS_COLS + MM_ST_STAGED_ITEMS], 1ull);
    }
}

// The block's fallback lists, collected by its window scan: a warp scans a
// list of up to kWarpList entries, the whole block one of up to kBlockList
// (a round trip of its 16 warps covers 2048 entries); a longer one (a hub,
// which would keep one block busy while the others wait) goes to the shared
// list, at the price of one more grid barrier in that round.  From p.share_from
// lists on all of them go there (share_all; launch_match says when).
constexpr int kWarpList = 512;
constexpr int kBlockList = 32768;

// All the block's fallback lists to the round's shared list, an atomic a warp.
__device__ __forceinline__ void share_all(const Params &p, Smem &sm, int ns, long long rbase)
{
    const int lane = threadIdx.x & 31;
    for (int i0 = (int)threadIdx.x - lane; i0 < ns; i0 += kThreads) {
        const bool in = i0 + lane < ns;
        const int2 it = in ? sm.fb.item[i0 + lane] : make_int2(0, 0);
        const int2 r = in ? __ldg(p.ranges + it.x) : make_int2(0, 0);
        const int pieces = in ? pieces_of(degree_of(r)) : 0;
        int upto = pieces;  // inclusive sum in lane order
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, upto, o);
            if (lane >= o) upto += y;
        }
        const int count = min(32, ns - i0), all = __shfl_sync(kFull, upto, 31);
        unsigned long long old = 0;
        if (lane == 0)
            old = atomicAdd(&p.ctl->staged_pack, ((unsigned long long)count << 32) | (unsigned long long)(unsigned)all);
        old = __shfl_sync(kFull, old, 0);
        if (in) put_shared(p, it.x, ItemReq{p, sm, rbase, it.y}, r, (int)(old >> 32) + lane, (int)(unsigned)old + upto - pieces, pieces);
    }
    if (threadIdx.x == 0) sm.flag = 1;
}

template <bool kW, bool kStats, bool kSolo>
__device__ __noinline__ void scan_fallback(const Params &p, const Mem<kSolo> m, Smem &sm, int t, long long rbase)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ns = min(sm.stage_n, kStageCap);
    if (!kSolo && ns >= p.share_from) {
        share_all(p, sm, ns, rbase);
        return;
    }
    for (int i = warp; i < ns; i += kWarps) {
        const int2 it = sm.fb.item[i];
        const int2 r = __ldg(p.ranges + it.x);
        const int deg = degree_of(r);
        if (deg > kBlockList) {
            if (lane == 0) stage_shared(p, sm, it.x, ItemReq{p, sm, rbase, it.y}, r);
        } else if (deg > kWarpList) {
            if (lane == 0) sm.fb.big[atomicAdd(&sm.big_n, 1)] = (unsigned short)i;
        } else {
            const unsigned long long key = warp_max_u64(scan_rows<kW>(p, m, r.x, r.y, 0, 32 * kRows));
            if (lane == 0) {
                count_fallback<kStats>(p, t, deg);
                propose_key<kW, kStats>(p, m, ItemReq{p, sm, rbase, it.y}, it.x, r.x, deg, key, t);
            }
        }
    }
    __syncthreads();
    const int nbig = sm.big_n;
    for (int i = 0; i < nbig; ++i) {
        const int2 it = sm.fb.item[sm.fb.big[i]];
        const int2 r = __ldg(p.ranges + it.x);
        const int deg = degree_of(r);
        const unsigned long long mine = warp_max_u64(scan_rows<kW>(p, m, r.x, r.y, warp * 32 * kRows, kThreads * kRows));
        if (lane == 0) sm.red_key[warp] = mine;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long key = 0ull;
            for (int w = 0; w < kWarps; ++w) key = sm.red_key[w] > key ? sm.red_key[w] : key;
            count_fallback<kStats>(p, t, deg);
            propose_key<kW, kStats>(p, m, ItemReq{p, sm, rbase, it.y}, it.x, r.x, deg, key, t);
        }
        __syncthreads();  // the keys are reused
    }
}

// Phase A1 over the block's cb blue items.  The first items go to the threads
// in order, the rest to the warps from a counter in shared memory.  A lane
// holds one vertex at a time and reads its window eight entries a step (two
// 32-byte loads, then the eight colours); as soon as a lane's vertex is
// decided it takes the next one, whose window offsets it has prefetched, loads
// the offsets of the one after that, whose id it has prefetched, and prefetches
// another id.  So every lane keeps an independent chain of loads in flight and
// no lane waits for the slowest vertex of its warp or block.
template <bool kW, bool kStats, bool kPolicy, bool kSolo>
__device__ __forceinline__ void scan_window(const Params &p, const Mem<kSolo> &m, Smem &sm, int t, int *list, long long rbase, int cb, int cr)
{
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    bool dry = 3 * kThreads >= cb;  // warp-uniform: the block's items are handed out
    // Items for the lanes in `mask`: one shared atomic per warp.  Returns this
    // lane's item, or -1.
    auto grab = [&](unsigned mask) -> int {
        const int leader = __ffs(mask) - 1;
        int base = 0;
        if (lane == leader) base = atomicAdd(&sm.wnext, __popc(mask));
        base = __shfl_sync(kFull, base, leader);
        dry = base + __popc(mask) >= cb;
        const int k = base + __popc(mask & below);
        return ((mask >> lane) & 1u) && k < cb ? k : -1;
    };
    // the lane's vertex, its next (window offsets loaded) and the one after (id loaded)
    int ci = threadIdx.x, ni = threadIdx.x + kThreads, mi = threadIdx.x + 2 * kThreads;
    ci = ci < cb ? ci : -1;
    ni = ni < cb ? ni : -1;
    mi = mi < cb ? mi : -1;
    int cv = ci >= 0 ? m.item(list + ci) : -1, nv = ni >= 0 ? m.item(list + ni) : -1, mv = mi >= 0 ? m.item(list + mi) : -1;
    int2 nraw = make_int2(0, 0);
    int g = 0, gend = 0, lo = 0, hi = 0;
    bool longer = false;
    if (cv >= 0) window_place<kW>(window_raw<kW>(p, cv), g, gend, lo, hi, longer);
    if (nv >= 0) nraw = window_raw<kW>(p, nv);
    bool has = cv >= 0, alive = false;
    bool narrow = kW && t == 0;
    int seen = 0, last = 0;  // instrumented: entries read, the choice's place in its step
    while (__any_sync(kFull, has)) {
        if (has) {
            // eight entries a step (one dependent round trip for each 8: the scan
            // is bound by the latency of its load chains); the first step of a
            // weighted type's round 0, where most vertices stop at their first or
            // second entry, reads four (a list of a random type starts anywhere in
            // its first group)
            int nb[8], jv[8];
#pragma unroll
            for (int x = 0; x < 8; ++x) {
                nb[x] = -1;
                jv[x] = 0;
            }
            if (g < gend) window_group<kW>(p, g, lo, hi, nb, jv);
            if (!narrow && g + 1 < gend) window_group<kW>(p, g + 1, lo, hi, nb + 4, jv + 4);
            g += narrow ? 1 : 2;
            narrow = false;
            // the colours' words first, all in flight together, then the choice
            // from the last entry down (straight-line code: with a branch an
            // entry the loads went out one after another, RGG 2^20's round 1 20.6
            // us for 17.4)
            unsigned c[8];
#pragma unroll
            for (int x = 0; x < 8; ++x) c[x] = nb[x] >= 0 ? m.word(nb[x]) : 0xffffffffu;
            bool found = false;
            int cj = -1, ct = 0;
#pragma unroll
            for (int x = 7; x >= 0; --x) {
                const unsigned b = colour_bits(c[x], nb[x]);
                alive |= b != kMatched;
                if (window_choice<kW>(p, b, jv[x])) {
                    found = true;
                    cj = jv[x];
                    ct = nb[x];
                    if (kStats) last = x;
                }
            }
            if (kStats) {
#pragma unroll
                for (int x = 0; x < 8; ++x) seen += nb[x] >= 0 && (!found || x <= last);
            }
            if (found || g >= gend) {
                const ItemReq rq{p, sm, rbase, ci};
                if (kStats) {
                    atomicAdd(&p.stats[(size_t)t * MM_STATS_COLS + MM_ST_WINDOW_ENTRIES], (unsigned long long)seen);
                    if (found || !longer) {
                        const int2 r = __ldg(p.ranges + cv);
                        atomicAdd(&p.stats[(size_t)t * MM_STATS_COLS + MM_ST_REQ_ENTRIES],
                                  request_seen<kW>(r.x, degree_of(r), found ? cj : -1));
                        atomicAdd(&p.stats[(size_t)t * MM_STATS_COLS + MM_ST_BLUE_DEG], (unsigned long long)degree_of(r));
                    }
                }
                if (found) {
                    if (kW && p.sym) propose_weight(m, rq, cv, __int_as_float(cj), ct);
                    else propose_to<kW>(p, m, rq, cv, kW ? (p.contiguous ? 0 : __ldg(p.ranges + cv).x) : lo, cj & 0x7fffffff, ct);
                } else if (!longer) {
                    no_proposal(p, rq, cv, alive, t);
                } else {
                    // the whole list is scanned after the windows; only a list that
                    // finds the block's buffer full goes to the shared list at once
                    const int slot = atomicAdd(&sm.stage_n, 1);
                    if (slot < kStageCap) sm.fb.item[slot] = make_int2(cv, ci);
                    else stage_shared(p, sm, cv, rq, __ldg(p.ranges + cv));
                }
                has = false;
            }
        }
        // lanes whose vertex is decided take their prefetched one
        const unsigned need = __ballot_sync(kFull, !has && nv >= 0);
        if (need) {
            const bool take = !has && nv >= 0;
            if (take) {
                cv = nv;
                ci = ni;
                window_place<kW>(nraw, g, gend, lo, hi, longer);
                has = true;
                alive = false;
                narrow = kW && t == 0;
                seen = 0;
                nv = mv;
                ni = mi;
                mv = mi = -1;
                if (nv >= 0) nraw = window_raw<kW>(p, nv);
            }
            if (!dry) {
                const int i = grab(need);
                if (i >= 0) {
                    mi = i;
                    mv = m.item(list + i);
                }
            }
        }
    }
    if (kPolicy && p.sym && t >= kRetireFrom) retire_red<kPolicy>(p, m, t, list, cr);
    if (threadIdx.x < 2) sm.count[(t & 1) ^ 1][threadIdx.x] = 0;  // for the commit phase (read after the barrier)
    __syncthreads();
    if (sm.stage_n > 0) scan_fallback<kW, kStats>(p, m, sm, t, rbase);
}

// ---- phase A2: shared fallback lists ----
//
// A warp scans a piece of kPiece entries.  A list of several pieces
// max-combines them in part_key; the piece that arrives last proposes.
template <bool kW, bool kStats, bool kSolo>
__device__ __noinline__ void scan_shared(const Params &p, const Mem<kSolo> m, int t)
{
    const unsigned long long pack = __ldcg(&p.ctl->staged_pack);
    const int npieces = (int)(pack & 0xffffffffull);
    const int lane = threadIdx.x & 31;
    for (int s = (int)(blockIdx.x * kWarps + (threadIdx.x >> 5)); s < npieces; s += (int)(gridDim.x * kWarps)) {
        const int4 it = __ldcg(p.staged + __ldcg(p.piece_item + s));
        const int deg = degree_of(it), pieces = pieces_of(deg);
        const int b = it.y + (s - it.w) * kPiece, e = b + min(kPiece, it.z - b), v = it.x;
        const unsigned long long key = warp_max_u64(scan_rows<kW>(p, m, b, e, 0, 32 * kRows));
        if (lane != 0) continue;
        count_fallback<kStats>(p, t, e - b);
        if (pieces == 1) {
            propose_key<kW, kStats>(p, m, VertexReq{p, v}, v, it.y, deg, key, t);
            continue;
        }
        if (key) atomicMax(&p.part_key[v], key);
        // acq_rel: this piece's max is visible before its arrival counts, and the
        // last arrival sees every other piece's max
        int done;
        asm volatile("atom.add.acq_rel.gpu.s32 %0, [%1], 1;" : "=r"(done) : "l"(p.part_cnt + v) : "memory");
        if (done == pieces - 1) {
            const unsigned long long all = atomicExch(&p.part_key[v], 0ull);
            atomicExch(&p.part_cnt[v], 0);
            propose_key<kW, kStats>(p, m, VertexReq{p, v}, v, it.y, deg, all, t);
        }
    }
}

// Phase B: commit proposals, recolour survivors with the next seed, compact
// the block's lists of round t+1.  Colours are
// written only where they change.
template <bool kW, bool kStats, bool kPolicy, bool kSolo, int W>
__device__ __forceinline__ void commit_tiles(const Params &p, const Mem<kSolo> &m, Smem &sm, int t, bool has_next, const int *list, int *next,
                                             long long rbase, int cb, int cr)
{
    const uint32_t next_seed = has_next ? p.seeds[t + 1] : 0u;
    const int total = cb + cr;
    constexpr int tsize = 32 * W;
    for (int base = (int)(threadIdx.x >> 5) * tsize; base < total; base += kWarps * tsize) {
        // The loads of the tile's items go out together, pass by pass: item and
        // request, then the best proposal (blue: its target's, red: its own).
        int vv[W], tg[W], base_v[W];
        uint32_t low[W];
        bool blue[W], gone[W];
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const int i = base + k * 32 + (int)(threadIdx.x & 31);
            const bool in = i < total;
            blue[k] = in && i < cb;
            vv[k] = in ? m.item(list + (i < cb ? i : p.region - 1 - (i - cb))) : -1;
            tg[k] = kReqNone;
            low[k] = 0u;
            if (blue[k]) {
                tg[k] = i < kPropCap ? sm.req.target[i] : __ldcs(p.prop + rbase + i);
                if (!p.sym) low[k] = __ldcs(p.prop_key + rbase + i);
            }
            // learned colouring: a red item retired in phase A carries its id complemented
            gone[k] = kPolicy && in && vv[k] < 0;
            if (gone[k]) vv[k] = ~vv[k];
        }
        unsigned long long key[W];
#pragma unroll
        for (int k = 0; k < W; ++k) {
            if (blue[k] && tg[k] == kReqShared) {  // a shared fallback list's request is in req
                const int2 q = __ldcg(p.req + vv[k]);
                tg[k] = q.x;
                low[k] = (uint32_t)q.y;
            }
            if (p.sym) low[k] = ~(uint32_t)vv[k];
            // blue: a request whose key is not 0
            const int at = blue[k] ? (low[k] != 0u ? tg[k] : -1) : vv[k];
            key[k] = at >= 0 ? m.best(at) : 0ull;
            base_v[k] = p.vbase && vv[k] >= 0 ? __ldg(p.vbase + vv[k]) : 0;
        }
        int partner[W];
        bool nb[W];
#pragma unroll
        for (int k = 0; k < W; ++k) {
            partner[k] = -1;
            if (key[k]) {
                const uint32_t kl = (uint32_t)key[k];
                // the low half of a red vertex's key names the proposer: its id on
                // the symmetric path, else the position of the red's entry for it
                if (blue[k]) partner[k] = kl == low[k] ? tg[k] : -1;
                else partner[k] = p.sym ? (int)~kl : __ldg(p.nbrs + (int)~kl);
            }
            // the next colour, straight-line for all items (the matched ones' is not used)
            nb[k] = kPolicy ? false : colour_of((uint32_t)(vv[k] - base_v[k]), next_seed, p.barrier) == kBlue;
        }
        int dest[W];
        unsigned long long matched = 0, seen = 0, rdeg = 0, act = 0, nblue = 0;
#pragma unroll
        for (int k = 0; k < W; ++k) {
            dest[k] = kDrop;
            const int v = vv[k];
            if (v < 0) continue;
            if (kStats && !blue[k]) {
                const int2 r = __ldg(p.ranges + v);
                const int deg = degree_of(r);
                rdeg += deg;
                // random mode: grRespond stops at its first proposer, whose position
                // is the key's low half (symmetric path: found in the sorted list)
                int at = -1;
                if (!kW && key[k]) {
                    at = (int)~(uint32_t)key[k];
                    if (p.sym) {
                        int lo = r.x, hi = r.y;
                        while (lo < hi) {
                            const int mid = (int)(((long long)lo + hi) >> 1);
                            if (__ldg(p.nbrs + mid) < at) lo = mid + 1;
                            else hi = mid;
                        }
                        at = lo;
                    }
                }
                seen += at >= 0 ? (unsigned long long)(at - r.x + 1) : (unsigned long long)deg;
            }
            unsigned delta = 0u;
            if (partner[k] >= 0) {
                trace_left<kPolicy>(p, t, v);
                p.match[v] = 4 + min(v, partner[k]) - base_v[k];
                if (p.last) p.last[v] = (uint8_t)t;
                delta = blue[k] ? kMatched ^ kBlue : kMatched ^ kRed;
                ++matched;
            } else if ((blue[k] && tg[k] == kReqDead) || gone[k]) {
                // unmatchable (marked in phase A; learned colouring: red ones too)
                trace_left<kPolicy>(p, t, v);
            } else if (!has_next) {
                dest[k] = blue[k] ? kToBlue : kToRed;
            } else {
                if (kPolicy) {
                    const float role = blue[k] ? (tg[k] >= 0 && low[k] != 0u ? 1.0f : 0.5f) : 0.0f;
                    nb[k] = colour_blue<kPolicy>(p, v, base_v[k], role, t + 1, next_seed);
                }
                ++act;
                nblue += nb[k];
                delta = nb[k] != blue[k] ? kBlue ^ kRed : 0u;
                dest[k] = nb[k] ? kToBlue : kToRed;
            }
            if (delta) m.flip(v, delta);
        }
        if (kStats) {
            stat_add(p, t, MM_ST_MATCHED, matched);
            stat_add(p, t, MM_ST_RESP_ENTRIES, seen);
            stat_add(p, t, MM_ST_RED_DEG, rdeg);
            if (has_next) {
                stat_add(p, t + 1, MM_ST_ACTIVE, act);
                stat_add(p, t + 1, MM_ST_BLUE, nblue);
                stat_add(p, t + 1, MM_ST_RED, act - nblue);
            }
        }
        compact_tile<kSolo>(sm.count[(t & 1) ^ 1], next, p.region, dest, vv);
    }
}

template <bool kW, bool kStats, bool kPolicy, bool kSolo>
__device__ __forceinline__ void commit_phase(const Params &p, const Mem<kSolo> &m, Smem &sm, int t, bool has_next,
                                             const int *list, int *next, long long rbase, int cb, int cr)
{
    if (cb + cr > kWideItems) commit_tiles<kW, kStats, kPolicy, kSolo, kPer>(p, m, sm, t, has_next, list, next, rbase, cb, cr);
    else commit_tiles<kW, kStats, kPolicy, kSolo, 1>(p, m, sm, t, has_next, list, next, rbase, cb, cr);
    if (threadIdx.x == 0) {  // for the next window scan (read after the barrier)
        sm.wnext = 3 * kThreads;
        sm.stage_n = sm.big_n = sm.flag = 0;
    }
}

// ---- finish phase ----
//
// After the first rounds the vertices that can still be matched form a sparse
// subgraph: on R-MAT 2^23 at round 5, 334 k active vertices share 40 k entries
// that point at another active vertex, and its connected components have at
// most 7 members (grids, random geometric and Erdos-Renyi graphs reach the same
// state by round 3).  A vertex's future depends only on the colours and choices
// of the active vertices it can reach: matched neighbours never change, and
// where every entry has a reverse entry no active vertex has an unmatchable
// neighbour (a vertex became unmatchable because every neighbour was matched;
// the colours would not tell one).  So each component
// can play all its remaining rounds on its own, with the same seeds, and the
// grid needs no further barrier.
//
// The phase runs at the start of round t in two passes over the round's
// worklist items, each ended by a grid barrier:
//   scan   every item scans its own list: no active neighbour (a singleton),
//          an active neighbour with a smaller id (a member: another vertex
//          speaks for its component), or else a root candidate.  It records
//          its first four active neighbours with their preference keys.  A
//          singleton walks its own hash sequence at once: it leaves (match
//          value 2) in the first round it is blue, or keeps red to the cap.
//   roots  each root candidate's lane follows the records breadth first to
//          its component and, if no member has a smaller id, plays it: per
//          round colour, request (the best red neighbour by the same keys as
//          the scans), respond (the largest proposal key), commit.  A
//          component that a lane cannot hold (records incomplete, more than
//          kFinTMembers members) is searched and played by the warp, lane l
//          holding member l (up to kFinMembers members, kFinEntries entries).
// A larger component or a list longer than kFinMaxDeg calls the attempt off,
// and round t runs as
// usual; values already written are the ones the rounds write again.  The
// instrumented kernel checks first and resolves in a third pass, so that its
// counters never include a called-off attempt.
// Every vertex's match value is then final, and the matching executed
// max(last active round) + 2 rounds, the reference's closing round included
// (at most the cap).
constexpr int kFinShort = 32;      // lists a thread scans on its own; longer ones its warp scans
constexpr int kFinMaxDeg = 2048;   // longest list the finish phase accepts
// Default: first attempt once the active set is at most 1/kFinDiv of round 0's.
// A round costs 7-8 us once the set is small; an attempt a round too early
// meets components that lanes cannot hold (RGG 2^20 at 1/13: 188 us a call,
// at 1/27: 176), a round too late costs that round.  Sparse graphs fall apart
// sooner (512 x 512 grid at 1/14: 74 us, at 1/28: 78).
constexpr int kFinDiv = 24;
constexpr int kFinDivSparse = 12;
constexpr int kFinSparse = 6;      // entries a vertex on average, at most
enum : int { kFinSingle = 1, kFinMember = 2, kFinRootCand = 3 };
enum : int { kFinNotRoot = 0, kFinRoot = 1, kFinTooBig = 2 };

// Item i of the block's lists (cb blue, then the red ones).
template <bool kSolo>
__device__ __forceinline__ int item_at(const Params &p, const int *list, int cb, int i)
{
    return Mem<kSolo>::item(list + (i < cb ? i : p.region - 1 - (i - cb)));
}

// Preference key of an entry of weight w, as the finish phase compares them.
// at: its position in the arrays; on the symmetric path the neighbour's id, as
// a list is strictly increasing there, so the smaller id is the earlier
// position.  1: a neighbour that is never chosen.
template <bool kW>
__device__ __forceinline__ unsigned long long fin_key(int at, float w)
{
    return cand_key<kW>(at, w);
}

// Own-list scan of vertex v, entries [b, e): active neighbours (blue or red),
// whether one has a smaller id, and the positions and ids of the first kFinRec
// of them.
constexpr int kFinRec = 4;  // active neighbours a record holds
__device__ __forceinline__ void fin_scan_thread(const Params &p, int v, int b, int e, int &nint, bool &lower,
                                                int (&jr)[kFinRec], int (&ur)[kFinRec])
{
    // (with an unsigned position for the count the kernel spilled: R-MAT 2^23 821 us for 793)
    for (int left = e - b; left > 0; left -= 8) {
        int u[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) u[k] = k < left ? __ldg(p.nbrs + (e - left + k)) : -1;
        unsigned c[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) c[k] = u[k] >= 0 ? colour_bits(p.col[(unsigned)u[k] >> 4], u[k]) : (unsigned)kMatched;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (c[k] <= kRed) {
#pragma unroll
                for (int q = 0; q < kFinRec; ++q) {
                    if (nint == q) {
                        jr[q] = e - left + k;
                        ur[q] = u[k];
                    }
                }
                ++nint;
                lower |= u[k] < v;
            }
        }
    }
}

// The same scan by a whole warp, rows of 32 entries, for a list longer than
// kFinShort; every lane gets the results (the first kFinRec active
// neighbours in list order too).
__device__ __forceinline__ void fin_scan_warp(const Params &p, int v, int b, int e, int &nint, bool &lower,
                                              int (&jr)[kFinRec], int (&ur)[kFinRec])
{
    const int lane = threadIdx.x & 31;
    int cnt = 0;
    bool lo = false;
    for (Pos r0 = b; r0 < (Pos)e; r0 += 32 * 4) {
        int u[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) u[k] = r0 + 32 * k + lane < (Pos)e ? __ldg(p.nbrs + (r0 + 32 * k + lane)) : -1;
        unsigned c[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) c[k] = u[k] >= 0 ? colour_bits(p.col[(unsigned)u[k] >> 4], u[k]) : (unsigned)kMatched;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const bool in = c[k] <= kRed;
            lo |= in && u[k] < v;
            unsigned m = __ballot_sync(kFull, in);
            while (m && cnt < kFinRec) {
                const int sb = __ffs(m) - 1;
                m &= m - 1;
                const int us = __shfl_sync(kFull, u[k], sb);
#pragma unroll
                for (int q = 0; q < kFinRec; ++q) {
                    if (cnt == q) {
                        jr[q] = (int)(r0 + 32 * k + sb);
                        ur[q] = us;
                    }
                }
                ++cnt;
            }
            cnt += __popc(m);
        }
    }
    nint = cnt;
    lower = __any_sync(kFull, lo);
}

// Component search for root candidate v by its warp.  Members are numbered in
// discovery order (member 0 is v; lane l's `mem` holds member l); each
// member's entries that point at a member are stored in order, from
// fw.eoff[member].  Returns kFinNotRoot as soon as a member has a smaller id
// than v, kFinTooBig if the component does not fit, else kFinRoot with *k
// members.
template <bool kW>
__device__ __forceinline__ int fin_search(const Params &p, FinWarp &fw, int v, int *mem_out, int *k_out,
                                          unsigned long long *scanned)
{
    const int lane = threadIdx.x & 31;
    int mem = lane == 0 ? v : -1;
    int k = 1, ne = 0;
    unsigned long long seen = 0;
    for (int f = 0; f < k; ++f) {
        const int x = __shfl_sync(kFull, mem, f);
        const int2 r = __ldg(p.ranges + x);
        const int b = r.x, e = r.y > r.x ? r.y : r.x;
        if (e - b > kFinMaxDeg) return kFinTooBig;
        if (lane == 0) {
            fw.eoff[f] = ne;
        }
        seen += (unsigned long long)(e - b);
        for (Pos j0 = b; j0 < (Pos)e; j0 += 32) {
            const Pos j = j0 + lane;
            int u = -1;
            float wj = 0.0f;
            unsigned c = kMatched;
            if (j < (Pos)e) {
                u = __ldg(p.nbrs + j);
                if (kW) wj = __ldg(p.w + j);  // with the id: no dependent load once the colour is known
                c = colour_bits(p.col[(unsigned)u >> 4], u);
            }
            const bool in = c <= kRed;
            if (__any_sync(kFull, in && u < v)) return kFinNotRoot;
            unsigned m = __ballot_sync(kFull, in);
            unsigned long long pref = 0;
            if (in) pref = fin_key<kW>(p.sym ? u : (int)j, wj);
            while (m) {
                const int s = __ffs(m) - 1;
                m &= m - 1;
                const int us = __shfl_sync(kFull, u, s);
                const unsigned hit = __ballot_sync(kFull, lane < k && mem == us);
                int slot;
                if (hit) {
                    slot = __ffs(hit) - 1;
                } else {
                    if (k == kFinMembers) return kFinTooBig;
                    slot = k;
                    if (lane == k) mem = us;
                    ++k;
                }
                if (ne == kFinEntries) return kFinTooBig;
                if (lane == s) {
                    fw.pref[ne] = pref;
                    fw.tgt[ne] = (uint8_t)slot;
                }
                ++ne;
            }
        }
    }
    if (lane == 0) fw.eoff[k] = ne;
    __syncwarp();
    *mem_out = mem;
    *k_out = k;
    if (scanned) *scanned = seen;
    return kFinRoot;
}

// Adjacency entries the reference's respond loop inspects for red vertex v
// (entries [b, b + deg)) whose best proposal key is kb: in random mode it
// stops at its first proposer in list order: kb's low half complemented is its
// position, or on the symmetric path its id, found in the sorted list.
template <bool kW>
__device__ __forceinline__ unsigned long long respond_seen(const Params &p, int b, int deg, unsigned long long kb)
{
    if (kW || !kb) return (unsigned long long)deg;
    const int first = (int)~(uint32_t)kb;
    if (!p.sym) return (unsigned long long)(first - b + 1);  // a position
    int lo = b, hi = b + deg;
    while (lo < hi) {
        const int mid = (int)(((long long)lo + hi) >> 1);
        if (__ldg(p.nbrs + mid) < first) lo = mid + 1;
        else hi = mid;
    }
    return (unsigned long long)(lo - b + 1);
}

// Play a component found by fin_search (k members, lane l = member l) from
// round t0 until none of its members can be matched or the cap is reached;
// writes every member's match value (and batch round marks).  Returns, in
// every lane, the last round in which a member was active.
template <bool kW, bool kStats>
__device__ __forceinline__ int fin_play(const Params &p, FinWarp &fw, int t0, int mem, int k)
{
    const int lane = threadIdx.x & 31;
    const bool own = lane < k;
    const int g = own ? mem : 0;
    const int base = own ? base_of(p, g) : 0;
    const uint32_t hid = (uint32_t)(g - base);
    const uint32_t bar = p.fin_retire ? p.policy_bar : p.barrier;
    int eb = 0, ee = 0, deg = 0, beg = 0;
    if (own) {
        eb = fw.eoff[lane];
        ee = fw.eoff[lane + 1];
        fw.best[lane] = 0ull;
        if (kStats) {
            const int2 r = __ldg(p.ranges + g);
            deg = degree_of(r);
            beg = r.x;
        }
    }
    // learned colouring: whether a red member may retire (its list is short enough)
    const bool may_retire = p.fin_retire && own && degree_of(__ldg(p.ranges + g)) <= kRetireMaxDeg;
    bool act = own, blue = false;
    int val = 0, lastr = -1;
    __syncwarp();
    for (int t = t0; t < p.cap && __any_sync(kFull, act); ++t) {
        if (act) {
            blue = colour_of(hid, p.seeds[t], bar) == kBlue;
            lastr = t;
        }
        if (own) fw.st[lane] = act ? (blue ? kBlue : kRed) : (val == 2 ? kDead : kMatched);
        __syncwarp();
        // learned colouring: from round kRetireFrom a red member whose neighbours
        // are all matched leaves at once (the round kernel's retire_red; its
        // neighbours outside the component are matched)
        bool retired = false;
        if (may_retire && act && !blue && t >= kRetireFrom) {
            bool alive = false;
            for (int e = eb; e < ee; ++e) alive |= fw.st[fw.tgt[e]] != kMatched;
            if (!alive) {
                val = 2;
                retired = true;
            }
        }
        // request: the best red neighbour among the members (matched ones
        // outside the component neither attract nor keep a vertex alive)
        unsigned long long best = 0ull;
        int choice = 0;
        if (act && blue) {
            for (int e = eb; e < ee; ++e) {
                const int tg = fw.tgt[e];
                const uint8_t c = fw.st[tg];
                const unsigned long long key = c == kRed ? fw.pref[e] : (c == kMatched ? 0ull : 1ull);
                if (key > best) {
                    best = key;
                    choice = tg;
                }
            }
        }
        unsigned long long crk = 0ull;
        if (act && blue && best >= 2) {
            // the proposal's key: on the symmetric path the target's entry for this
            // vertex has the same weight; else the reverse key of the chosen entry
            // (0: the target never picks it)
            if (p.sym)
                crk = kW ? (((best >> 32) << 32) | (unsigned long long)(uint32_t)~(uint32_t)g)
                         : (unsigned long long)(uint32_t)~(uint32_t)g;
            else
                crk = __ldg(p.revkey + (int)~(uint32_t)best);
            if (crk) atomicMax(&fw.best[choice], crk);
        }
        __syncwarp();
        const int gp = __shfl_sync(kFull, g, choice);
        bool matched = false, dead = false;
        unsigned long long kb = 0ull;
        if (act) {
            if (blue) {
                if (crk && (uint32_t)fw.best[choice] == (uint32_t)crk) {
                    val = 4 + min(g, gp) - base;
                    matched = true;
                } else if (best == 0) {
                    val = 2;
                    dead = true;
                }
            } else {
                kb = fw.best[lane];
                if (kb) {
                    const int from = (int)~(uint32_t)kb;
                    val = 4 + min(g, p.sym ? from : __ldg(p.nbrs + from)) - base;
                    matched = true;
                }
            }
        }
        if (kStats) {
            const bool b = act && blue, r = act && !blue;
            if (t > t0) {  // round t0's colouring was counted by the commit that made it
                stat_add(p, t, MM_ST_ACTIVE, act ? 1ull : 0ull);
                stat_add(p, t, MM_ST_BLUE, b ? 1ull : 0ull);
                stat_add(p, t, MM_ST_RED, r ? 1ull : 0ull);
            }
            stat_add(p, t, MM_ST_BLUE_DEG, b ? (unsigned long long)deg : 0ull);
            stat_add(p, t, MM_ST_RED_DEG, r ? (unsigned long long)deg : 0ull);
            stat_add(p, t, MM_ST_REQ_ENTRIES,
                     b ? (kW || best < 2 ? (unsigned long long)deg : respond_seen<kW>(p, beg, deg, best)) : 0ull);
            stat_add(p, t, MM_ST_RESP_ENTRIES, r ? respond_seen<kW>(p, beg, deg, kb) : 0ull);
            stat_add(p, t, MM_ST_MATCHED, matched ? 1ull : 0ull);
        }
        __syncwarp();
        if (own) fw.best[lane] = 0ull;
        if (matched || dead || retired) act = false;
    }
    if (own) {
        // members still unmatched at the cap keep their last colour
        p.match[g] = act ? (blue ? 0 : 1) : val;
        if (p.last) p.last[g] = (uint8_t)lastr;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) lastr = max(lastr, __shfl_xor_sync(kFull, lastr, o));
    return lastr;
}

// Lane-level components.  Most components of the finish round are pairs and
// short paths.  A warp that searched its lanes' roots one after another, each
// rescanning its members' lists, made every warp a chain of dependent loads
// (on RGG 2^20 at round 3, 9 root candidates a tile and 52 us a warp).  So each
// lane searches its own root's component through the records and plays it in
// per-thread storage.
constexpr int kFinTMembers = 16;
constexpr int kFinTEntries = 32;
enum : int { kFinOverflow = 3 };

struct FinComp {
    unsigned long long pref[kFinTEntries];
    int mem[kFinTMembers];
    uint8_t tgt[kFinTEntries];
    uint8_t eoff[kFinTMembers + 1];
    int k;
};

// The finish phase's record of an item: rec_stride int4, the i-th record's from
// rec[rec_stride * i], i counted from the block's own part of the record
// array: {meta, v, id 0, id 1}, {id 2, id 3, weight 0, weight 1}, {weight 2,
// weight 3, 0, 0}, the ids and weight orders (0: never chosen) of its first
// kFinRec entries that point at an active vertex; off the symmetric path also
// {position 0, .., position 3}.  meta = class | count << 8, count = its active
// neighbours, kFinRec + 1 if more than a record holds.
__device__ __forceinline__ int fin_meta_class(int meta) { return meta & 0xff; }
__device__ __forceinline__ int fin_meta_count(int meta) { return (meta >> 8) & 0xff; }

// As fin_search, by one thread for root candidate v (record i), following the
// records instead of the lists: each member costs two loads from L2 (its
// record's index, its record).  kFinOverflow when a member's record is
// incomplete or the component does not fit FinComp.
template <bool kW>
__device__ __forceinline__ int fin_search_thread(const Params &p, int v, int i, FinComp &cp)
{
    int ix[kFinTMembers];
    int k = 1, ne = 0;
    cp.mem[0] = v;
    ix[0] = i;
    for (int f = 0; f < k; ++f) {
        const int4 *rec = p.rec + (long long)p.rec_stride * ix[f];
        const int4 r0 = __ldcg(rec), r1 = __ldcg(rec + 1), r2 = __ldcg(rec + 2);
        const int4 r3 = p.sym ? make_int4(r0.z, r0.w, r1.x, r1.y) : __ldcg(rec + 3);
        const int cnt = fin_meta_count(r0.x);
        if (cnt > kFinRec) return kFinOverflow;
        cp.eoff[f] = (uint8_t)ne;
        const int uu[kFinRec] = {r0.z, r0.w, r1.x, r1.y};
        const int ww[kFinRec] = {r1.z, r1.w, r2.x, r2.y};
        const int aa[kFinRec] = {r3.x, r3.y, r3.z, r3.w};
#pragma unroll
        for (int q = 0; q < kFinRec; ++q) {
            if (q >= cnt) break;
            const int u = uu[q];
            if (u < v) return kFinNotRoot;
            int slot = -1;
            for (int m = 0; m < k; ++m)
                if (cp.mem[m] == u) slot = m;
            if (slot < 0) {
                if (k == kFinTMembers) return kFinOverflow;
                slot = k;
                cp.mem[k] = u;
                ix[k] = __ldcg(p.req + u).x;  // its record (written by the scan pass)
                ++k;
            }
            if (ne == kFinTEntries) return kFinOverflow;
            cp.pref[ne] = !kW ? (unsigned long long)(uint32_t)~aa[q]
                              : (ww[q] ? (((unsigned long long)(uint32_t)ww[q] << 32) | (uint32_t)~aa[q]) : 1ull);
            cp.tgt[ne] = (uint8_t)slot;
            ++ne;
        }
    }
    cp.eoff[k] = (uint8_t)ne;
    cp.k = k;
    return kFinRoot;
}

// Singletons of a tile (mine): each leaves in the first round from t on in
// which it is blue (blue0: its colour in round t), or keeps red to the cap.
template <bool kStats>
__device__ __forceinline__ void fin_singles(const Params &p, int t, bool mine, int v, int deg, bool blue0, int &last_all)
{
    const uint32_t bar = p.fin_retire ? p.policy_bar : p.barrier;
    const uint32_t hid = mine ? (uint32_t)(v - base_of(p, v)) : 0u;
    // learned colouring: a short list retires as soon as it is red from round
    // kRetireFrom (a singleton's neighbours are all matched)
    const bool may_retire = p.fin_retire && deg <= kRetireMaxDeg;
    bool act = mine, blue = blue0;
    int lastr = -1;
    for (int r = t; r < p.cap && __any_sync(kFull, act); ++r) {
        if (act) {
            if (r > t) blue = colour_of(hid, p.seeds[r], bar) == kBlue;
            lastr = r;
        }
        if (kStats) {
            const bool b = act && blue, rd = act && !blue;
            if (r > t) {  // round t's colouring was counted by the commit that made it
                stat_add(p, r, MM_ST_ACTIVE, act ? 1ull : 0ull);
                stat_add(p, r, MM_ST_BLUE, b ? 1ull : 0ull);
                stat_add(p, r, MM_ST_RED, rd ? 1ull : 0ull);
            }
            stat_add(p, r, MM_ST_BLUE_DEG, b ? (unsigned long long)deg : 0ull);
            stat_add(p, r, MM_ST_RED_DEG, rd ? (unsigned long long)deg : 0ull);
            stat_add(p, r, MM_ST_REQ_ENTRIES, b ? (unsigned long long)deg : 0ull);
            stat_add(p, r, MM_ST_RESP_ENTRIES, rd ? (unsigned long long)deg : 0ull);
        }
        if (act && (blue || (may_retire && r >= kRetireFrom))) act = false;
    }
    if (mine) {
        // still red at the cap: it keeps that colour
        p.match[v] = act ? 1 : 2;
        if (p.last) p.last[v] = (uint8_t)lastr;
        last_all = max(last_all, lastr);
    }
}

// The part of the block's `cnt` items that this warp handles in the finish
// passes: equal shares, so that a small set still spreads over all warps.
__device__ __forceinline__ void fin_share(int cnt, int &lo, int &hi)
{
    const int warp = threadIdx.x >> 5, share = (cnt + kWarps - 1) / kWarps;
    lo = min(cnt, warp * share);
    hi = min(cnt, lo + share);
}

// Finish pass 1 over the block's items of round t: scan each item's own list
// (a thread each, its warp for lists longer than kFinShort), classify it,
// record its first active neighbours (and in req[v].x the record's index),
// and, with kSingles, resolve the singletons at once.  Returns whether the
// attempt has to be called off: a list longer than kFinMaxDeg, or more items
// than the block has records for.
template <bool kW, bool kStats, bool kSingles>
__device__ __forceinline__ bool finish_scan(const Params &p, int t, const int *list, int cb, int cr)
{
    const int lane = threadIdx.x & 31;
    const int cnt_all = cb + cr;
    if (cnt_all > p.rec_region) return true;
    bool abort = false;
    int last_all = -1, lo_i, hi_i;
    fin_share(cnt_all, lo_i, hi_i);
    for (int base = lo_i; base < hi_i; base += 32) {
        const int i = base + lane;
        const int v = i < hi_i ? item_at<false>(p, list, cb, i) : -1;
        const int2 r = v >= 0 ? __ldg(p.ranges + v) : make_int2(0, 0);
        const int deg = degree_of(r);
        int nint = 0, jr[kFinRec] = {0, 0, 0, 0}, ur[kFinRec] = {0, 0, 0, 0};
        bool lower = false, bad = false;
        if (v >= 0 && deg <= kFinShort) fin_scan_thread(p, v, r.x, r.x + deg, nint, lower, jr, ur);
        unsigned longs = __ballot_sync(kFull, v >= 0 && deg > kFinShort);
        while (longs) {
            const int s = __ffs(longs) - 1;
            longs &= longs - 1;
            const int vs = __shfl_sync(kFull, v, s), bs = __shfl_sync(kFull, r.x, s);
            const int ds = __shfl_sync(kFull, deg, s);
            if (ds > kFinMaxDeg) {
                if (lane == s) bad = true;
                continue;
            }
            int n2, j2[kFinRec], u2[kFinRec];
            bool l2;
            fin_scan_warp(p, vs, bs, bs + ds, n2, l2, j2, u2);
            if (lane == s) {
                nint = n2;
                lower = l2;
#pragma unroll
                for (int q = 0; q < kFinRec; ++q) {
                    jr[q] = j2[q];
                    ur[q] = u2[q];
                }
            }
        }
        const int c = v < 0 ? 0 : (nint == 0 ? kFinSingle : (lower ? kFinMember : kFinRootCand));
        abort |= bad;
        if (v >= 0) {
            const int cnt = min(nint, kFinRec + 1);
            const int at = blockIdx.x * p.rec_region + i;
            int4 *rec = p.rec + (long long)p.rec_stride * at;
            rec[0] = make_int4(c | (cnt << 8), v, ur[0], ur[1]);
            if (nint > 0) {
                p.req[v].x = at;
                if (cnt <= kFinRec) {
                    int o[kFinRec];
#pragma unroll
                    for (int q = 0; q < kFinRec; ++q) {
                        o[q] = 0;
                        if (kW && q < cnt) {
                            const float x = __ldg(p.w + jr[q]);
                            if (x > -1.0f) o[q] = (int)weight_order(x);
                        }
                    }
                    rec[1] = make_int4(ur[2], ur[3], o[0], o[1]);
                    rec[2] = make_int4(o[2], o[3], 0, 0);
                    if (!p.sym) rec[3] = make_int4(jr[0], jr[1], jr[2], jr[3]);
                }
            }
        }
        if (kStats) {
            stat_add(p, t, MM_ST_FINISH_ITEMS, v >= 0 ? 1ull : 0ull);
            stat_add(p, t, MM_ST_FINISH_ENTRIES, (unsigned long long)deg);
        }
        if (__any_sync(kFull, abort)) break;
        if (kSingles) fin_singles<kStats>(p, t, c == kFinSingle, v, deg, i < cb, last_all);
    }
    if (kSingles) {
        last_all = __reduce_max_sync(kFull, last_all);
        if (lane == 0 && last_all >= 0) atomicMax(&p.ctl->fin_last, last_all);
    }
    return abort;
}

// Finish pass 2 over the block's items: each root candidate's lane searches its
// component through the records and, with kPlay, plays it; a component that
// a lane cannot hold goes to the warp (list scans, up to kFinMembers members),
// and one larger than that calls the attempt off.  With kSingles (the
// instrumented kernel's last pass) the singletons are resolved here too.
template <bool kW, bool kStats, bool kPlay, bool kSingles>
__device__ __forceinline__ bool finish_roots(const Params &p, Smem &sm, int t, int cb, int cr)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    FinWarp &fw = sm.fin[warp];
    bool abort = false;
    int last_all = -1, lo_i, hi_i;
    fin_share(cb + cr, lo_i, hi_i);
    for (int base = lo_i; base < hi_i; base += 32) {
        const int i = base + lane;
        const int at = blockIdx.x * p.rec_region + i;
        const int4 r0 = i < hi_i ? __ldcg(p.rec + (long long)p.rec_stride * at) : make_int4(0, -1, 0, 0);
        const int c = fin_meta_class(r0.x);
        if (kSingles) {
            const bool single = c == kFinSingle;
            fin_singles<kStats>(p, t, single, r0.y, single ? degree_of(__ldg(p.ranges + r0.y)) : 0, i < cb, last_all);
        }
        const int v = c == kFinRootCand ? r0.y : -1;
        int rres = kFinNotRoot;
        FinComp cp;
        if (c == kFinRootCand) rres = fin_search_thread<kW>(p, v, at, cp);
        // the lanes' components, packed into the warp and played together, a lane
        // per member (a lane playing its component alone would colour its
        // members one after another)
        unsigned pend = __ballot_sync(kFull, kPlay && rres == kFinRoot);
        while (pend) {
            const bool mine = (pend >> lane) & 1u;
            const int km = mine ? cp.k : 0, nem = mine ? (int)cp.eoff[cp.k] : 0;
            int pk = km, pe = nem;  // inclusive prefix sums in lane order
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(kFull, pk, o), z = __shfl_up_sync(kFull, pe, o);
                if (lane >= o) {
                    pk += y;
                    pe += z;
                }
            }
            const bool take = mine && pk <= kFinMembers && pe <= kFinEntries;
            const unsigned batch = __ballot_sync(kFull, take);  // a prefix of pend
            const int lastl = 31 - __clz(batch);
            const int ktot = __shfl_sync(kFull, pk, lastl), etot = __shfl_sync(kFull, pe, lastl);
            if (take) {
                const int mo = pk - km, eo = pe - nem;
                for (int l = 0; l < km; ++l) {
                    fw.mem[mo + l] = cp.mem[l];
                    fw.eoff[mo + l] = eo + cp.eoff[l];
                }
                for (int e = 0; e < nem; ++e) {
                    fw.pref[eo + e] = cp.pref[e];
                    fw.tgt[eo + e] = (uint8_t)(mo + cp.tgt[e]);
                }
            }
            if (lane == 0) fw.eoff[ktot] = etot;
            __syncwarp();
            const int ml = lane < ktot ? fw.mem[lane] : 0;
            last_all = max(last_all, fin_play<kW, kStats>(p, fw, t, ml, ktot));
            __syncwarp();  // fw is refilled by the next batch
            pend &= ~batch;
        }
        unsigned roots = __ballot_sync(kFull, rres == kFinOverflow);
        while (roots) {
            const int s = __ffs(roots) - 1;
            roots &= roots - 1;
            int mem, k;
            unsigned long long seen = 0;
            const int r = fin_search<kW>(p, fw, __shfl_sync(kFull, v, s), &mem, &k, kStats && !kPlay ? &seen : nullptr);
            if (kStats && !kPlay && lane == 0) atomicAdd(&p.stats[(size_t)t * MM_STATS_COLS + MM_ST_FINISH_ENTRIES], seen);
            if (r == kFinTooBig) {
                abort = true;
                break;
            }
            if (kPlay && r == kFinRoot) last_all = max(last_all, fin_play<kW, kStats>(p, fw, t, mem, k));
            __syncwarp();  // fw is reused by the next root
        }
        if (__any_sync(kFull, abort)) break;
    }
    if (kPlay) {
        last_all = __reduce_max_sync(kFull, last_all);
        if (lane == 0 && last_all >= 0) atomicMax(&p.ctl->fin_last, last_all);
    }
    return abort;
}

// One barrier of k_match, with the block's summand (two words of shared memory)
// and the sum over the blocks.
__device__ __forceinline__ bool barrier_sum(const Params &p, Smem &sm, unsigned &turn, const int *part, unsigned *sum, int mark)
{
    return grid_sync(sm, p.ctl, turn, part, sum, p.result, p.tstamp, mark, p.spin_limit, p.skip_mark);
}

// The finish phase of round t.  Returns -1 if a barrier wait gave up, else
// whether the phase completed (0: called off, the round has to be played).
// Profile: the first pass is reported as round t's window scan, the rest as
// its fallback scan.
template <bool kW, bool kStats>
__device__ __forceinline__ int finish_phase(const Params &p, Smem &sm, unsigned &turn, int t, const int *list, int cb, int cr)
{
    unsigned off;
    auto call_off = [&](bool abort) {  // the block's summand: sm.flag + sm.zero
        if (abort) sm.flag = 1;
    };
    // counters must not count a called-off attempt: the instrumented kernel
    // checks, then resolves; the plain one is speculative (a called-off attempt
    // leaves only values that the rounds write again)
    call_off(finish_scan<kW, kStats, !kStats>(p, t, list, cb, cr));
    if (!barrier_sum(p, sm, turn, &sm.flag, &off, 3 * t + 1)) return -1;
    if (kStats && !off) {
        call_off(finish_roots<kW, kStats, false, false>(p, sm, t, cb, cr));
        if (!barrier_sum(p, sm, turn, &sm.flag, &off, -1)) return -1;
    }
    if (!off) {
        call_off(finish_roots<kW, kStats, true, kStats>(p, sm, t, cb, cr));
        if (!barrier_sum(p, sm, turn, &sm.flag, &off, 3 * t + 2)) return -1;
    }
    if (off) {
        if (threadIdx.x == 0) sm.flag = 0;
        __syncthreads();  // the working areas change hands
        return 0;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const int last = max(__ldcg(&p.ctl->fin_last), __ldcg(&p.ctl->iso_last) - 1);
        p.result->rounds = p.maximal ? min(last + 2, p.cap) : p.cap;
        if (p.tstamp) p.tstamp[3 * t + 3] = p.tstamp[3 * t + 2];
    }
    return 1;
}

// The whole matching in one cooperative launch: set-up, then per round the
// window scan (A1), the shared fallback scan (A2, only in rounds that have
// such lists) and the commit phase (B), separated by grid barriers, until the
// finish phase plays the remaining rounds or no vertex is left.  Every block
// gets the same sums from the barriers, so all blocks take the same branches
// and leave the loop at the same round.  Vertices that could still be matched
// at the end keep their last colour as their match value (the reference
// leaves match[v] = 0 / 1 for them).
template <bool kW, bool kStats, bool kPolicy, bool kSolo>
__global__ void __launch_bounds__(kThreads, kSolo ? 1 : 2) k_match(const __grid_constant__ Params p)
{
    extern __shared__ __align__(16) unsigned char dsmem[];
    Smem &sm = *reinterpret_cast<Smem *>(dsmem);
    SoloMem &solo = *reinterpret_cast<SoloMem *>(dsmem + kSmemBytes);
    const Mem<kSolo> m = kSolo ? Mem<kSolo>{solo.col, solo.best} : Mem<kSolo>{p.col, p.best};
    const long long rbase = (long long)blockIdx.x * p.region;
    const bool first = blockIdx.x == 0 && threadIdx.x == 0;
    // the next call's control block (no block of this call reads it)
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < (int)(sizeof(Ctl) / 8); i += kThreads)
            reinterpret_cast<unsigned long long *>(p.ctl_next)[i] = 0ull;
    unsigned turn = 0, act = 0, shared = 0;
    int t = 0;
    init_phase<kW, kStats, kPolicy>(p, m, sm, kSolo ? solo.lists[0] : p.lists[0] + rbase);
    if (!barrier_sum(p, sm, turn, sm.count[0], &act, 0)) return;
    const unsigned active0 = act;  // active vertices at round 0
    unsigned fin_next = active0;   // finish phase: attempt once the active set is this small
    for (;; ++t) {
        int *list = kSolo ? solo.lists[t & 1] : p.lists[t & 1] + rbase;
        int *next = kSolo ? solo.lists[(t & 1) ^ 1] : p.lists[(t & 1) ^ 1] + rbase;
        const int cb = sm.count[t & 1][0], cr = sm.count[t & 1][1];
        // the finish phase; in one block the rounds cost less than it does
        if (!kSolo && p.fin && t > 0 && act > 0 && act <= fin_next &&
            (unsigned long long)act * (unsigned)p.fin_div <= active0) {
            const int done = finish_phase<kW, kStats>(p, sm, turn, t, list, cb, cr);
            if (done < 0) return;
            if (done) break;
            fin_next = act / 2;  // called off: again when the set has halved
        }
        scan_window<kW, kStats, kPolicy>(p, m, sm, t, list, rbase, cb, cr);
        if (!barrier_sum(p, sm, turn, &sm.flag, &shared, 3 * t + 1)) return;
        if (shared) {
            scan_shared<kW, kStats>(p, m, t);
            if (!barrier_sum(p, sm, turn, &sm.flag, &shared, -1)) return;
            if (first) p.ctl->staged_pack = 0ull;  // empty again for the next round
        }
        if (p.tstamp && first) p.tstamp[3 * t + 2] = global_ns();
        bool has_next = t + 1 < p.cap;
        const bool seeds_short = has_next && t + 1 >= p.nseeds;
        if (seeds_short) has_next = false;
        commit_phase<kW, kStats, kPolicy>(p, m, sm, t, has_next, list, next, rbase, cb, cr);
        if (!barrier_sum(p, sm, turn, sm.count[(t & 1) ^ 1], &act, 3 * t + 3)) return;
        if (has_next && act > 0) continue;
        // the loop ends; survivors of the last round keep its colours
        if (first) {
            int rounds = p.maximal && act == 0 ? min(t + 2, p.cap) : p.cap;
            // vertices without neighbours resolved at set-up
            const int iso = __ldcg(&p.ctl->iso_last) - 1;
            if (p.maximal && iso >= 0) rounds = max(rounds, min(iso + 2, p.cap));
            p.result->rounds = rounds;
            if (seeds_short) p.result->status = 1;
        }
        const int eb = sm.count[(t & 1) ^ 1][0], er = sm.count[(t & 1) ^ 1][1];
        for (int i = threadIdx.x; i < eb + er; i += kThreads) {
            const int v = item_at<kSolo>(p, next, eb, i);
            p.match[v] = i < eb ? kBlue : kRed;
            if (p.last) p.last[v] = (uint8_t)t;
        }
        break;
    }
}

// ---------------------------------------------------------------------------
// Preparation: degree classes and reverse proposal keys.

// (block sums: an atomic a warp and word had all warps queue on six words)
__global__ void __launch_bounds__(256) k_scan_ranges(const int2 *ranges, int n, long long nnz, RangeInfo *info, long long *deg_out)
{
    unsigned long long sum = 0, nlong = 0, elong = 0, groups = 0, even = 0;
    int mx = 0, nc = 0, bad = 0;
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const int2 r = ranges[v];
        // the ends are compared before their difference is taken: (-1, 2^31 - 1)
        // has none in 32 bits
        const bool out = r.y > r.x && (r.x < 0 || (long long)r.y > nnz);
        if (out) bad = 1;
        const int d = out ? 0 : degree_of(r), wl = win_len(d);
        sum += (unsigned long long)d;
        mx = max(mx, d);
        if (d > kWin) {
            nlong += 1;
            elong += (unsigned long long)d;
        }
        groups += (wl + 3) >> 2;
        even += (wl + 1) & ~1;
        if (deg_out) deg_out[v] = d;
        if (r.y < r.x) nc = 1;
        if (v == 0 && r.x != 0) nc = 1;
        if (v + 1 < n && ranges[v + 1].x != r.y) nc = 1;
        if (v == n - 1 && (long long)r.y != nnz) nc = 1;
    }
    block_add(&info->sum_deg, sum);
    block_add(&info->long_count, nlong);
    block_add(&info->long_entries, elong);
    block_add(&info->win_groups, groups);
    block_add(&info->win_even, even);
    __shared__ int s_max;
    if (threadIdx.x == 0) s_max = 0;
    __syncthreads();
    mx = __reduce_max_sync(kFull, mx);
    nc = __any_sync(kFull, nc);
    bad = __any_sync(kFull, bad);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&s_max, mx);
        if (nc) atomicOr(&info->noncontig, 1);
        if (bad) atomicOr(&info->bad, 1);
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_max) atomicMax(&info->max_deg, (unsigned long long)s_max);
}

// One item per (owner, slot): key = (min << B | max) << 1 | (owner == max).
__global__ void k_pair_items(const int2 *ranges, const int *nbrs, int n, int bits, int contiguous,
                             const long long *slot_off, unsigned long long *keys, int *vals)
{
    const int lane = threadIdx.x & 31;
    const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long v = warp0; v < n; v += nwarps) {
        const int2 r = ranges[v];
        const long long s0 = contiguous ? (long long)r.x : slot_off[v];
        for (Pos i = lane; i < (Pos)degree_of(r); i += 32) {
            const unsigned long long a = (unsigned long long)v, b = (unsigned long long)nbrs[r.x + i];
            const unsigned long long lo = a < b ? a : b, hi = a < b ? b : a;
            const long long slot = s0 + i;
            keys[slot] = (((lo << bits) | hi) << 1) | (a > b ? 1ull : 0ull);
            vals[slot] = (int)slot;
        }
    }
}

// Key red `owner` gives the entry at `slot` of its own list (the revkey form:
// 0 for weights the reference can never pick).
template <bool kW>
__device__ __forceinline__ unsigned long long red_key(const int2 *ranges, const float *w, int contiguous,
                                                      const long long *slot_off, long long owner, long long slot)
{
    const long long pos = contiguous ? slot : (long long)ranges[owner].x + (slot - slot_off[owner]);
    if (kW) {
        const float x = w[pos];
        return x > -1.0f ? (((unsigned long long)weight_order(x) << 32) | (uint32_t)~(int)pos) : 0ull;
    }
    return (unsigned long long)(uint32_t)~(int)pos;
}

// For each group of equal unordered pair, give every item the best key of the
// opposite direction.  Groups are walked by their first item.
template <bool kW>
__global__ void k_pair_groups(const unsigned long long *keys, const int *vals, long long count, int bits,
                              const int2 *ranges, const float *w, int contiguous, const long long *slot_off,
                              unsigned long long *revkey)
{
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < count;
         q += (long long)gridDim.x * blockDim.x) {
        const unsigned long long kq = keys[q] >> 1;
        if (q > 0 && (keys[q - 1] >> 1) == kq) continue;
        const long long lo = (long long)(kq >> bits), hi = (long long)(kq & ((1ull << bits) - 1));
        long long end = q + 1;
        while (end < count && (keys[end] >> 1) == kq) ++end;
        if (lo == hi) {  // self-loops never carry a proposal
            for (long long x = q; x < end; ++x) revkey[vals[x]] = 0ull;
            continue;
        }
        unsigned long long best_dir[2] = {0ull, 0ull};
        for (long long x = q; x < end; ++x) {
            const int dir = (int)(keys[x] & 1ull);
            const long long owner = dir ? hi : lo;
            const unsigned long long k = red_key<kW>(ranges, w, contiguous, slot_off, owner, vals[x]);
            best_dir[dir] = k > best_dir[dir] ? k : best_dir[dir];
        }
        for (long long x = q; x < end; ++x) revkey[vals[x]] = best_dir[(keys[x] & 1ull) ^ 1ull];
    }
}

// ---- preference windows (weighted types) ----
//
// pwin holds, for every vertex, its best min(deg, 32) entries in the order in
// which the reference's gwRequest would prefer them: candidates (weight > -1)
// by weight, then earlier position; entries whose weight can never be picked
// after them, flagged by bit 31 of the position.  A vertex's window starts at
// group pwin_off[v] (bit 31 apart), four entries a group, read by one 32-byte
// load; the last group is filled up.
__device__ __forceinline__ unsigned long long pref_key(float w, int j)
{
    return w > -1.0f ? (((unsigned long long)weight_order(w) << 32) | (uint32_t)~j) : (unsigned long long)(uint32_t)~j;
}

// One compare-exchange step of a bitonic network across the warp: the lower
// lane of each pair keeps the larger key in a descending block.
__device__ __forceinline__ void cas_step(unsigned long long &k, int &nb, int &j, int lane, int stride, bool desc)
{
    const unsigned long long ok = __shfl_xor_sync(kFull, k, stride);
    const int onb = __shfl_xor_sync(kFull, nb, stride);
    const int oj = __shfl_xor_sync(kFull, j, stride);
    const bool lower = (lane & stride) == 0;
    if (lower == desc ? ok > k : ok < k) {
        k = ok;
        nb = onb;
        j = oj;
    }
}

__device__ __forceinline__ void warp_sort_desc(unsigned long long &k, int &nb, int &j, int lane)
{
#pragma unroll
    for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) cas_step(k, nb, j, lane, stride, (lane & size) == 0);
}

// Window offsets as the kernels read them: the first group of four entries,
// and in bit 31 whether the list is longer than its window.
__global__ void k_win_offsets(const int2 *ranges, const long long *off, int n, int *pwin_off)
{
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v <= n; v += gridDim.x * blockDim.x)
        pwin_off[v] = (int)((unsigned)off[v] | (v < n && degree_of(ranges[v]) > kWin ? 0x80000000u : 0u));
}

// Groups of each vertex's window.
__global__ void k_win_sizes(const int2 *ranges, int n, long long *groups)
{
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v <= n; v += gridDim.x * blockDim.x)
        groups[v] = v < n ? (win_len(degree_of(ranges[v])) + 3) >> 2 : 0;
}

constexpr int kWinRows = 8;       // rows of 32 entries tested against the window threshold per step
constexpr int kWinChunk = 4096;   // lists longer than this are split into chunks of this many entries

// Merge entries [from, to) of a list into its sorted best 32 (k, nb, j): a row
// can change them only if one of its keys beats the 32nd.
__device__ __forceinline__ void win_merge_range(const int *nbrs, const float *w, int from, int to, int lane,
                                                unsigned long long &k, int &nb, int &j)
{
    // offsets within the range (at most kWinChunk entries): positions past its end
    // may not fit an int, and unsigned ones took the last chunk of an upload 60 us longer
    const int len = to - from;
    nbrs += from;
    w += from;
    for (int base = 0; base < len; base += 32 * kWinRows) {
        float wr[kWinRows];
#pragma unroll
        for (int q = 0; q < kWinRows; ++q) {
            const int i = base + q * 32 + lane;
            wr[q] = i < len ? __ldg(w + i) : 0.0f;
        }
#pragma unroll
        for (int q = 0; q < kWinRows; ++q) {
            const int i = base + q * 32 + lane;
            if (base + q * 32 >= len) break;
            const unsigned long long thr = __shfl_sync(kFull, k, 31);
            unsigned long long k2 = i < len ? pref_key(wr[q], from + i) : 0ull;
            if (!__any_sync(kFull, k2 > thr)) continue;
            int nb2 = i < len ? __ldg(nbrs + i) : 0, j2 = i < len ? from + i : 0;
            warp_sort_desc(k2, nb2, j2, lane);
            // the larger of T[l] and R[31 - l] is a bitonic sequence holding
            // the best 32 of both; sort it descending
            const unsigned long long rk = __shfl_sync(kFull, k2, 31 - lane);
            const int rnb = __shfl_sync(kFull, nb2, 31 - lane), rj = __shfl_sync(kFull, j2, 31 - lane);
            if (rk > k) {
                k = rk;
                nb = rnb;
                j = rj;
            }
#pragma unroll
            for (int stride = 16; stride > 0; stride >>= 1) cas_step(k, nb, j, lane, stride, true);
        }
    }
}

// Best 32 entries of [from, to): the first 32 sorted, then the rest merged in.
__device__ __forceinline__ void win_top32(const int *nbrs, const float *w, int from, int to, int lane,
                                          unsigned long long &k, int &nb, int &j)
{
    k = 0ull;
    nb = 0;
    j = 0;
    if (lane < to - from) {
        j = from + lane;
        nb = __ldg(nbrs + j);
        k = pref_key(__ldg(w + j), j);
    }
    warp_sort_desc(k, nb, j, lane);
    if (to - from > 32) win_merge_range(nbrs, w, from + 32, to, lane, k, nb, j);
}

__device__ __forceinline__ void win_store(int2 *pwin, long long off, int deg, int lane, unsigned long long k, int nb, int j)
{
    const int wl = win_len(deg);
    if (lane < wl) pwin[off + lane] = make_int2(nb, k >= (1ull << 32) ? j : (int)((unsigned)j | 0x80000000u));
    else if (lane < ((wl + 3) & ~3)) pwin[off + lane] = make_int2(-1, (int)0x80000000u);  // fillers
}

// Windows of lists of at most kWinChunk entries, a warp per list (vertices
// dealt round-robin, so long lists spread over the grid); longer lists are
// queued for the chunked kernels.
__global__ void __launch_bounds__(256) k_win_build(const int2 *ranges, const int *nbrs, const float *w, int va, int vb,
                                                   const int *pwin_off, int2 *pwin, int *big, int *nbig)
{
    const int lane = threadIdx.x & 31;
    const long long gwarp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long v = va + gwarp; v < vb; v += nwarps) {
        const int2 r = ranges[v];
        const int deg = degree_of(r);
        if (deg == 0) continue;
        if (deg > kWinChunk) {
            if (lane == 0) big[atomicAdd(nbig, 1)] = (int)v;
            continue;
        }
        unsigned long long k;
        int nb, j;
        win_top32(nbrs, w, r.x, r.y, lane, k, nb, j);
        win_store(pwin, 4ll * (pwin_off[v] & 0x7fffffff), deg, lane, k, nb, j);
    }
}

// Chunked lists, step 1: the best 32 of every kWinChunk-entry chunk of every
// queued list, a warp per chunk.  cand holds 32 {key, nb, j} per chunk.
struct WinCand {
    unsigned long long k;
    int nb;
    int j;
};

__global__ void __launch_bounds__(256) k_win_chunks(const int2 *ranges, const int *nbrs, const float *w,
                                                    const int *big, int nbig, const long long *chunk_off,
                                                    WinCand *cand)
{
    const int lane = threadIdx.x & 31;
    const long long gwarp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    const long long total = chunk_off[nbig];
    for (long long c = gwarp; c < total; c += nwarps) {
        int lo = 0, hi = nbig - 1;  // the list holding chunk c: largest i with chunk_off[i] <= c
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (chunk_off[mid] <= c) lo = mid;
            else hi = mid - 1;
        }
        const int2 r = ranges[big[lo]];
        const int from = r.x + (int)(c - chunk_off[lo]) * kWinChunk;
        const int to = from + min(kWinChunk, r.y - from);
        unsigned long long k;
        int nb, j;
        win_top32(nbrs, w, from, to, lane, k, nb, j);
        cand[c * 32 + lane] = WinCand{k, nb, j};
    }
}

__global__ void k_win_chunk_counts(const int2 *ranges, const int *big, int nbig, long long *counts)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nbig; i += gridDim.x * blockDim.x)
        counts[i] = (degree_of(ranges[big[i]]) + kWinChunk - 1) / kWinChunk;
}

// Chunked lists, step 2: a warp per list merges its chunks' sorted best 32s.
__global__ void __launch_bounds__(256) k_win_chunk_merge(const int2 *ranges, const int *big, int nbig,
                                                         const long long *chunk_off, const WinCand *cand,
                                                         const int *pwin_off, int2 *pwin)
{
    const int lane = threadIdx.x & 31;
    const long long gwarp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long i = gwarp; i < nbig; i += nwarps) {
        const long long c0 = chunk_off[i], c1 = chunk_off[i + 1];
        WinCand x = cand[c0 * 32 + lane];
        unsigned long long k = x.k;
        int nb = x.nb, j = x.j;
        for (long long c = c0 + 1; c < c1; ++c) {
            const WinCand y = cand[c * 32 + (31 - lane)];  // reversed: the pairwise larger is bitonic
            if (y.k > k) {
                k = y.k;
                nb = y.nb;
                j = y.j;
            }
#pragma unroll
            for (int stride = 16; stride > 0; stride >>= 1) cas_step(k, nb, j, lane, stride, true);
        }
        const int v = big[i];
        win_store(pwin, 4ll * (pwin_off[v] & 0x7fffffff), degree_of(ranges[v]), lane, k, nb, j);
    }
}

// ---- reverse keys from sorted lists ----------------------------------------
// When every neighbour list is sorted, the entries of u that point back at v
// form one run in u's list, found by binary search.  Of the two entries of a
// pair {v, u} only the one whose partner list is shorter searches (ties by
// id): it finds the run of entries pointing back in the partner's list, stores
// the best of their keys in its own slot (pull) and max-combines its own key
// into the slots of that run (push), which nobody else writes.  Each pair thus
// costs one search in its shorter list; hub lists are never searched by their
// many neighbours.  Slots are cut into chunks of kRevChunk; k_chunk_owner
// finds the vertex owning each chunk's first slot, k_revkey_sorted resolves
// the owner of every slot in shared memory and checks sortedness on the way
// (any descending neighbour pair sets *unsorted and the pair-sort build runs).
// revkey must be zero on entry.
constexpr int kRevChunk = 2048;
constexpr int kRevThreads = 256;

__device__ __forceinline__ long long slot_prefix(const int2 *ranges, int contiguous, const long long *slot_off,
                                                 long long v)
{
    return contiguous ? (long long)ranges[v].x : slot_off[v];
}

// Owner of slot s: the largest v with prefix(v) <= s.
__device__ __forceinline__ int owner_of(const int2 *ranges, int contiguous, const long long *slot_off, int lo, int hi,
                                        long long s)
{
    while (lo < hi) {
        const int mid = (int)(((long long)lo + hi + 1) >> 1);
        if (slot_prefix(ranges, contiguous, slot_off, mid) <= s) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

__global__ void k_chunk_owner(const int2 *ranges, int n, int contiguous, const long long *slot_off, long long S,
                              int *chunk_v)
{
    const long long chunks = (S + kRevChunk - 1) / kRevChunk;
    for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c <= chunks;
         c += (long long)gridDim.x * blockDim.x) {
        const long long s = c * kRevChunk < S ? c * kRevChunk : S - 1;
        chunk_v[c] = owner_of(ranges, contiguous, slot_off, 0, n - 1, s);
    }
}

// Key red `owner` gives its entry at absolute position q (0: never picked).
template <bool kW>
__device__ __forceinline__ unsigned long long entry_red_key(const float *w, int q)
{
    if (kW) {
        const float x = __ldg(w + q);
        return x > -1.0f ? (((unsigned long long)weight_order(x) << 32) | (uint32_t)~q) : 0ull;
    }
    return (unsigned long long)(uint32_t)~q;
}

template <bool kW>
__global__ void __launch_bounds__(kRevThreads) k_revkey_sorted(const int2 *ranges, const int *nbrs, const float *w,
                                                               int contiguous, const long long *slot_off, long long S,
                                                               const int *chunk_v, unsigned long long *revkey,
                                                               int *unsorted)
{
    constexpr int kCap = kRevChunk + 1;
    __shared__ int pre[kCap];  // prefix(v0 + i) - chunk start
    __shared__ int bad;
    if (threadIdx.x == 0) bad = 0;
    const long long chunks = (S + kRevChunk - 1) / kRevChunk;
    for (long long c = blockIdx.x; c < chunks; c += gridDim.x) {
        const long long s0 = c * kRevChunk;
        const int v0 = chunk_v[c], v1 = chunk_v[c + 1];
        const int cnt = v1 - v0 + 1;
        const bool in_smem = cnt <= kCap;
        __syncthreads();
        if (in_smem)
            for (int i = threadIdx.x; i < cnt; i += kRevThreads)
                pre[i] = (int)(slot_prefix(ranges, contiguous, slot_off, v0 + i) - s0);
        __syncthreads();
        for (int k = threadIdx.x; k < kRevChunk; k += kRevThreads) {
            const long long s = s0 + k;
            if (s >= S) break;
            int v;
            if (in_smem) {
                int lo = 0, hi = cnt - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (pre[mid] <= k) lo = mid;
                    else hi = mid - 1;
                }
                v = v0 + lo;
            } else {
                v = owner_of(ranges, contiguous, slot_off, v0, v1, s);
            }
            const int2 rv = ranges[v];
            const int pos = contiguous ? (int)s : (int)(rv.x + (s - slot_off[v]));
            const int u = nbrs[pos];
            if (pos + 1 < rv.y && nbrs[pos + 1] < u) bad = 1;
            if (u == v) continue;  // self-loops never carry a proposal
            const int2 ru = ranges[u];
            const int dv = degree_of(rv), du = degree_of(ru);
            if (du > dv || (du == dv && u > v)) continue;  // u's entries search my list and push here
            int lo = ru.x, hi = ru.x + du;  // first entry >= v in u's list
            while (lo < hi) {
                const int mid = (int)(((long long)lo + hi) >> 1);
                if (__ldg(nbrs + mid) < v) lo = mid + 1;
                else hi = mid;
            }
            const unsigned long long mine = entry_red_key<kW>(w, pos);
            const long long su0 = contiguous ? 0ll : slot_off[u] - ru.x;  // slot of entry q of u: su0 + q
            unsigned long long key = 0ull;
            for (int q = lo; q < ru.x + du && __ldg(nbrs + q) == v; ++q) {
                const unsigned long long kq = entry_red_key<kW>(w, q);
                key = kq > key ? kq : key;
                if (mine) atomicMax(revkey + su0 + q, mine);
            }
            if (key) revkey[s] = key;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && bad) atomicOr(unsorted, 1);
}


int bits_for(long long n)
{
    int b = 1;
    while ((1ll << b) < n) ++b;
    return b;
}

// Weight features of the learned colouring: max and mean of the weights a
// blue vertex could pick (> -1), 0 without any; a warp per vertex.
__global__ void k_wfeat(const int2 *ranges, const float *w, int n, float2 *wfeat)
{
    const int lane = threadIdx.x & 31;
    const long long gwarp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long v = gwarp; v < n; v += nwarps) {
        const int2 r = ranges[v];
        float mx = 0.0f, sum = 0.0f;
        int cnt = 0;
        for (Pos i = lane; i < (Pos)degree_of(r); i += 32) {
            const float x = __ldg(w + r.x + i);
            if (x > -1.0f) {
                mx = cnt ? fmaxf(mx, x) : x;
                sum += x;
                ++cnt;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float m2 = __shfl_xor_sync(kFull, mx, o);
            const int c2 = __shfl_xor_sync(kFull, cnt, o);
            mx = c2 && (!cnt || m2 > mx) ? m2 : mx;
            sum += __shfl_xor_sync(kFull, sum, o);
            cnt += c2;
        }
        if (lane == 0) wfeat[v] = make_float2(mx, cnt ? sum / (float)cnt : 0.0f);
    }
}

// Last active round of each graph of a batch (-1: none; cleared to that before):
// the maximum of its vertices' last[].  A warp takes 1024 vertices, 16 bytes a
// lane and load, and mostly finds them in one graph; a warp a graph left one
// warp with a graph of 2^18 vertices (0.3 ms of a batch that matches in 0.75).
constexpr int kLastSpan = 1024;

// The graph of vertex v: the largest i with goff[i] <= v (empty graphs before it share its start).
__device__ __forceinline__ int graph_of(const int *goff, int ngraphs, int v)
{
    int lo = 0, hi = ngraphs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(goff + mid) <= v) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

__global__ void __launch_bounds__(256) k_batch_last(const uint8_t *last, int n, const int *goff, int ngraphs, int *out)
{
    const int lane = threadIdx.x & 31;
    const long long gwarp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long v0 = gwarp * kLastSpan; v0 < n; v0 += nwarps * kLastSpan) {
        const int v1 = (int)min((long long)n, v0 + kLastSpan);
        const int g = graph_of(goff, ngraphs, lane == 0 ? (int)v0 : v1 - 1);  // lane 0: the first, others: the last
        const int g0 = __shfl_sync(kFull, g, 0), g1 = __shfl_sync(kFull, g, 31);
        if (g0 == g1) {
            int mx = 0;
            for (int v = (int)v0 + lane * 16; v < v1; v += 32 * 16) {
                if (v + 16 <= v1) {
                    const uint4 x = __ldg(reinterpret_cast<const uint4 *>(last + v));
                    const unsigned m = __vmaxu4(__vmaxu4(x.x, x.y), __vmaxu4(x.z, x.w));
                    mx = max(mx, (int)max(max(m & 255u, (m >> 8) & 255u), max((m >> 16) & 255u, m >> 24)));
                } else {
                    for (int q = v; q < v1; ++q) mx = max(mx, (int)last[q]);
                }
            }
            mx = __reduce_max_sync(kFull, mx);
            if (lane == 0 && __ldcg(out + g0) < mx) atomicMax(out + g0, mx);
        } else {
            // several graphs: each with its own vertices in the span
            for (int gi = g0; gi <= g1; ++gi) {
                const int lo = max((int)v0, __ldg(goff + gi)), hi = min(v1, __ldg(goff + gi + 1));
                int mx = -1;
                for (int v = lo + lane; v < hi; v += 32) mx = max(mx, (int)last[v]);
                mx = __reduce_max_sync(kFull, mx);
                if (lane == 0 && mx >= 0 && __ldcg(out + gi) < mx) atomicMax(out + gi, mx);
            }
        }
    }
}

constexpr int kStampCount = 3 * kMaxRounds + 1;
constexpr size_t kResultBytes = 256;

struct PushState {
    // one allocation: the arrays from col to ctl
    void *arena = nullptr;
    uint32_t *col = nullptr;
    int2 *req = nullptr;
    unsigned long long *best = nullptr;
    unsigned long long *part_key = nullptr;
    int *part_cnt = nullptr;
    int *list_mem = nullptr;          // the two parities' lists, list_cap items each
    size_t list_cap = 0;
    int *prop = nullptr;              // list_cap requests
    int4 *staged = nullptr;
    int *piece_item = nullptr;
    Ctl *ctl = nullptr;               // two control blocks, used by alternate calls
    int ctl_turn = 0;
    uint32_t *prop_key = nullptr;     // list_cap key halves, once a type off the symmetric path needs them
    int4 *rec = nullptr;              // finish phase: records, once a call needs them
    size_t rec_cap = 0;               // int4 that rec holds
    Result *result = nullptr;         // pinned: written by the kernel
    unsigned long long *stats = nullptr;
    unsigned long long *tstamp = nullptr;
    // The last call on this state ended with every grid barrier complete (the
    // next call's control block is clear) and every fallback list combined
    // (part_key and part_cnt all zero); false after a call that gave up or failed.
    bool at_rest = false;
    bool zero_next = true;  // the call being launched resets them (the last one did not end at rest)
    float2 *wfeat = nullptr;              // learned colouring: (max, mean) incident weight per vertex
};

void free_state(PushState *s)
{
    // callers have synchronised the device (graph destroy or a failed set-up)
    dev_free(s->arena, 0);
    dev_free(s->prop_key, 0);
    dev_free(s->rec, 0);
    pinned_put(s->result, kResultBytes);
    dev_free(s->stats, 0);
    dev_free(s->tstamp, 0);
    dev_free(s->wfeat, 0);
    delete s;
}

constexpr size_t smem_bytes(bool solo) { return kSmemBytes + (solo ? sizeof(SoloMem) : 0); }

template <bool kW, bool kStats, bool kPolicy, bool kSolo>
int coresident_blocks(int sms)
{
    int occ = 0;
    if (cudaFuncSetAttribute(k_match<kW, kStats, kPolicy, kSolo>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem_bytes(kSolo)) != cudaSuccess)
        return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_match<kW, kStats, kPolicy, kSolo>, kThreads,
                                                      smem_bytes(kSolo)) != cudaSuccess)
        return 0;
    return occ * sms;
}

constexpr int kMaxBlocks = 1024;

// What the device allows, found out once (the kernels' shared memory limits are
// set on the way).
struct DeviceLimits {
    bool known = false;
    int coop = 0;
    int sms = 0;
    int grid[2][3] = {{0, 0, 0}, {0, 0, 0}};  // co-resident blocks of k_match by weighting and mode
    int solo = 0;                             // the one-block kernels fit
};
std::mutex g_limits_mu;
DeviceLimits g_limits[256];

mm_status device_limits(int dev, DeviceLimits *out)
{
    if (dev < 0 || dev >= 256) {
        set_error("push: device ordinal out of range");
        return MM_ERR_UNSUPPORTED;
    }
    std::lock_guard<std::mutex> lock(g_limits_mu);
    DeviceLimits &d = g_limits[dev];
    if (!d.known) {
        DeviceLimits x;
        cudaDeviceGetAttribute(&x.sms, cudaDevAttrMultiProcessorCount, dev);
        cudaDeviceGetAttribute(&x.coop, cudaDevAttrCooperativeLaunch, dev);
        x.grid[0][0] = coresident_blocks<false, false, false, false>(x.sms);
        x.grid[0][1] = coresident_blocks<false, true, false, false>(x.sms);
        x.grid[0][2] = coresident_blocks<false, false, true, false>(x.sms);
        x.grid[1][0] = coresident_blocks<true, false, false, false>(x.sms);
        x.grid[1][1] = coresident_blocks<true, true, false, false>(x.sms);
        x.grid[1][2] = coresident_blocks<true, false, true, false>(x.sms);
        x.solo = coresident_blocks<false, false, false, true>(x.sms) > 0 && coresident_blocks<true, false, false, true>(x.sms) > 0;
        const cudaError_t le = cudaGetLastError();
        if (le != cudaSuccess) return cuda_fail(le, "push: kernel attributes");
        x.known = true;
        d = x;
    }
    bool over = false, under = !d.coop || !d.solo;
    for (int a = 0; a < 2; ++a)
        for (int b = 0; b < 3; ++b) {
            over |= d.grid[a][b] > kMaxBlocks;
            under |= d.grid[a][b] < 1;
        }
    if (over) {
        set_error("push: more co-resident blocks than the lists are sized for");
        return MM_ERR_UNSUPPORTED;
    }
    if (under) {
        set_error("push: the device cannot run the cooperative round kernel");
        return MM_ERR_UNSUPPORTED;
    }
    *out = d;
    return MM_OK;
}

// Blocks that a graph can use: one for 512 vertices, and one a multiprocessor
// where the lists longer than a window have the entries for it, as those lists
// are what a whole round can come to.  (Random maximal matching, 8192 vertices of
// degree 512: 16 blocks 2760 us, 128 blocks 1580, 256 blocks 2200: two blocks on a
// multiprocessor, the one that waits at a barrier takes the other's L1.)
constexpr long long kBlockEntries = 32768;
int useful_blocks(const mm_graph *g, int sms)
{
    const long long by_vertices = ((long long)g->n + kThreads - 1) / kThreads;
    const long long by_entries = std::min<long long>(sms, g->long_entries / kBlockEntries);
    return (int)std::min<long long>(std::max({1ll, by_vertices, by_entries}), kMaxBlocks);
}

// One block matches a graph of at most kSoloVertices vertices while its long
// lists are few: below these many entries the grid barriers cost more than one
// multiprocessor's scans.  A random type's window is a list's first entries, which
// are the same few vertices for many lists, so it scans many lists whole; a
// weighted type's are the heaviest, and it scans few.  (One block against the
// grid, random maximal: 1024 vertices of degree 64 132 us / 162, 128 255 / 333; 4096 of
// degree 64 335 / 250, 512 6400 / 990.  Weighted: 4096 of degree 512 132 / 380, 4000 372 / 133.)
constexpr long long kSoloEntries[2] = {1 << 17, 1 << 23};

// Dense graphs: this many entries a vertex in long lists, on average.
//
// Random types, where those lists come near the length from which the whole block
// scans one (kSharedLength on average): a block that finds more than kOwnEntries
// of them to scan whole in a round leaves its lists to all blocks.  A round of such
// a graph is such scans, in list order from the same few ends, one after another
// in a block and uneven over the blocks.  (Random, own scans / shared ones: 65536
// vertices of degree 400, 20 rounds, 464 us / 546; of 512, maximal, 4510 / 1850; 4096 of 512
// 1070 / 990, of 4000 16060 / 5560.  Weighted types scan too few lists to gain: 4096 of
// 4000 133 / 204.)
//
// Finish phase: an active set of 1/d of the vertices falls apart once its vertices
// have about one active neighbour each, so d is the average degree there; attempts
// at 1/24 meet components that no warp can hold, and are called off one after
// another (weighted maximal, 200 000 vertices of degree 512: 790 us / 206).
constexpr long long kDenseEntries = 384;
constexpr long long kSharedLength = 448;
constexpr long long kOwnEntries = 4096;
bool is_dense(const mm_graph *g) { return g->long_count > 0 && g->long_entries >= kDenseEntries * g->n; }

// The state's arrays, allocated and cleared on the call's stream (each call
// ends with its stream synchronised, so the next may come on another).
mm_status alloc_state(mm_graph *g, cudaStream_t stream, PushState **out)
{
    PushState *s = new (std::nothrow) PushState();
    if (!s) {
        set_error("push: host allocation failed");
        return MM_ERR_NOMEM;
    }
    const size_t n = (size_t)(g->n > 0 ? g->n : 1);
    // list capacities: every vertex is in at most one list per parity; only
    // lists longer than the window can fall back
    const size_t npiece_cap = (size_t)(g->long_entries / kPiece + g->long_count) + 1;
    const size_t nstaged = (size_t)(g->long_count > 0 ? g->long_count : 1);
    const size_t nparts = g->long_count > 0 ? n : 1;
    // whatever the grid, its blocks' regions fit: (n / kChunk / blocks + 1) chunks each
    DeviceLimits dev;
    const mm_status lim = device_limits(g->device, &dev);
    if (lim != MM_OK) {
        delete s;
        return lim;
    }
    s->list_cap = n + (size_t)kChunk * ((size_t)useful_blocks(g, dev.sms) + 1);
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t o = at;
        at += (bytes + 255) / 256 * 256;
        return o;
    };
    // the cleared ones first
    const size_t o_ctl = take(2 * sizeof(Ctl)), o_pk = take(nparts * sizeof(unsigned long long)),
                 o_pc = take(nparts * sizeof(int)), cleared = at;
    const size_t o_col = take((n + 15) / 16 * sizeof(uint32_t)), o_req = take(n * sizeof(int2)),
                 o_best = take(n * sizeof(unsigned long long)), o_lists = take(2 * s->list_cap * sizeof(int)),
                 o_prop = take(s->list_cap * sizeof(int)), o_staged = take(nstaged * sizeof(int4)),
                 o_piece = take(npiece_cap * sizeof(int));
    cudaError_t e = dev_alloc(&s->arena, at, stream);
    if (e == cudaSuccess) e = pinned_get((void **)&s->result, kResultBytes);
    if (e == cudaSuccess) e = cudaMemsetAsync(s->arena, 0, cleared, stream);
    if (e != cudaSuccess) {
        cudaDeviceSynchronize();
        free_state(s);
        cudaGetLastError();
        set_error(std::string("push: device allocation failed: ") + cudaGetErrorString(e));
        return MM_ERR_NOMEM;
    }
    char *base = (char *)s->arena;
    s->ctl = (Ctl *)(base + o_ctl);
    s->part_key = (unsigned long long *)(base + o_pk);
    s->part_cnt = (int *)(base + o_pc);
    s->col = (uint32_t *)(base + o_col);
    s->req = (int2 *)(base + o_req);
    s->best = (unsigned long long *)(base + o_best);
    s->list_mem = (int *)(base + o_lists);
    s->prop = (int *)(base + o_prop);
    s->staged = (int4 *)(base + o_staged);
    s->piece_item = (int *)(base + o_piece);
    s->at_rest = true;
    *out = s;
    return MM_OK;
}

struct PolicyArgs {
    const float *mlp = nullptr;  // host, MM_POLICY_FLOATS
    bool constant = false;       // output weights all zero: the threshold is constant_bar
    uint32_t constant_bar = 0u;
    float level = 0.0f;
    float *trace = nullptr;
    int trace_rounds = 0;
};

// One matching call, between begin_call and end_call.
struct Call {
    mm_graph *g = nullptr;
    PushState *s = nullptr;
    int type = 0;
    uint32_t barrier = 0u;
    const uint32_t *seeds = nullptr;
    int nseeds = 0;
    int *match = nullptr;
    bool stats = false, timing = false;
    const PolicyArgs *pol = nullptr;
    cudaStream_t stream = 0;
};

template <bool kW, bool kStats, bool kPolicy>
mm_status launch_match(const Call &c)
{
    mm_graph *g = c.g;
    PushState *s = c.s;
    const PolicyArgs *pol = c.pol;
    DeviceLimits dev;
    const mm_status lim = device_limits(g->device, &dev);
    if (lim != MM_OK) return lim;
    Params p;
    std::memset(&p, 0, sizeof p);
    p.n = g->n;
    p.contiguous = g->contiguous ? 1 : 0;
    p.sym = (kW ? g->sym_weights : g->sym_struct) ? 1 : 0;
    p.ranges = g->d_ranges;
    p.nbrs = g->d_nbrs;
    p.w = g->d_w;
    p.revkey = g->d_revkey[kW ? 1 : 0];
    p.slot_off = g->d_slot_off;
    p.pwin = g->d_pwin;
    p.pwin_off = g->d_pwin_off;
    p.col = s->col;
    p.req = s->req;
    p.best = s->best;
    p.part_key = s->part_key;
    p.part_cnt = s->part_cnt;
    p.lists[0] = s->list_mem;
    p.lists[1] = s->list_mem + s->list_cap;
    p.prop = s->prop;
    p.staged = s->staged;
    p.piece_item = s->piece_item;
    p.vbase = g->ngraphs > 0 ? g->d_vbase : nullptr;
    p.last = g->ngraphs > 0 ? g->d_last : nullptr;
    p.wfeat = s->wfeat;
    p.match = c.match;
    p.barrier = c.barrier;
    p.cap = max_rounds_of(c.type);
    p.maximal = is_maximal(c.type) ? 1 : 0;
    p.nseeds = c.nseeds < 256 ? c.nseeds : 256;
    std::memcpy(p.seeds, c.seeds, sizeof(uint32_t) * (size_t)p.nseeds);
    p.ctl = s->ctl + s->ctl_turn;
    p.ctl_next = s->ctl + (s->ctl_turn ^ 1);
    p.result = s->result;
    p.stats = kStats ? s->stats : nullptr;
    p.tstamp = c.timing ? s->tstamp : nullptr;
    p.zero_parts = s->zero_next ? 1 : 0;
    const bool sparse = g->sum_degree <= (long long)kFinSparse * g->n;
    const int fin_default = is_dense(g) ? (int)(g->sum_degree / g->n) : (sparse && !kPolicy ? kFinDivSparse : kFinDiv);
    p.fin_div = g->opt_fin_div < 0 ? 0 : (g->opt_fin_div == 0 ? fin_default : max(g->opt_fin_div, 2));
    p.spin_limit = debug_spin_limit();
    p.skip_mark = debug_skip_mark();
    if (kPolicy) {
        std::memcpy(p.mlp, pol->mlp, sizeof(p.mlp));
        p.policy_const = pol->constant ? 1 : 0;
        p.policy_bar = pol->constant_bar;
        p.level = pol->level;
        p.trace = pol->trace;
        p.trace_rounds = pol->trace_rounds;
        // the finish phase knows the policy's threshold, not its features
        p.fin_retire = pol->constant && !pol->trace ? 1 : 0;
    }
    // blocks: all that fit at once, or the tuned number per SM (never more), and
    // no more than the graph has work for
    const int mode = kPolicy ? 2 : (kStats ? 1 : 0);
    const int bps = g->opt_blocks_per_sm;
    int grid = bps > 0 ? min(dev.grid[kW][mode], bps * dev.sms) : dev.grid[kW][mode];
    grid = g->n <= kSoloVertices && g->long_entries <= kSoloEntries[kW] ? 1 : min(grid, useful_blocks(g, dev.sms));
    p.share_from = INT_MAX;
    if (!kW && is_dense(g) && g->long_entries >= kSharedLength * g->long_count)
        p.share_from = (int)(kOwnEntries / (g->long_entries / g->long_count)) + 1;
    const int chunks = (int)(((long long)g->n + kChunk - 1) / kChunk);
    p.region = (chunks + grid - 1) / grid * kChunk;
    p.turn_magic = grid > 1 ? (uint32_t)((1ull << 32) / (unsigned)grid + 1) : 0u;
    // the finish phase plays constant colourings of lists that are symmetric in
    // structure, whatever their order and weights (the policy's retirement rule
    // is the symmetric path's)
    p.fin = p.fin_div > 0 && grid > 1 && (kPolicy ? p.fin_retire && p.sym : p.sym || g->sym_pairs);
    p.rec_stride = p.sym ? 3 : 4;
    if (!p.sym) {
        if (!s->prop_key)
            MM_CUDA_TRY(dev_alloc((void **)&s->prop_key, sizeof(uint32_t) * s->list_cap, c.stream), "request keys");
        p.prop_key = s->prop_key;
    }
    if (p.fin) {
        // records for twice a block's share of the largest set the finish phase
        // accepts (a block that holds more calls the attempt off)
        p.rec_region = min(p.region, 2 * (p.region / p.fin_div) + kChunk);
        const size_t need = (size_t)p.rec_region * grid * p.rec_stride;
        if (need > s->rec_cap) {
            dev_free(s->rec, c.stream);
            s->rec = nullptr;
            s->rec_cap = 0;
            MM_CUDA_TRY(dev_alloc((void **)&s->rec, sizeof(int4) * need, c.stream), "finish records");
            s->rec_cap = need;
        }
        p.rec = s->rec;
    }
    void *args[] = {&p};
    // one block, in its shared memory (the instrumented and policy kernels keep
    // global memory: they are not for speed, or for larger graphs)
    constexpr bool kMaySolo = !kStats && !kPolicy;
    const bool solo = kMaySolo && grid == 1 && g->n <= kSoloVertices;
    const void *kernel = solo ? (const void *)k_match<kW, kStats, kPolicy, kMaySolo>
                              : (const void *)k_match<kW, kStats, kPolicy, false>;
    MM_CUDA_TRY(cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(kThreads), args, smem_bytes(solo), c.stream),
                "round kernel launch");
    return MM_OK;
}

// Shared set-up of one matching call: preparation, state, control block.
mm_status begin_call(Call &c)
{
    mm_graph *g = c.g;
    mm_status st = push_prepare(g, is_weighted(c.type) ? 1 : 0, c.stream);
    if (st != MM_OK) return st;
    PushState *s = (PushState *)g->push_exec;
    if (!s) {
        st = alloc_state(g, c.stream, &s);
        if (st != MM_OK) return st;
        g->push_exec = s;
    }
    c.s = s;
    // the control blocks are reset only after a call that did not end at rest;
    // until this call ends well, the state counts as not at rest
    s->zero_next = !s->at_rest;
    s->at_rest = false;
    if (s->zero_next) MM_CUDA_TRY(cudaMemsetAsync(s->ctl, 0, 2 * sizeof(Ctl), c.stream), "control block");
    // the previous call on this graph synchronised its stream before returning
    s->result->rounds = -1;
    s->result->status = 0;
    return MM_OK;
}

// A call that could not be launched leaves nothing in flight on its stream.
mm_status call_failed(const Call &c, mm_status st)
{
    cudaStreamSynchronize(c.stream);
    return st;
}

mm_status end_call(Call &c, int *rounds_out, long long *stats, int stats_rounds, unsigned long long *stamps)
{
    PushState *s = c.s;
    if (stats && stats_rounds > 0)
        MM_CUDA_TRY(cudaMemcpyAsync(stats, s->stats,
                                    sizeof(long long) * MM_STATS_COLS *
                                        (size_t)(stats_rounds < kMaxRounds ? stats_rounds : kMaxRounds),
                                    cudaMemcpyDeviceToHost, c.stream),
                    "stats read");
    if (stamps)
        MM_CUDA_TRY(cudaMemcpyAsync(stamps, s->tstamp, sizeof(unsigned long long) * kStampCount,
                                    cudaMemcpyDeviceToHost, c.stream),
                    "timestamps read");
    MM_CUDA_TRY(cudaStreamSynchronize(c.stream), "round loop");
    const Result out = *s->result;
    // every barrier completed unless one gave up (status 2)
    s->at_rest = out.status != 2 && out.rounds >= 0;
    s->ctl_turn ^= 1;  // cleared by this call
    if (!s->at_rest) {
        set_error("mm_match: a bounded grid-barrier wait in the round kernel gave up");
        return MM_ERR_DEVICE;
    }
    if (out.status == 1 || out.rounds > c.nseeds) {
        set_error("mm_match: fewer seeds than rounds");
        return MM_ERR_SEEDS;
    }
    *rounds_out = out.rounds;
    return MM_OK;
}

// The counters' and timestamps' device arrays, once a call asks for them.
mm_status run_rounds(Call &c)
{
    PushState *s = c.s;
    if (c.stats) {
        const size_t bytes = sizeof(unsigned long long) * kMaxRounds * MM_STATS_COLS;
        if (!s->stats) MM_CUDA_TRY(dev_alloc((void **)&s->stats, bytes, c.stream), "stats");
        MM_CUDA_TRY(cudaMemsetAsync(s->stats, 0, bytes, c.stream), "stats clear");
    }
    if (c.timing) {
        const size_t bytes = sizeof(unsigned long long) * kStampCount;
        if (!s->tstamp) MM_CUDA_TRY(dev_alloc((void **)&s->tstamp, bytes, c.stream), "timestamps");
        MM_CUDA_TRY(cudaMemsetAsync(s->tstamp, 0, bytes, c.stream), "timestamps clear");
    }
    if (is_weighted(c.type))
        return c.pol ? launch_match<true, false, true>(c)
                     : (c.stats ? launch_match<true, true, false>(c) : launch_match<true, false, false>(c));
    return c.pol ? launch_match<false, false, true>(c)
                 : (c.stats ? launch_match<false, true, false>(c) : launch_match<false, false, false>(c));
}

}  // namespace


namespace {

// Degrees, classes, contiguity, slot offsets (once per graph; for lists that
// tile the arrays the upload's pass over the ranges has done it).
mm_status scan_graph(mm_graph *g, cudaStream_t stream)
{
    const int n = g->n;
    if (n == 0) return MM_OK;
    if (!g->scanned) {
        RangeInfo *d_info = nullptr;
        long long *d_deg = nullptr;
        MM_CUDA_TRY(dev_alloc((void **)&d_info, sizeof(RangeInfo), stream), "prep info");
        cudaError_t e = cudaMemsetAsync(d_info, 0, sizeof(RangeInfo), stream);
        if (e == cudaSuccess) e = dev_alloc((void **)&d_deg, sizeof(long long) * (size_t)n, stream);
        if (e == cudaSuccess) e = scan_ranges(g->d_ranges, n, g->nnz, d_info, d_deg, stream);
        RangeInfo info = {};
        if (e == cudaSuccess) e = cudaMemcpyAsync(&info, d_info, sizeof info, cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
        dev_free(d_info, stream);
        if (e != cudaSuccess) {
            dev_free(d_deg, stream);
            return cuda_fail(e, "prep scan");
        }
        apply_ranges(g, info);
        if (!g->contiguous && g->sum_degree < (1ll << 31) - 1) {
            e = dev_alloc((void **)&g->d_slot_off, sizeof(long long) * (size_t)n, stream);
            void *tmp = nullptr;
            size_t tmp_bytes = 0;
            if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, d_deg, g->d_slot_off, n, stream);
            if (e == cudaSuccess) e = dev_alloc((void **)&tmp, tmp_bytes, stream);
            if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, d_deg, g->d_slot_off, n, stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
            dev_free(tmp, stream);
            if (e != cudaSuccess) {
                dev_free(d_deg, stream);
                dev_free(g->d_slot_off, stream);
                g->d_slot_off = nullptr;
                return cuda_fail(e, "slot offsets");
            }
        }
        dev_free(d_deg, stream);
        g->scanned = true;
    }
    if (g->sum_degree >= (1ll << 31) - 1) {
        set_error("push: more than 2^31 - 2 adjacency slots are not supported");
        return MM_ERR_UNSUPPORTED;
    }
    return MM_OK;
}

// Reverse proposal keys of one weighting (built once per graph).
mm_status build_revkey(mm_graph *g, int weighted, cudaStream_t stream)
{
    const int wi = weighted ? 1 : 0;
    if (g->d_revkey[wi]) return MM_OK;
    const int n = g->n;
    if (n == 0) return MM_OK;
    const long long S = g->sum_degree;

    unsigned long long *revkey = nullptr;
    cudaError_t e = dev_alloc((void **)&revkey, sizeof(unsigned long long) * (size_t)(S > 0 ? S : 1), stream);
    if (e != cudaSuccess) return cuda_fail(e, "reverse keys");
    if (S == 0) {
        g->d_revkey[wi] = revkey;
        return MM_OK;
    }
    // Sorted lists: binary-search build.
    {
        const long long chunks = (S + kRevChunk - 1) / kRevChunk;
        int *chunk_v = nullptr;
        e = dev_alloc((void **)&chunk_v, sizeof(int) * (size_t)(chunks + 2), stream);
        if (e == cudaSuccess) e = cudaMemsetAsync(chunk_v + chunks + 1, 0, sizeof(int), stream);
        if (e == cudaSuccess) e = cudaMemsetAsync(revkey, 0, sizeof(unsigned long long) * (size_t)S, stream);
        if (e == cudaSuccess) {
            k_chunk_owner<<<grid_for(chunks + 1, 256, 148 * 8), 256, 0, stream>>>(
                g->d_ranges, n, g->contiguous ? 1 : 0, g->d_slot_off, S, chunk_v);
            const int grid = grid_for(chunks, 1, 148 * 8);
            if (weighted)
                k_revkey_sorted<true><<<grid, kRevThreads, 0, stream>>>(g->d_ranges, g->d_nbrs, g->d_w,
                                                                        g->contiguous ? 1 : 0, g->d_slot_off, S,
                                                                        chunk_v, revkey, chunk_v + chunks + 1);
            else
                k_revkey_sorted<false><<<grid, kRevThreads, 0, stream>>>(g->d_ranges, g->d_nbrs, g->d_w,
                                                                         g->contiguous ? 1 : 0, g->d_slot_off, S,
                                                                         chunk_v, revkey, chunk_v + chunks + 1);
            e = cudaGetLastError();
        }
        int unsorted = 1;
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(&unsorted, chunk_v + chunks + 1, sizeof(int), cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
        dev_free(chunk_v, stream);
        if (e != cudaSuccess) {
            dev_free(revkey, stream);
            return cuda_fail(e, "reverse key build (sorted lists)");
        }
        if (!unsorted) {
            g->d_revkey[wi] = revkey;
            return MM_OK;
        }
    }

    // General lists: sort the (unordered pair, direction) items.
    const int bits = bits_for(n);
    unsigned long long *k0 = nullptr, *k1 = nullptr;
    int *v0 = nullptr, *v1 = nullptr;
    void *tmp = nullptr;
    size_t tmp_bytes = 0;
    e = dev_alloc((void **)&k0, sizeof(unsigned long long) * S, stream);
    if (e == cudaSuccess) e = dev_alloc((void **)&k1, sizeof(unsigned long long) * S, stream);
    if (e == cudaSuccess) e = dev_alloc((void **)&v0, sizeof(int) * S, stream);
    if (e == cudaSuccess) e = dev_alloc((void **)&v1, sizeof(int) * S, stream);
    if (e == cudaSuccess) {
        k_pair_items<<<grid_for(n * 32ll, 256, 148 * 16), 256, 0, stream>>>(
            g->d_ranges, g->d_nbrs, n, bits, g->contiguous ? 1 : 0, g->d_slot_off, k0, v0);
        e = cudaGetLastError();
    }
    cub::DoubleBuffer<unsigned long long> kb(k0, k1);
    cub::DoubleBuffer<int> vb(v0, v1);
    const int end_bit = 2 * bits + 1;
    if (e == cudaSuccess) e = cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, kb, vb, (int)S, 0, end_bit, stream);
    if (e == cudaSuccess) e = dev_alloc((void **)&tmp, tmp_bytes, stream);
    if (e == cudaSuccess) e = cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, kb, vb, (int)S, 0, end_bit, stream);
    if (e == cudaSuccess) {
        const int grid = grid_for(S, 256, 148 * 16);
        if (weighted)
            k_pair_groups<true><<<grid, 256, 0, stream>>>(kb.Current(), vb.Current(), S, bits, g->d_ranges, g->d_w,
                                                          g->contiguous ? 1 : 0, g->d_slot_off, revkey);
        else
            k_pair_groups<false><<<grid, 256, 0, stream>>>(kb.Current(), vb.Current(), S, bits, g->d_ranges, g->d_w,
                                                           g->contiguous ? 1 : 0, g->d_slot_off, revkey);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    dev_free(tmp, stream);
    dev_free(k0, stream);
    dev_free(k1, stream);
    dev_free(v0, stream);
    dev_free(v1, stream);
    if (e != cudaSuccess) {
        dev_free(revkey, stream);
        return cuda_fail(e, "reverse key build");
    }
    g->d_revkey[wi] = revkey;
    return MM_OK;
}

}  // namespace

cudaError_t scan_ranges(const int2 *ranges, int n, long long nnz, RangeInfo *d_info, long long *deg_out, cudaStream_t stream)
{
    k_scan_ranges<<<grid_for(n, 256, 148 * 8), 256, 0, stream>>>(ranges, n, nnz, d_info, deg_out);
    return cudaGetLastError();
}

void apply_ranges(mm_graph *g, const RangeInfo &info)
{
    g->sum_degree = (long long)info.sum_deg;
    g->max_degree = (long long)info.max_deg;
    g->long_count = (long long)info.long_count;
    g->long_entries = (long long)info.long_entries;
    g->win_groups = (long long)info.win_groups;
    g->win_even = (long long)info.win_even;
    g->contiguous = info.noncontig == 0;
}

// Preference windows of the weighted types, built once per graph in three
// steps so that the upload can build the windows of the lists that have
// arrived while later chunks are still in transfer: windows_begin sizes and
// allocates them (it needs only the ranges), windows_range builds those of
// vertices [va, vb) and queues lists longer than kWinChunk, windows_end builds
// the queued lists and publishes d_pwin.
// Memory comes from and goes back to `mem`: the upload builds on a stream of its
// own and passes the legacy one, as for every other array of a graph.  (Blocks
// that came from two streams were found free or not as the moment had it, and
// the pool then remapped what it had to make room, inside a later call: first
// matchings of R-MAT 2^23 of 9 to 83 ms, for 8.9.)
mm_status windows_begin(mm_graph *g, cudaStream_t stream, cudaStream_t mem)
{
    const int n = g->n;
    // the limit is in entries, window by window rounded up to even; fewer than that
    // many have group numbers of 30 bits, where pwin_off has 31
    if (g->win_even >= (1ll << 31)) {
        set_error("push: more than 2^31 - 1 preference-window slots are not supported");
        return MM_ERR_UNSUPPORTED;
    }
    int2 *win = nullptr;
    int *big = nullptr;  // [n + 1]: queued long lists, then their count
    int *packed = nullptr;
    void *tmp = nullptr;
    const size_t nv = (size_t)n + 1;
    size_t tmp_bytes = 0;
    cudaError_t e = cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, (long long *)nullptr, (long long *)nullptr, n + 1, stream);
    // the groups of every window, their sums and the scan's own memory, at once
    const size_t sums = 2 * sizeof(long long) * nv, all = (sums + 255) / 256 * 256 + tmp_bytes;
    if (e == cudaSuccess) e = dev_alloc((void **)&packed, sizeof(int) * nv, mem);
    if (e == cudaSuccess)
        e = dev_alloc((void **)&win, 4 * sizeof(int2) * (size_t)(g->win_groups > 0 ? g->win_groups : 1), mem);
    if (e == cudaSuccess) e = dev_alloc((void **)&big, sizeof(int) * nv, mem);
    if (e == cudaSuccess) e = dev_alloc(&tmp, all, mem);
    if (e == cudaSuccess && mem != stream) e = cudaStreamSynchronize(mem);
    long long *groups = (long long *)tmp, *off = groups + nv;
    if (e == cudaSuccess) e = cudaMemsetAsync(big + n, 0, sizeof(int), stream);
    if (e == cudaSuccess) {
        k_win_sizes<<<grid_for(n + 1ll, 256, 148 * 8), 256, 0, stream>>>(g->d_ranges, n, groups);
        e = cub::DeviceScan::ExclusiveSum((char *)tmp + (all - tmp_bytes), tmp_bytes, groups, off, n + 1, stream);
    }
    if (e == cudaSuccess) {
        k_win_offsets<<<grid_for(n + 1ll, 256, 148 * 8), 256, 0, stream>>>(g->d_ranges, off, n, packed);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        if (mem != stream) cudaStreamSynchronize(stream);
        dev_free(tmp, mem);
        dev_free(win, mem);
        dev_free(big, mem);
        dev_free(packed, mem);
        return cuda_fail(e, "window buffers");
    }
    g->win_tmp[0] = tmp;
    g->win_tmp_bytes = all;
    g->win_build = win;
    g->win_big = big;
    g->d_pwin_off = packed;
    return MM_OK;
}

mm_status windows_range(mm_graph *g, int va, int vb, cudaStream_t stream)
{
    if (vb <= va) return MM_OK;
    k_win_build<<<grid_for((long long)(vb - va) * 32, 256, 148 * 16), 256, 0, stream>>>(
        g->d_ranges, g->d_nbrs, g->d_w, va, vb, g->d_pwin_off, g->win_build, g->win_big, g->win_big + g->n);
    MM_CUDA_TRY(cudaGetLastError(), "preference windows");
    return MM_OK;
}

mm_status windows_end(mm_graph *g, cudaStream_t stream, cudaStream_t mem)
{
    const int n = g->n;
    int *big = g->win_big;
    int2 *win = g->win_build;
    const int *off = g->d_pwin_off;
    int nbig = 0;
    cudaError_t e = cudaSuccess;
    if (g->max_degree > kWinChunk) {  // else nothing was queued
        e = cudaMemcpyAsync(&nbig, big + n, sizeof(int), cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    }
    // scratch: from what the offsets needed, which is free again, else allocated
    // (after the last copy of an upload an allocation is waited for)
    size_t at = 0;
    int own = 1;
    auto take = [&](void **out, size_t bytes) {
        bytes = (bytes + 255) / 256 * 256;
        if (at + bytes <= g->win_tmp_bytes) {
            *out = (char *)g->win_tmp[0] + at;
            at += bytes;
            return cudaSuccess;
        }
        cudaError_t x = dev_alloc(out, bytes, mem);
        if (x == cudaSuccess) g->win_tmp[own++] = *out;
        if (x == cudaSuccess && mem != stream) x = cudaStreamSynchronize(mem);
        return x;
    };
    if (e == cudaSuccess && nbig > 0) {
        const size_t nb = (size_t)nbig + 1;
        size_t tmp_bytes = 0;
        long long nchunks = 0;
        void *tmp = nullptr;
        WinCand *cand = nullptr;
        e = cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, (long long *)nullptr, (long long *)nullptr, nbig + 1, stream);
        const size_t all = (2 * sizeof(long long) * nb + 255) / 256 * 256 + tmp_bytes;
        if (e == cudaSuccess) e = take(&tmp, all);
        long long *ccnt = (long long *)tmp, *coff = ccnt + nb;
        if (e == cudaSuccess) e = cudaMemsetAsync(ccnt + nbig, 0, sizeof(long long), stream);
        if (e == cudaSuccess) {
            k_win_chunk_counts<<<grid_for(nbig, 256, 148 * 4), 256, 0, stream>>>(g->d_ranges, big, nbig, ccnt);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess)
            e = cub::DeviceScan::ExclusiveSum((char *)tmp + (all - tmp_bytes), tmp_bytes, ccnt, coff, nbig + 1, stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(&nchunks, coff + nbig, sizeof nchunks, cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
        if (e == cudaSuccess) e = take((void **)&cand, sizeof(WinCand) * 32 * (size_t)(nchunks > 0 ? nchunks : 1));
        if (e == cudaSuccess) {
            k_win_chunks<<<grid_for(nchunks * 32, 256, 148 * 16), 256, 0, stream>>>(g->d_ranges, g->d_nbrs, g->d_w, big,
                                                                                  nbig, coff, cand);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) {
            k_win_chunk_merge<<<grid_for((long long)nbig * 32, 256, 148 * 16), 256, 0, stream>>>(
                g->d_ranges, big, nbig, coff, cand, off, win);
            e = cudaGetLastError();
        }
    }
    if (e != cudaSuccess) {
        if (mem != stream) cudaStreamSynchronize(stream);
        windows_discard(g);
        return cuda_fail(e, "preference windows");
    }
    if (mem == stream) windows_settle(g, mem);
    g->d_pwin = win;
    g->pwin_weights = false;
    g->win_build = nullptr;
    return MM_OK;
}

namespace {

// Symmetric weighted path: a window entry's second word becomes the entry's
// weight, so a proposal needs no dependent load of it (the proposal key is the
// weight and the proposer's id).  An entry flagged as never chosen keeps a
// weight that fails the same test (<= -1 or NaN).
// Eight lanes a window: a list's weights lie together (a thread a window took
// R-MAT 2^20 0.13 ms).
__global__ void __launch_bounds__(256) k_win_weights(const float *w, const int *pwin_off, int2 *pwin, int n)
{
    const int l = threadIdx.x & 7;
    const long long stride = (long long)gridDim.x * blockDim.x / 8;
    for (long long v = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / 8; v < n; v += stride) {
        const int g0 = pwin_off[v] & 0x7fffffff, g1 = pwin_off[v + 1] & 0x7fffffff;
        for (long long e = 4ll * g0 + l; e < 4ll * g1; e += 8) {
            int2 x = pwin[e];
            if (x.x < 0) continue;  // a filler
            x.y = __float_as_int(__ldg(w + (x.y & 0x7fffffff)));
            pwin[e] = x;
        }
    }
}

}  // namespace

// Free what a build needed besides the windows, on `mem` (after windows_end; on
// another stream than the build's once that has been waited for).
void windows_settle(mm_graph *g, cudaStream_t mem)
{
    for (void *&x : g->win_tmp) {
        dev_free(x, mem);
        x = nullptr;
    }
    dev_free(g->win_big, mem);
    g->win_big = nullptr;
}

void windows_discard(mm_graph *g)
{
    windows_settle(g, 0);
    dev_free(g->win_build, 0);
    if (!g->d_pwin) {
        dev_free(g->d_pwin_off, 0);
        g->d_pwin_off = nullptr;
    }
    g->win_build = nullptr;
}

namespace {

mm_status build_windows(mm_graph *g, cudaStream_t stream)
{
    mm_status st = windows_begin(g, stream, stream);
    if (st == MM_OK) st = windows_range(g, 0, g->n, stream);
    if (st == MM_OK) st = windows_end(g, stream, stream);
    return st;
}

}  // namespace

mm_status push_prepare(mm_graph *g, int weighted, cudaStream_t stream)
{
    // the symmetric path computes each proposal's key: no reverse index
    const bool sym = weighted ? g->sym_weights : g->sym_struct;
    mm_status st = scan_graph(g, stream);
    if (st == MM_OK && !sym) st = build_revkey(g, weighted, stream);
    if (st == MM_OK && weighted && g->n > 0 && !g->d_pwin) st = build_windows(g, stream);
    if (st == MM_OK && weighted && g->d_pwin && g->sym_weights && !g->pwin_weights) {
        k_win_weights<<<grid_for(g->n * 8ll, 256, 148 * 8), 256, 0, stream>>>(g->d_w, g->d_pwin_off, g->d_pwin, g->n);
        MM_CUDA_TRY(cudaGetLastError(), "window weights");
        g->pwin_weights = true;
    }
    return st;
}

mm_status push_match(mm_graph *g, int type, uint32_t barrier, const uint32_t *seeds, int nseeds, int *d_match,
                     int *rounds_out, long long *stats, int stats_rounds, cudaStream_t stream)
{
    const bool maximal = is_maximal(type);
    if (g->n == 0) {
        // The reference still runs (and draws a seed for) its first round.
        *rounds_out = maximal ? 1 : max_rounds_of(type);
        if (nseeds < *rounds_out) {
            set_error("mm_match: fewer seeds than rounds");
            return MM_ERR_SEEDS;
        }
        return MM_OK;
    }
    Call c{g, nullptr, type, barrier, seeds, nseeds, d_match, stats != nullptr, false, nullptr, stream};
    mm_status st = begin_call(c);
    if (st == MM_OK) st = run_rounds(c);
    if (st != MM_OK) return call_failed(c, st);
    return end_call(c, rounds_out, stats, stats_rounds, nullptr);
}

// The round kernel with the learned colouring: each vertex's blue probability
// comes from the policy (MM_POLICY_FLOATS weights, host) instead of the select
// barrier.  trace (device, trace_rounds * n * 8 floats, or null) receives the
// features, colour and outcome of every vertex coloured in those rounds.
mm_status push_match_policy(mm_graph *g, int type, uint32_t barrier, const uint32_t *seeds, int nseeds,
                            const float *mlp_host, float level, int *d_match, int *rounds_out, float *trace,
                            int trace_rounds, cudaStream_t stream)
{
    if (g->n == 0) return push_match(g, type, barrier, seeds, nseeds, d_match, rounds_out, nullptr, 0, stream);
    Call c{g, nullptr, type, barrier, seeds, nseeds, d_match, false, false, nullptr, stream};
    mm_status st = begin_call(c);
    if (st != MM_OK) return call_failed(c, st);
    PushState *s = c.s;
    if (!s->wfeat) {
        float2 *wfeat = nullptr;
        cudaError_t e = dev_alloc((void **)&wfeat, sizeof(float2) * (size_t)g->n, stream);
        if (e == cudaSuccess) {
            k_wfeat<<<grid_for((long long)g->n * 32, 256, 148 * 16), 256, 0, stream>>>(g->d_ranges, g->d_w, g->n, wfeat);
            e = cudaGetLastError();
        }
        if (e != cudaSuccess) {  // the state's arrays may still be being cleared on this stream
            dev_free(wfeat, stream);
            return call_failed(c, cuda_fail(e, "policy state"));
        }
        s->wfeat = wfeat;
    }
    PolicyArgs pol;
    pol.mlp = mlp_host;
    // the output layer's weights W2 (after W1 and b1): all zero means every
    // vertex gets sigmoid(b2), the same clamp and scaling as on the device
    {
        constexpr int kW2 = kHid * kFeat + kHid;
        bool zero = true;
        for (int j = 0; j < kHid; ++j) zero = zero && mlp_host[kW2 + j] == 0.0f;
        if (zero) {
            float prob = 1.0f / (1.0f + std::exp(-mlp_host[kW2 + kHid]));
            prob = std::fmin(std::fmax(prob, 1.0f / 16.0f), 15.0f / 16.0f);
            pol.constant = true;
            pol.constant_bar = (uint32_t)((double)prob * 4294967296.0);
        }
    }
    pol.level = level;
    pol.trace = trace;
    pol.trace_rounds = trace ? trace_rounds : 0;
    c.pol = &pol;
    st = run_rounds(c);
    if (st != MM_OK) return call_failed(c, st);
    return end_call(c, rounds_out, nullptr, 0, nullptr);
}

// Same launch as push_match with barrier timestamps on: block 0 reads the
// global timer as each grid barrier completes, giving every round's window
// scan (A1), fallback scan (A2) and commit (B) durations.
mm_status push_profile(mm_graph *g, int type, uint32_t barrier, const uint32_t *seeds, int nseeds, int *d_match,
                       int *rounds_out, float *ms_phases, int cap_rounds, int *launched, cudaStream_t stream)
{
    if (g->n == 0) return push_match(g, type, barrier, seeds, nseeds, d_match, rounds_out, nullptr, 0, stream);
    Call c{g, nullptr, type, barrier, seeds, nseeds, d_match, false, true, nullptr, stream};
    mm_status st = begin_call(c);
    if (st == MM_OK) st = run_rounds(c);
    if (st != MM_OK) return call_failed(c, st);
    unsigned long long stamps[kStampCount];
    st = end_call(c, rounds_out, nullptr, 0, stamps);
    if (st != MM_OK) return st;
    if (ms_phases) {
        const int r_exec = *rounds_out;
        for (int r = 0; r < cap_rounds; ++r) {
            float a = 0.f, b = 0.f, c = 0.f;
            if (r < r_exec && stamps[3 * r] && stamps[3 * r + 1] && stamps[3 * r + 2] && stamps[3 * r + 3]) {
                a = (float)((double)(stamps[3 * r + 1] - stamps[3 * r]) * 1e-6);
                b = (float)((double)(stamps[3 * r + 2] - stamps[3 * r + 1]) * 1e-6);
                c = (float)((double)(stamps[3 * r + 3] - stamps[3 * r + 2]) * 1e-6);
            }
            ms_phases[(size_t)r * MM_PROFILE_KERNELS + 0] = a;
            ms_phases[(size_t)r * MM_PROFILE_KERNELS + 1] = b;
            ms_phases[(size_t)r * MM_PROFILE_KERNELS + 2] = c;
            ms_phases[(size_t)r * MM_PROFILE_KERNELS + 3] = a + b + c;
        }
    }
    if (launched) *launched = 1;
    return MM_OK;
}

// Per-graph round counts of the last matching of a batch (after push_match).
mm_status push_batch_rounds(mm_graph *g, int type, int *rounds_host, cudaStream_t stream)
{
    // The reference's loop for a graph runs until a round finds none of its
    // vertices unmatched at the colouring, so it executes its last active round
    // and one more (at most the cap; an empty graph runs one round).
    const int cap = max_rounds_of(type);
    if (!is_maximal(type)) {
        for (int i = 0; i < g->ngraphs; ++i) rounds_host[i] = cap;
        return MM_OK;
    }
    const size_t bytes = sizeof(int) * (size_t)g->ngraphs;
    MM_CUDA_TRY(cudaMemsetAsync(g->d_glast, 0xff, bytes, stream), "batch rounds");
    if (g->n > 0) {
        k_batch_last<<<grid_for(((long long)g->n + kLastSpan - 1) / kLastSpan * 32, 256, 148 * 8), 256, 0, stream>>>(
            g->d_last, g->n, g->d_goff, g->ngraphs, g->d_glast);
        MM_CUDA_TRY(cudaGetLastError(), "batch rounds");
    }
    MM_CUDA_TRY(cudaMemcpyAsync(rounds_host, g->d_glast, bytes, cudaMemcpyDeviceToHost, stream), "batch rounds");
    MM_CUDA_TRY(cudaStreamSynchronize(stream), "batch rounds");
    for (int i = 0; i < g->ngraphs; ++i) rounds_host[i] = rounds_host[i] + 2 < cap ? rounds_host[i] + 2 : cap;
    return MM_OK;
}

void push_release(mm_graph *g)
{
    PushState *s = (PushState *)g->push_exec;
    if (s) {
        free_state(s);
        g->push_exec = nullptr;
    }
    for (int i = 0; i < 2; ++i) {
        dev_free(g->d_revkey[i], 0);
        g->d_revkey[i] = nullptr;
    }
    dev_free(g->d_slot_off, 0);
    g->d_slot_off = nullptr;
    windows_discard(g);
    dev_free(g->d_pwin, 0);
    g->d_pwin = nullptr;
    g->pwin_weights = false;
    dev_free(g->d_pwin_off, 0);
    g->d_pwin_off = nullptr;
}

}  // namespace mm
