// kernels.cu — the rule-evaluation engine for sm_100a.
//
// One persistent kernel serves both phases of every rule.  Blocks pull
// tasks (a plan and a range of roots) from a device queue.  A task is
// evaluated as a depth-first search over *chunks*: the block keeps, for each
// plan level, a bounded frontier of partial bindings in shared memory and
// always extends the deepest level that still has work.  Each frontier item
// carries the neighbour segment of its next step (looked up once, when the
// item is created).  Extending a level lays the segments of up to B items end
// to end (a block-wide prefix sum) and hands the resulting candidates to
// threads one per slot, so a hub with 50,000 neighbours is spread over the
// whole block instead of serialising one thread.  Frontier memory is bounded
// by construction (each round produces at most `cap` items), so any fan-out
// fits.
//
// Outputs:
//  * kExist: roots with at least one complete grounding (a bit per root);
//    support counts head triples, body size with hS == hO counts hS values.
//  * kPairs: distinct (root, hO) pairs for the body size; each root is one
//    hS value, the hO value is replaced by its rank in the value domain of
//    the atom that binds it, and the pairs go into a per-task bitmap in
//    shared memory (or a per-plan bitmap in global memory for very large
//    domains).  Counting is done on insertion (atomicOr returns the old
//    word), so there is no separate popcount pass, and shared bitmaps never
//    touch HBM.  A partial binding whose (root, hO) pair is already present
//    is dropped, which is the reference's early prune
//    (CPU_01_nonparallel/SupportCounting.cpp:284-290).
//
// Block sizes 128, 256 and 512 are instantiated; shared memory scales with
// the block (16 ints of frontier and 32 bitmap words per thread), so 8, 4 or
// 2 blocks stay resident per SM.
//
// What bounds it: 1,024 threads an SM (64 registers, 55 KB of shared memory
// for 256 threads), which fill 48 % of the issue slots; a warp waits for block
// barriers (4.6 cycles per issue), dependent loads (3.6) and fixed latencies
// (3.2), and DRAM is idle (the index lies in L2; 5,000 miner candidates,
// 1.9e9 warp instructions in 3.9 ms).  So a step pays that saves instructions
// or rounds.
//
// The reference's kernels (GPU_03/gpu_kernels.cuh:34-443) run one thread
// per head triple or per first-atom triple with template-unrolled
// recursion; this engine replaces them as a whole.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>

#include "common.hpp"

namespace gr {

namespace cg = cooperative_groups;

// Counts the global-memory bytes the algorithm requests (the roofline's
// algorithmic bytes).  Compiled out of the timed kernel.
template <bool kOn>
struct Meter {
    unsigned long long bytes = 0;
    __device__ __forceinline__ void add(unsigned long long n) {
        if constexpr (kOn) bytes += n;
    }
};

// What a round needs to know of its level, worked out once per task (one
// thread per level) instead of by every thread in every round: in rounds of
// a few dozen candidates that was a third of the instructions.
enum LevelFlag : int {
    kLvLeaf = 1,         // the step is the plan's last
    kLvHo = 2,           // kPairs: the step binds hO (its values' ranks are read)
    kLvHasRank = 4,      // kPairs: the level's items carry hO's rank
    kLvFilters = 8,      // checks or used-triple tests follow the step
    kLvSig = 16,         // the next step expands the value this one binds: its signature is tested
    kLvLook = 32,        // a new item is stored only if its row has a value that can take the step after
    kLvLookHigh = 64,    // ... whose signature bit is in the high word
    kLvScan = 128, kLvSameVar = 256, kLvRowScan = 512,
    kLvTwo = 1024,       // the step binds two values
    kLvWide = 2048,      // rounds may overflow the next level (see `wide`)
    kLvClaims = 4096,    // hub or memo items are claimed (see kHubSeen)
    kLvPath = 13,        // shift of the path kind (0 none, 1 hub, 2 memo, 3 existence, 4 three-step, 5 scan)
};
struct alignas(16) Level {
    const int* vals;             // the step's values, by edge (or row)
    const int* ranks;            // their ranks in hO's domain (kLvHo)
    const uint32_t* sigs;        // their signature words (every second word; kLvSig)
    int flags;
    int len;                     // tuple length of the level's items
    int at, nextAt;              // pool offsets of this level's and the next level's items
    int nextLen;
    int sigShift, lookShift;     // bits of the two signature tests
    int rankBase;                // row scans: the predicate's first row
    int maxTake;                 // candidates of a round
    int pad[3];
};

// What a block does after a group of a task's roots.
enum GroupNext : int { kGroupGoOn, kGroupGive, kGroupLeave };

template <int B>
struct BlockState {
    static constexpr int kWarps = B / 32;
    Level lv[kMaxBody];
    int task;
    int stop;                       // the block's deadline passed: abandon the task
    unsigned long long deadline;    // global-timer ns (0: none)
    int curItem[kMaxBody + 1];      // a level's position, saved when the search descends below it
    int curOff[kMaxBody + 1];
    int count[kMaxBody + 1];
    int firstFail;                  // first candidate of a wide round that found the next level full
    unsigned safeLevels;            // bit l: level l takes capacity-sized rounds until exhausted
    int levelOff[kMaxBody + 1];
    int warpSum[kWarps];
    unsigned long long red[kWarps];
    int exRank[kWarps][kMaxVars];   // per warp: hO-domain ranks of the bound values of a hub item
    int spill;                      // 1: the block gives its open items away
    long long lookAt;               // thread 0: the clock at which it next looks at the queue
    uint32_t* rows;                 // the group's dedup rows, of rowsWords words when in shared memory (else 0)
    int rowsWords;
    int rowsSup;                    // 1: their fused support is still to be counted
    int rootsEnd;                   // end of the task's roots (the group's may lie before it)
    int idle;                       // blocks that were past the queue's end when the group began
    int next;                       // what follows the group (GroupNext): thread 0's one decision for the block
    int base;                       // the level the task's search starts at
    int nTasks;                     // of the launch, and its counter
    const int* queue;
    int spillN[kMaxBody + 1];       // records per level, then their write positions
    int spillAt;                    // first task slot, first record slot
    int spillRec;
    uint32_t* spillRows;
};

template <int B>
struct Smem {
    DevPlan plan;
    BlockState<B> st;
    int wBeg[B];
    int wLen[B];
    int wLoc[B];   // inclusive prefix of wLen within the item's warp
    int pool[Geom::pool_for(B)];   // frontier levels, then the dedup bitmap at plan.bitmapOff
};

template <bool kC>
__device__ __forceinline__ int2 row_lookup(const DevIndex& ix, int pred, int dir, int key, Meter<kC>& mt) {
    if (key < 0) return make_int2(0, 0);
    const uint32_t tag = (uint32_t)pred * 2u + (uint32_t)dir;
    uint32_t i = slot_hash(tag, (uint32_t)key) & ix.hashMask;
    for (uint32_t probe = 0; probe <= ix.hashMask; ++probe) {
        const uint4 s = __ldg(reinterpret_cast<const uint4*>(ix.hash + i));
        mt.add(16);
        if (s.x == kEmptyTag) break;
        if (s.x == tag && s.y == (uint32_t)key) return make_int2((int)s.z, (int)s.w);
        i = (i + 1) & ix.hashMask;
    }
    return make_int2(0, 0);
}

// A row and what its slot says of it.
struct RowHit {
    int2 seg;
    uint2 sig;   // union of the values' signatures
    int rank, hub;
};

template <bool kC>
__device__ __forceinline__ RowHit row_find(const DevIndex& ix, int pred, int dir, int key, Meter<kC>& mt) {
    RowHit h{make_int2(0, 0), make_uint2(0u, 0u), -1, -1};
    if (key < 0) return h;
    const uint32_t tag = (uint32_t)pred * 2u + (uint32_t)dir;
    uint32_t i = slot_hash(tag, (uint32_t)key) & ix.hashMask;
    for (uint32_t probe = 0; probe <= ix.hashMask; ++probe) {
        const uint4* p = reinterpret_cast<const uint4*>(ix.hash + i);
        const uint4 s = __ldg(p), t = __ldg(p + 1);   // one sector
        mt.add(32);
        if (s.x == kEmptyTag) break;
        if (s.x == tag && s.y == (uint32_t)key) {
            h.seg = make_int2((int)s.z, (int)s.w);
            h.sig = make_uint2(t.x, t.y);
            h.rank = (int)t.z;
            h.hub = (int)t.w;
            break;
        }
        i = (i + 1) & ix.hashMask;
    }
    return h;
}

template <bool kC>
__device__ __forceinline__ bool has_edge(const DevIndex& ix, int pred, int dir, int key, int target, Meter<kC>& mt) {
    const int2 r = row_lookup(ix, pred, dir, key, mt);
    int lo = r.x, hi = r.y;
    const int* v = ix.val[dir];
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        mt.add(4);
        if (__ldg(v + mid) < target) lo = mid + 1; else hi = mid;
    }
    if (lo < r.y) mt.add(4);
    return lo < r.y && __ldg(v + lo) == target;
}

// Whether value x occurs in the sorted values v[beg, beg + len).
template <bool kC>
__device__ __forceinline__ bool seg_has(const int* v, int beg, int len, int x, Meter<kC>& mt) {
    int lo = beg, hi = beg + len;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        mt.add(4);
        if (__ldg(v + mid) < x) lo = mid + 1; else hi = mid;
    }
    return lo < beg + len && __ldg(v + lo) == x;
}

template <bool kC, class Val>
__device__ __forceinline__ bool pass_filters(const DevPlan& P, const DevIndex& ix, int lvl, Meter<kC>& mt, Val val) {
    const int cb = P.chkBeg[lvl], cn = P.chkN[lvl];
    for (int c = 0; c < cn; ++c) {
        const DevCheck& C = P.checks[cb + c];
        const int s = val(C.s), o = val(C.o);
        if (!has_edge(ix, C.pred, C.dir, C.dir == 0 ? s : o, C.dir == 0 ? o : s, mt)) return false;
    }
    const int ub = P.usedBeg[lvl], un = P.usedN[lvl];
    for (int u = 0; u < un; ++u) {
        const DevUsed& U = P.used[ub + u];
        if (val(U.sA) == val(U.sB) && val(U.oA) == val(U.oB)) return false;
    }
    return true;
}

// The range step `s` (0-based) enumerates for a binding resolved by `val`.
template <bool kC, class Val>
__device__ __forceinline__ RowHit step_row(const DevPlan& P, const DevIndex& ix, int s, Meter<kC>& mt, Val val) {
    const DevStep& st = P.steps[s];
    if (st.kind == kExpand) {
        RowHit h = row_find(ix, st.pred, st.dir, val(st.keyRef), mt);
        // a free variable's long row: the one edge past the last, whose value is kAnyValue
        if (st.free && h.seg.y - h.seg.x >= P.freeMin) {
            h.seg = make_int2((int)ix.nTriples, (int)ix.nTriples + 1);
            h.hub = -1;
        }
        return h;
    }
    mt.add(8);
    const int* at = (st.kind == kRowScan ? ix.predRow[st.dir] : ix.predEdge[0]) + st.pred;
    return RowHit{make_int2(__ldg(at), __ldg(at + 1)), make_uint2(~0u, ~0u), -1, -1};
}

template <int B>
struct Smem;

// Publishes a window's prefix sums with one barrier: every thread stores
// the inclusive sum of x over its warp's threads up to itself (wLoc) and
// every warp its total (warpSum), so item i's block-wide prefix is the
// totals of the warps before i's warp plus wLoc[i] (WinCursor reads it
// that way).  The barrier also ORs `flag` over the block.
// Warps without any of the window's nw items only take the barrier.
template <int B>
__device__ __forceinline__ bool publish_window(int x, bool flag, Smem<B>& sm, int nw) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp * 32 < nw) {
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += y;
        }
        sm.wLoc[threadIdx.x] = x;
        if (lane == 31) sm.st.warpSum[warp] = x;
    }
    return __syncthreads_or(flag) != 0;
}

// The window's candidate total: the warps' totals summed by shuffles.
// (Up to 256 threads the eight totals are added directly; the two forms
// differ only in the registers the kernel needs around them.)  Only warps
// with items among the window's nw have published theirs.
template <int B>
__device__ __forceinline__ int window_total(const Smem<B>& sm, int nw) {
    if constexpr (B <= 256) {
        int v = 0;
#pragma unroll
        for (int w = 0; w < B / 32; ++w)
            if (w * 32 < nw) v += sm.st.warpSum[w];
        return v;
    } else {
        const int lane = threadIdx.x & 31;
        int v = lane * 32 < nw ? sm.st.warpSum[lane] : 0;
#pragma unroll
        for (int d = 16; d; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
        return v;
    }
}

// The window item that holds candidate j, for j that never decreases:
// whole warps are stepped over by their totals, then the item is searched
// among its warp's 32 prefixes, starting after the previous item (a hub's
// long segment costs one probe per candidate).
template <int B>
struct WinCursor {
    int item = 0, warp = 0;
    int base = 0;   // candidates of the warps before `warp`
    __device__ __forceinline__ void seek(const Smem<B>& sm, int nw, int j) {
        if (base + sm.wLoc[item] > j) return;
        int end = base + sm.st.warpSum[warp];
        while (end <= j) {
            base = end;
            ++warp;
            end = base + sm.st.warpSum[warp];
        }
        int lo = max(item + 1, warp * 32), hi = min(nw, warp * 32 + 32) - 1;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (base + sm.wLoc[mid] > j) hi = mid; else lo = mid + 1;
        }
        item = lo;
    }
    // index of the item's first candidate
    __device__ __forceinline__ int first(const Smem<B>& sm) const { return base + sm.wLoc[item] - sm.wLen[item]; }
};

template <int B>
__device__ __forceinline__ unsigned long long block_sum(unsigned long long x, BlockState<B>& st) {
    constexpr int kWarps = B / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int d = 16; d; d >>= 1) x += __shfl_down_sync(0xffffffffu, x, d);
    if (lane == 0) st.red[warp] = x;
    __syncthreads();
    unsigned long long t = 0;
    if (threadIdx.x == 0)
        for (int w = 0; w < kWarps; ++w) t += st.red[w];
    return t;  // valid in thread 0
}

// List capacity of a three-step memo item's exceptions (plus one slot for
// the root's own rank) in the warp's kMaxVars-int buffer.
constexpr int kMemo3List = kMaxVars - 1;

// Three-step suffix memos, for body-size plans hS -> x -> v2 -> v3 -> hO
// (memoSteps == 3) at an item (a, x) whose x is a memoised hub row.  The
// memo of x holds S1 = {h : C(h) > 0} and C(h), the number of paths
// x -> v2 -> v3 -> h with x, v2, v3, h distinct, as a byte that saturates
// at 255.  The item's pairs are the h != a with a path that also avoids a,
// i.e. with C(h) > C_a(h), C_a(h) the paths through a:
//   a = v2 (when a is a neighbour of x): v3 in N2(a) \ {x, a, h}, h in N3(v3);
//   a = v3: v2 in N1(x) with a in N2(v2), v2 not in {x, a, h}, and h in N3(a).
// Only h reached that way (listed, at most kMemo3List by the check in
// classify_item) can have C_a(h) > 0; every other bit of S1 stands.  The
// same check bounds C_a(h) by kMemo3List + 64 < 255 (at most one path per
// v3 in N2(a), and per v2 in a's reverse row), so a saturated count still
// compares exactly.
// memo3_exceptions lists the ranks to clear from S1 and memo_item applies
// them.  Its parts are small leaf functions called one after the other, so
// that few of the caller's registers need to be free for them.
//
// memo3_count (whole warp): 2 * K + [a in N1(x)], K = #{v2 in N1(x) : a in
// N2(v2), v2 not in {x, a}} (lanes split a's reverse row under step 2).
template <bool kC>
__device__ __noinline__ int memo3_count(const DevPlan& P, const DevIndex& ix, const int* par, int lenK, int lane,
                                        Meter<kC>& mt) {
    const int p2 = P.steps[2].pred, d2 = P.steps[2].dir;
    const int* v1 = ix.val[P.steps[1].dir];
    const int a = par[kTupleHead], x = par[kTupleHead + 1];
    const int segBeg = par[lenK], segLen = par[lenK + 1];   // x's row under step 1
    const int2 rInv = row_lookup(ix, p2, 1 - d2, a, mt);
    int k = 0;
    for (int e = rInv.x + lane; e < rInv.y; e += 32) {
        const int u = __ldg(ix.val[1 - d2] + e);
        mt.add(4);
        if (u != x && u != a && seg_has(v1, segBeg, segLen, u, mt)) ++k;
    }
    return 2 * __reduce_add_sync(0xffffffffu, k) + (seg_has(v1, segBeg, segLen, a, mt) ? 1 : 0);
}

// memo3_list (one lane): the ranks of the h a path through a reaches, into
// ex[0..n) (repeats allowed), and a's own rank (h != a) into ex[n] (-1 when
// a is outside hO's domain); returns n.
template <bool kC>
__device__ __noinline__ int memo3_list(const DevPlan& P, const DevIndex& ix, const int* par, int kv, int* ex,
                                       Meter<kC>& mt) {
    const int p2 = P.steps[2].pred, d2 = P.steps[2].dir;
    const int p3 = P.steps[3].pred, d3 = P.steps[3].dir;
    const int a = par[kTupleHead], x = par[kTupleHead + 1];
    int n = 0;
    if (kv & 1) {
        const int2 r2a = row_lookup(ix, p2, d2, a, mt);
        for (int e2 = r2a.x; e2 < r2a.y; ++e2) {
            const int v3 = __ldg(ix.val[d2] + e2);
            if (v3 == x || v3 == a) continue;
            const int2 r3 = row_lookup(ix, p3, d3, v3, mt);
            for (int e3 = r3.x; e3 < r3.y && n < kMemo3List; ++e3) {
                const int h = __ldg(ix.val[d3] + e3);
                if (h != x && h != a && h != v3) ex[n++] = __ldg(ix.valRank[d3] + e3);
            }
        }
    }
    const int2 r3a = row_lookup(ix, p3, d3, a, mt);
    for (int e3 = r3a.x; e3 < r3a.y && n < kMemo3List; ++e3) {
        const int h = __ldg(ix.val[d3] + e3);
        if (h != x && h != a) ex[n++] = __ldg(ix.valRank[d3] + e3);
    }
    ex[n] = row_find(ix, p3, 1 - d3, a, mt).rank;
    return n;
}

// memo3_keep (one lane per listed rank r): whether a path avoiding a still
// reaches r's value h, i.e. C(h) > C_a(h).
template <bool kC>
__device__ __noinline__ bool memo3_keep(const DevPlan& P, const DevIndex& ix, const int* par, int lenK, int r,
                                        int kv, const uint32_t* C, Meter<kC>& mt) {
    const unsigned c = (__ldg(C + (r >> 2)) >> ((r & 3) * 8)) & 0xffu;   // saturates at 255
    mt.add(4);
    const int p3 = P.steps[3].pred, d3 = P.steps[3].dir;
    const int a = par[kTupleHead];
    const int h = __ldg(ix.rowKey[1 - d3] + __ldg(ix.predRow[1 - d3] + p3) + r);
    unsigned ca = 0;
    if (has_edge(ix, p3, d3, a, h, mt)) {   // paths with v3 = a
        const int p2 = P.steps[2].pred, d2 = P.steps[2].dir;
        const bool hIsV2 = has_edge(ix, p2, 1 - d2, a, h, mt) &&
                           seg_has(ix.val[P.steps[1].dir], par[lenK], par[lenK + 1], h, mt);
        ca = (unsigned)((kv >> 1) - (hIsV2 ? 1 : 0));
    }
    if (kv & 1) {   // paths with v2 = a
        const int p2 = P.steps[2].pred, d2 = P.steps[2].dir;
        const int x = par[kTupleHead + 1];
        const int2 r2a = row_lookup(ix, p2, d2, a, mt);
        for (int e2 = r2a.x; e2 < r2a.y && ca < c; ++e2) {
            const int v3 = __ldg(ix.val[d2] + e2);
            if (v3 != x && v3 != a && v3 != h && has_edge(ix, p3, d3, v3, h, mt)) ++ca;
        }
    }
    return c > ca;
}

// The exceptions of an item (whole warp): ex[0..n] holds the ranks to clear
// from S1 of memo slot `slot` (-1: none); returns n + 1.
template <bool kC>
__device__ __forceinline__ int memo3_exceptions(const DevPlan& P, const DevIndex& ix, const int* par, int lenK,
                                                int slot, int words, int* ex, int lane, Meter<kC>& mt) {
    const int kv = memo3_count(P, ix, par, lenK, lane, mt);
    int n = 0;
    if (lane == 0) n = memo3_list(P, ix, par, kv, ex, mt);
    n = __shfl_sync(0xffffffffu, n, 0);
    __syncwarp();
    if (lane < n) {
        const uint32_t* C = P.memo3Bits + (long long)slot * ((long long)words + ((P.wo + 3) >> 2)) + words;
        if (memo3_keep(P, ix, par, lenK, ex[lane], kv, C, mt)) ex[lane] = -1;   // still reached: keep its bit
    }
    __syncwarp();
    return n + 1;
}

// The variable whose row a memo item expands (-1: a constant's row; plans
// whose constant is its own neighbour get no memo).
__device__ __forceinline__ int memo_row_value(const DevStep& stA, const int* it) {
    return stA.keyRef >= kTupleHead ? it[stA.keyRef] : -1;
}

// One level-k item whose first suffix step expands a hub row x with a memo:
// for the plan suffix x -[stA]-> y -[stB]-> hO, the memo holds, over hO's
// rank domain, S1 = {h : at least one y in N1(x), y != x, with h in N2(y),
// h != y} and S2, S3 = {h : at least two, three such y}.  The item's valid hO are S1 minus the
// ranks of its bound values (injectivity on hO) minus the h left without a
// witness when bound values are witnesses themselves (u in N1(x), injectivity
// on y): with one such u, the h in N2(u) outside S2; with two, also the h in
// both N2(u)s outside S3.  Ranks within a row ascend with the values, so each
// lane merges its own run of words with the N2(u)s' sorted ranks.  The whole
// warp calls this; new pair bits are counted on insertion and returned (per
// lane).  Steps come by value and counts go back as the result, so that the
// caller's loop state never needs an address.
// Scan items (plans with a scanLevel: hO from the rows of (p, d), then only a
// free value behind it) are the same with every value in the place of N1(x):
// h = hO, its row's values as witnesses, and stB the step (p, 1 - d) from a
// witness to its h.
template <bool kC>
__device__ __noinline__ unsigned long long memo_item(const DevPlan& P, const DevIndex& ix, const DevStep stA,
                                                     const DevStep stB, const int* par, int lenK, int slot,
                                                     uint32_t* dst, int words, int* ex, int lane, Meter<kC>& mt,
                                                     bool sharedDst, int nEx3, bool scan) {
    unsigned long long myNew = 0;
    const bool three = nEx3 > 0;
    const uint32_t* S1 = scan ? P.scanBits
                              : (three ? P.memo3Bits + (long long)slot * ((long long)words + ((P.wo + 3) >> 2))
                                       : P.memoBits + (long long)slot * ((long long)kMemoMaps * words));
    int nEx = lenK - kTupleHead;
    unsigned wmask = 0;
    if (three) {
        nEx = nEx3;
    } else {
        const int exDir = 1 - stB.dir;
        const int segBeg = par[lenK], segLen = par[lenK + 1];
        bool isW = false;
        if (lane < nEx) {
            const int u = par[kTupleHead + lane];
            ex[lane] = row_find(ix, stB.pred, exDir, u, mt).rank;
            if (scan) {   // every bound value may be the free value of some row
                const int2 w = row_lookup(ix, stB.pred, stB.dir, u, mt);
                isW = w.y > w.x;
            } else {
                isW = u != memo_row_value(stA, par) && seg_has(ix.val[stA.dir], segBeg, segLen, u, mt);
            }
        }
        wmask = __ballot_sync(0xffffffffu, isW);
        __syncwarp();
    }
    // the witnesses' rows (the second is empty for most items)
    int e[2] = {0, 0}, e1[2] = {0, 0};
    const int* rk = ix.valRank[stB.dir];
    const int per = (words + 31) >> 5;
    const int wb = min(words, lane * per), we = min(words, wb + per);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        if (!wmask) break;
        const int2 r = row_lookup(ix, stB.pred, stB.dir, par[kTupleHead + __ffs(wmask) - 1], mt);
        wmask &= wmask - 1;
        e[k] = r.x;
        e1[k] = r.y;
        if (r.y > r.x && wb < we) {
            int lo = r.x, hi = r.y;
            const int key = wb << 5;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                mt.add(4);
                if (__ldg(rk + mid) < key) lo = mid + 1; else hi = mid;
            }
            e[k] = lo;
        }
    }
    const uint32_t* S2 = S1 + words;
    for (int w = wb; w < we; ++w) {
        uint32_t m = __ldg(S1 + w);
        mt.add(4);
        for (int q = 0; q < nEx; ++q)
            if (ex[q] >= 0 && (ex[q] >> 5) == w) m &= ~(1u << (ex[q] & 31));
        uint32_t hit[2] = {0u, 0u};
        const int lim = (w + 1) << 5;
#pragma unroll
        for (int k = 0; k < 2; ++k)
            while (e[k] < e1[k]) {
                const int r = __ldg(rk + e[k]);
                if (r >= lim) break;
                hit[k] |= 1u << (r & 31);
                ++e[k];
                mt.add(4);
            }
        if (hit[0] | hit[1]) {
            m &= ~((hit[0] | hit[1]) & ~__ldg(S2 + w));
            mt.add(4);
            if (hit[0] & hit[1]) { m &= ~(hit[0] & hit[1] & ~__ldg(S2 + words + w)); mt.add(4); }
        }
        if (m && !sharedDst) m &= ~__ldcg(dst + w);
        if (m) {
            const uint32_t old = atomicOr(dst + w, m);
            if (!sharedDst) mt.add(8);
            myNew += (unsigned long long)__popc(m & ~old);
        }
    }
    __syncwarp();
    return myNew;
}

// kExist counterpart of memo_item: the item's last step expands a hub row x
// with a memo and its only remaining test is the check (h, y) for a bound
// variable h.  A valid y exists iff h has a witness y in N1(x) other than
// the bound values: with n bound values among h's witnesses that is the bit
// of h in the n-th map after S1; beyond the last map the item is left to
// enumeration.
// Returns 1 (a grounding exists), 0 (none) or -1 (undecided).
template <bool kC>
__device__ __noinline__ int memo_exists(const DevPlan& P, const DevIndex& ix, const DevStep stA, const int* it,
                                        int lenK, int segBeg, int segLen, int slot, Meter<kC>& mt) {
    const int h = it[P.memoH];
    const int dDom = 1 - P.memoD2;
    const int rank = row_find(ix, P.memoP2, dDom, h, mt).rank;
    if (rank < 0) return 0;   // no y reaches h at all
    const int x = memo_row_value(stA, it);
    int nRem = 0;
    for (int q = kTupleHead; q < lenK; ++q) {
        const int u = it[q];
        if (u == h || u == x || !seg_has(ix.val[stA.dir], segBeg, segLen, u, mt)) continue;
        if (!has_edge(ix, P.memoP2, P.memoD2, u, h, mt)) continue;
        if (++nRem >= kMemoMaps) return -1;
    }
    const uint32_t* S = P.memoBits + ((long long)slot * kMemoMaps + nRem) * P.memoWords;
    mt.add(4);
    return (int)((__ldg(S + (rank >> 5)) >> (rank & 31)) & 1u);
}

// Whether an item (a, x) of a three-step memo plan is answered by its memo:
// the paths through a must reach at most kMemo3List values (the warp's
// list) and a's reverse row under the second step must be short.
template <bool kC>
__device__ __forceinline__ bool memo3_fits(const DevPlan& P, const DevIndex& ix, int a, int x, Meter<kC>& mt) {
    const DevStep s2 = P.steps[2], s3 = P.steps[3];
    const int2 rInv = row_lookup(ix, s2.pred, 1 - s2.dir, a, mt);
    if (rInv.y - rInv.x > 64) return false;
    const int2 r2 = row_lookup(ix, s2.pred, s2.dir, a, mt);
    if (r2.y - r2.x > kMemo3List) return false;
    const int2 r3a = row_lookup(ix, s3.pred, s3.dir, a, mt);
    int reach = r3a.y - r3a.x;
    for (int e2 = r2.x; e2 < r2.y && reach <= kMemo3List; ++e2) {
        const int v3 = __ldg(ix.val[s2.dir] + e2);
        if (v3 == x) continue;   // (its row is a hub's, and no path through a takes it)
        const int2 r3 = row_lookup(ix, s3.pred, s3.dir, v3, mt);
        reach += r3.y - r3.x;
    }
    return reach <= kMemo3List;
}

// Items of a round that may skip enumeration, kept out of line so that the
// main loop's registers stay free.  The item's segment is hub row `hub` (kind
// 5: none).  kind 2: an item at the memo level whose row has a memo and at
// most two bound values among its neighbours (returns the memo slot); 3: a
// kExist leaf item decided by the existence memo (returns -3, its found bit
// set; -4 when the bit is new and the task counts on insertion); 4: as 2 for
// the three-step memo of level 1; 5: an item of the scan level, for the scan
// memo (returns 0).  -1: enumerate as usual.
template <bool kC>
__device__ __noinline__ int classify_item(const DevPlan& P, const DevIndex& ix, const DevStep stp, const int* it,
                                          int lenK, int kind, int segBeg, int segLen, uint32_t* fb, bool heavy, int hub,
                                          Meter<kC>& mt) {
    if (kind == 5) {
        int nR = 0;   // bound values that are some row's free value
        for (int q = kTupleHead; q < lenK; ++q) {
            const int2 r = row_lookup(ix, stp.pred, 1 - stp.dir, it[q], mt);
            nR += r.y > r.x ? 1 : 0;
        }
        return nR <= 2 ? 0 : -1;
    }
    const int slot = __ldg((kind == 4 ? P.memo3Tab : P.memoTab) + hub);
    mt.add(4);
    if (slot < 0) return -1;
    if (kind == 4) return memo3_fits(P, ix, it[kTupleHead], it[kTupleHead + 1], mt) ? slot : -1;
    if (kind == 2) {
        // bound values that are also first-step neighbours are witnesses the
        // memo must not count (x itself never is one); up to two are
        // corrected exactly, more enumerate
        const int x = memo_row_value(stp, it);
        int nR = 0;
        for (int q = kTupleHead; q < lenK && nR < 3; ++q)
            nR += it[q] != x && seg_has(ix.val[stp.dir], segBeg, segLen, it[q], mt) ? 1 : 0;
        return nR <= 2 ? slot : -1;
    }
    const int res = memo_exists(P, ix, stp, it, lenK, segBeg, segLen, slot, mt);
    if (res < 0) return -1;
    if (res == 1) {
        const int root = it[0];
        const uint32_t mask = 1u << (root & 31);
        const uint32_t old = atomicOr(&fb[root >> 5], mask);
        if (heavy) {
            mt.add(8);
            if (!(old & mask)) return -4;
        }
    }
    return -3;
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Sort mode: appends the pair key of (row, rank) to the plan's key buffer.
// The threads that emit together take consecutive slots with one atomic; the
// cursor keeps counting past the capacity, so the host learns the exact
// number of keys when they did not fit (and runs again with that size).
__device__ __forceinline__ void emit_pair(const DevPlan& P, long long row, int rank) {
    const unsigned long long key = P.keyBase | ((unsigned long long)row << P.rankBits) | (unsigned)rank;
    cg::coalesced_group g = cg::coalesced_threads();
    unsigned long long base = 0;
    if (g.thread_rank() == 0) base = atomicAdd(P.keyCursor, (unsigned long long)g.size());
    base = g.shfl(base, 0);
    const unsigned long long slot = base + g.thread_rank();
    if (slot < P.keyCap) P.pairKeys[slot] = key;
}

// Claims a hub item of (root, hub) with middle value `mid` in the task's
// table (see kHubSeen); false when `need` other middle values are claimed
// already.
__device__ __forceinline__ bool hub_claim(unsigned long long* seen, int root, int hub, int mid, unsigned need) {
    const unsigned long long key = ((unsigned long long)root << 20) | (unsigned long long)hub;   // 30 bits
    unsigned long long* w = seen + (((uint32_t)key * 0x9E3779B1u) >> (32 - kHubSeenBits));
    const unsigned h = ((uint32_t)mid * 0x85EBCA6Bu) >> 16;
    unsigned long long old = __ldcg(w);
    for (int t = 0; t < 8; ++t) {
        unsigned long long want;
        const unsigned state = (unsigned)(old >> 32) & 3u;
        if ((old >> 34) == key && state != 0u) {
            if (state >= need) return false;
            const unsigned h1 = (unsigned)old & 0xffffu, h2 = (unsigned)(old >> 16) & 0xffffu;
            if (h == h1 || (state == 2u && h == h2)) return true;   // a claimed value again (or its hash)
            want = (old & ~(3ull << 32)) | ((unsigned long long)(state + 1u) << 32);
            if (state == 1u) want |= (unsigned long long)h << 16;
        } else {
            want = (key << 34) | (1ull << 32) | h;   // displaces another pair: it may repeat items, never lose one
        }
        const unsigned long long prev = atomicCAS(w, old, want);
        if (prev == old) return true;
        old = prev;
    }
    return true;
}

// The claims of a round's hub or memo items [0, cut) (items at `items`,
// `stride` ints apart): items that add nothing get wBeg -1.  Out of line,
// so that the caller's loop keeps its registers.
__device__ __noinline__ void hub_claims(unsigned long long* seen, const int* items, int stride, int cut, int midAt,
                                        int* wBeg, int nThreads, unsigned need) {
    for (int i = threadIdx.x; i < cut; i += nThreads) {
        const int wb = wBeg[i];
        if (wb <= -2) {
            const int* it = items + i * stride;
            if (!hub_claim(seen, it[0], -2 - wb, it[midAt], need)) wBeg[i] = -1;
        }
    }
}

// Fused support (plans with supN > 0): the head triples (hS, supPred[j],
// b), b != hS, of rule j whose pair (hS, b) is set in the plan's row of
// root i (rows at bm + i * rowWords for the roots rootBeg + i, i < G); with
// supDir 1 the roots are the objects of the head triples.
// Warps take the roots, lanes a root's head triples; returns this lane's
// count.  Out of line and small: it runs once per task, after the search.
// `part` of `nParts` takes every nParts-th group of 32 head triples.
template <bool kC>
__device__ __noinline__ unsigned long long fused_support(const DevPlan& P, const DevIndex& ix, int j, int rootBeg,
                                                         int G, const uint32_t* bm, int warp, int nWarps, int lane,
                                                         int part, int nParts, Meter<kC>& mt) {
    unsigned long long n = 0;
    const int hp = P.supPred[j], dp = P.supDomPred, dd = P.supDomDir;
    for (int i = warp; i < G; i += nWarps) {
        const int a = __ldg(ix.rowKey[P.rootDir] + rootBeg + i);
        mt.add(4);
        const int2 hr = row_lookup(ix, hp, P.supDir, a, mt);
        const uint32_t* row = bm + (long long)i * P.rowWords;
        for (int e = hr.x + 32 * part + lane; e < hr.y; e += 32 * nParts) {
            const int b = __ldg(ix.val[P.supDir] + e);
            mt.add(4);
            if (b == a) continue;
            const int rank = row_find(ix, dp, dd, b, mt).rank;
            if (rank < 0) continue;   // b never binds hO
            mt.add(4);
            if ((row[rank >> 5] >> (rank & 31)) & 1u) ++n;
        }
    }
    return n;
}

// Takes nTask task and nRec record slots of a list (one thread); false when
// it is full.  `at` gets the first slots, tasks << 32 | records.
__device__ __forceinline__ bool spill_take(unsigned long long* used, unsigned nTask, unsigned nRec,
                                           unsigned long long& at) {
    at = *reinterpret_cast<volatile unsigned long long*>(used);
    for (;;) {
        const unsigned t0 = (unsigned)(at >> 32), r0 = (unsigned)at;
        if (t0 + nTask > (unsigned)kSpillTasks || r0 + nRec > (unsigned)kSpillRecs) return false;
        const unsigned long long seen = atomicCAS(used, at, (unsigned long long)(t0 + nTask) << 32 | (r0 + nRec));
        if (seen == at) return true;
        at = seen;
    }
}

// Gives the roots [beg, end) of a task away, a task per group; false when the
// list is full.  The whole block calls this between two groups.
template <int B>
__device__ __noinline__ bool spill_groups(Smem<B>& sm, const SpillArgs& sp, int plan, int beg, int end) {
    BlockState<B>& S = sm.st;
    const int g = max(1, sm.plan.groupMax);
    if (threadIdx.x == 0) {
        unsigned long long at = 0;
        S.spill = spill_take(&sp.ctl->used[sp.out], (unsigned)((end - beg + g - 1) / g), 0u, at) ? 1 : 0;
        S.spillAt = (int)(at >> 32);
    }
    __syncthreads();
    if (!S.spill) return false;
    for (int b = beg + (int)threadIdx.x * g, j = S.spillAt + (int)threadIdx.x; b < end; b += B * g, j += B)
        sp.tasks[sp.out & 1][j] = SpillTask{plan, -1, 0, 0, b, min(g, end - b), nullptr};
    return true;
}

// What an item's rank slot holds before hO is bound: not looked at yet, with
// hub index h (-1 - h) or with a scanned range (kItemNew); enumerated as
// usual; nothing left to do; or kItemHub + the hub index (leaf items) or memo
// slot of an item that the hub or memo pass takes.
constexpr int kItemNew = 0, kItemEnum = 1, kItemDone = 2, kItemHub = 3;
__device__ __forceinline__ int item_state(const DevStep& next, int hub) {
    return next.kind != kExpand ? kItemNew : (hub >= 0 ? -1 - hub : kItemEnum);
}

// Clock cycles (about 32 us) between a block's looks at the task queue during
// a group of roots: shorter groups are not worth the records (first look after
// 100, 200 and 500 us: 10,000 rules 5.54 -> 5.66, 5.83 and 6.39 ms, of the
// biomedical sets one 1.25 -> 1.01-1.34 ms, others 1.59 -> 1.54-2.19 ms).  A
// sixteenth of the launch idle is enough (5,000 miner candidates 3.99 ms; a
// quarter on two looks 4.60 ms, an eighth on two 4.59 ms).
constexpr long long kSpillEvery = 64000;
// Records of a spill task, and candidates of a record, at inner levels and at
// the leaf: about a round's work each.
constexpr int kSpillChunk = 8, kSpillChunkLeaf = 32;
constexpr int kSpillSeg = 256, kSpillSegLeaf = 8192;

// Gives the open items of levels S.base..k away (see SpillTask), and the
// groups of roots behind them; false when a list is full (the block then
// carries on).  Rows in shared memory move to global ones.  The whole block
// calls this between two rounds; level k continues at item w0, `off`
// candidates of it consumed.  Out of line: it runs at most once per group.
template <int B>
__device__ __noinline__ bool spill_items(Smem<B>& sm, const DevTask& task, const SpillArgs& sp, int k, int w0,
                                         int off) {
    const DevPlan& P = sm.plan;
    BlockState<B>& S = sm.st;
    const int tid = threadIdx.x;
    uint32_t* const rows = S.rows;
    const int nWords = S.rowsWords, kBase = S.base, rootsEnd = S.rootsEnd;
    const bool shared = nWords > 0, sup = S.rowsSup != 0;
    // a level's first open item and the candidates of it already consumed
    auto level_pos = [&](int l, int& at, int& skip) {
        at = l == k ? w0 : S.curItem[l];
        skip = l == k ? off : S.curOff[l];
    };
    // records an item takes: none when nothing is left of it, one when a memo
    // or hub row answers it, else its segment in pieces
    auto pieces = [&](int l, const int* it, int skip) {
        const int lenL = P.tupleLen[l];
        const bool hasRank = P.mode == kPairs && P.hoLevel >= 1 && l >= P.hoLevel;
        const int left = it[lenL + 1] - skip;
        if (left <= 0 || (!hasRank && it[1] == kItemDone)) return 0;
        if (!hasRank && it[1] >= kItemHub) return 1;
        // (not classified yet at a level that may: whole, or its row would not be known as a hub's)
        if (!hasRank && it[1] <= kItemNew &&
            (l + 1 == P.m || l + 1 == P.memoLevel || l + 1 == P.scanLevel || (l == 1 && P.memo3Tab)))
            return 1;
        const int seg = l + 1 == P.m ? kSpillSegLeaf : kSpillSeg;
        return (left + seg - 1) / seg;
    };
    for (int l = tid; l <= kMaxBody; l += B) S.spillN[l] = 0;
    __syncthreads();
    for (int l = kBase; l <= k; ++l) {
        int at, skip;
        level_pos(l, at, skip);
        const int cnt = min(S.count[l], P.cap), stride = P.tupleLen[l] + 2;
        int n = 0;
        for (int i = at + tid; i < cnt; i += B)
            n += pieces(l, sm.pool + S.levelOff[l] + i * stride, i == at ? skip : 0);
        n = __reduce_add_sync(0xffffffffu, n);
        if ((tid & 31) == 0 && n) atomicAdd(&S.spillN[l], n);
    }
    __syncthreads();
    if (tid == 0) {
        unsigned nRec = 0, nTask = 0;
        for (int l = kBase; l <= k; ++l) {
            const int c = l + 1 == P.m ? kSpillChunkLeaf : kSpillChunk;
            nRec += S.spillN[l];
            nTask += (S.spillN[l] + c - 1) / c;
        }
        nTask += (rootsEnd - task.end + P.groupMax - 1) / max(P.groupMax, 1);   // the groups behind it, a task each
        bool ok = nTask > 1 && nRec <= (unsigned)kSpillRecs;   // one task would gain nothing
        uint32_t* dst = rows;
        int supAt = -1;
        if (ok && shared) {
            const unsigned long long need = (unsigned long long)((nWords + 3) & ~3);
            const unsigned long long at = atomicAdd(&sp.ctl->rowWords, need);
            ok = at + need <= (unsigned long long)kSpillRowWords;
            dst = sp.rows + at;
        }
        if (ok && sup) {   // (also of rows that are global already: this task's fused count is put off either way)
            supAt = atomicAdd(&sp.ctl->sups, 1);
            ok = supAt < kSpillSups;
        }
        unsigned long long old = 0;
        if (ok) ok = spill_take(&sp.ctl->used[sp.out], nTask, nRec, old);
        // (rows or a support slot taken before a list turned out full are lost to this launch)
        if (supAt >= 0 && supAt < kSpillSups)
            sp.sups[supAt] = SpillSup{ok ? task.plan : -1, task.beg, task.end - task.beg, 0, dst};
        S.spill = ok ? 1 : 0;
        S.spillAt = (int)(old >> 32);
        S.spillRec = (int)(unsigned)old;
        S.spillRows = dst;
    }
    __syncthreads();
    if (!S.spill) return false;
    uint32_t* const dst = S.spillRows;
    if (shared)
        for (int i = tid; i < nWords; i += B) dst[i] = rows[i];
    // tasks, level by level; records of a level in the order of their claims
    int t = S.spillAt, r = S.spillRec;
    for (int l = kBase; l <= k; ++l) {
        const int n = S.spillN[l], c = l + 1 == P.m ? kSpillChunkLeaf : kSpillChunk;
        for (int j = tid; j * c < n; j += B)
            sp.tasks[sp.out & 1][t + j] = SpillTask{task.plan, l, r + j * c, min(c, n - j * c), task.beg,
                                                task.end - task.beg, dst};
        t += (n + c - 1) / c;
        r += n;
    }
    for (int b = task.end + tid * P.groupMax, j = t + tid; b < rootsEnd; b += B * P.groupMax, j += B)
        sp.tasks[sp.out & 1][j] = SpillTask{task.plan, -1, 0, 0, b, min(P.groupMax, rootsEnd - b), nullptr};
    __syncthreads();
    if (tid == 0) {
        int at = S.spillRec;
        for (int l = kBase; l <= k; ++l) {
            const int n = S.spillN[l];
            S.spillN[l] = at;
            at += n;
        }
    }
    __syncthreads();
    for (int l = kBase; l <= k; ++l) {
        int at, skip0;
        level_pos(l, at, skip0);
        const int lenL = P.tupleLen[l], cnt = min(S.count[l], P.cap), stride = lenL + 2;
        const int seg = l + 1 == P.m ? kSpillSegLeaf : kSpillSeg;
        for (int i = at + tid; i < cnt; i += B) {
            const int* it = sm.pool + S.levelOff[l] + i * stride;
            const int skip = i == at ? skip0 : 0;
            const int n = pieces(l, it, skip);
            if (!n) continue;
            const int slot = atomicAdd(&S.spillN[l], n);
            for (int q = 0; q < n; ++q) {
                int* rec = sp.recs[sp.out & 1] + (long long)(slot + q) * kSpillRecInts;
                for (int j = 0; j < lenL; ++j) rec[j] = it[j];
                const int b = skip + q * seg;
                rec[lenL] = it[lenL] + b;
                rec[lenL + 1] = n == 1 ? it[lenL + 1] - b : min(seg, it[lenL + 1] - b);
            }
        }
    }
    return true;
}

// Fills the record of level l (one thread).
template <int B>
__device__ __noinline__ void level_info(Smem<B>& sm, const DevIndex& ix, int l, bool pairs, bool sortMode, bool sliced,
                                        bool claims, int leafChunk, int wideChunk) {
    const DevPlan& P = sm.plan;
    Level& L = sm.st.lv[l];
    const DevStep& st = P.steps[l];
    const bool leaf = l + 1 == P.m;
    const int len = P.tupleLen[l];
    int at = 0;
    for (int q = 0; q < l; ++q) at += P.cap * (P.tupleLen[q] + 2);
    L.len = len;
    L.at = at;
    L.nextAt = at + P.cap * (len + 2);
    L.nextLen = leaf ? 0 : P.tupleLen[l + 1];
    const bool filters = (P.chkN[l + 1] | P.usedN[l + 1]) != 0;
    int f = (leaf ? kLvLeaf : 0) | (pairs && st.hoWhich ? kLvHo : 0) |
            (pairs && P.hoLevel >= 1 && l >= P.hoLevel ? kLvHasRank : 0) | (filters ? kLvFilters : 0) |
            (st.kind == kScan ? kLvScan : 0) | (st.sameVar ? kLvSameVar : 0) | (st.kind == kRowScan ? kLvRowScan : 0) |
            (st.nNew == 2 ? kLvTwo : 0) | (claims && l == P.claimLevel ? kLvClaims : 0);
    L.vals = st.kind == kExpand ? ix.val[st.dir] : (st.kind == kRowScan ? ix.rowKey[st.dir] : ix.src[0]);
    L.ranks = st.kind == kExpand ? ix.valRank[st.dir] : (st.hoWhich == 1 ? ix.srcRank[0] : ix.valRank[0]);
    L.rankBase = st.kind == kRowScan ? ix.predRow[st.dir][st.pred] : 0;
    // When the next step expands from the value this step binds, that value's
    // row signature (stored beside it) drops most candidates whose next row
    // is absent before any lookup.
    L.sigs = nullptr;
    L.sigShift = 0;
    if (!leaf && st.kind == kExpand && P.steps[l + 1].kind == kExpand && P.steps[l + 1].keyRef == len) {
        const int bit = sig_bit(P.steps[l + 1].pred, P.steps[l + 1].dir);
        L.sigs = reinterpret_cast<const uint32_t*>(ix.valSig[st.dir]) + (bit >> 5);
        L.sigShift = bit & 31;
        f |= kLvSig | (sortMode ? 0 : kLvWide);
    }
    // A new item of the next level whose segment holds no value with a row
    // under the step after it (keyed on that value) is not stored.
    L.lookShift = 0;
    if (l + 2 < P.m && P.steps[l + 1].kind == kExpand && P.steps[l + 2].kind == kExpand &&
        P.steps[l + 2].keyRef == P.tupleLen[l + 1]) {
        const int bit = sig_bit(P.steps[l + 2].pred, P.steps[l + 2].dir);
        L.lookShift = bit & 31;
        f |= kLvLook | (bit & 32 ? kLvLookHigh : 0);
    }
    L.maxTake = leaf ? leafChunk : ((f & kLvWide) ? wideChunk : P.cap);
    // Hub path: when the leaf binds hO and tests nothing but injectivity, an
    // item whose segment is a whole hub row is counted by OR-ing the row's
    // rank bitmap into its pair row (32 candidates per word) instead of
    // candidate by candidate.
    // Memo path: the plan ends in two expand steps x -> y -> hO with nothing
    // but injectivity to test; an item whose first segment is a hub row with
    // a suffix memo is counted from the memo's maps (see memo_item).  A
    // four-step plan may also have the three-step memo, at level 1.
    // Scan path: the plan ends in a row scan binding hO and the free value
    // behind it; the rows are counted from their scan memo.
    int path = 0;
    const bool whole = !(sliced && l == 0);   // (a slice is never a whole row)
    if (pairs && !sortMode) {
        if (leaf) {
            if (st.hoWhich != 0 && st.kind == kExpand && st.nNew == 1 && !filters && ix.nHub > 0 && whole) path = 1;
        } else if (P.memoTab != nullptr && l + 1 == P.memoLevel) path = 2;
        else if (P.memo3Tab != nullptr && l == 1) path = 4;
        else if (P.scanBits != nullptr && l + 1 == P.scanLevel && whole) path = 5;
    } else if (!pairs && leaf && P.memoTab != nullptr && l + 1 == P.memoLevel && whole) path = 3;
    L.flags = f | path << kLvPath;
}

// kS: the task may be spilled; st: the spill task to resume (`task` its
// roots), or null.
template <int B, bool kC, bool kD, bool kS>
__device__ __forceinline__ void run_task(Smem<B>& sm, const DevIndex& ix, const DevTask& task,
                                         unsigned long long* results, int* status, Meter<kC>& mt, const SpillArgs& sp,
                                         const SpillTask* st) {
    constexpr int kLeafChunk = 16 * B;
    // candidates of a non-leaf round whose next step has a signature test
    // (most candidates die on it): more than the next level's capacity, so
    // a round may find that level full (see `wide` below)
    constexpr int kWideChunk = 8 * B;
    // A window takes at most this many candidates of one item, so that its
    // prefix sums fit 32 bits; no round consumes as many, so a longer item
    // always has candidates left for the next window.
    constexpr int kMaxSeg = 1 << 21;
    static_assert(kLeafChunk < kMaxSeg && (long long)B * kMaxSeg <= 1 << 30, "window sums fit an int");
    const DevPlan& P = sm.plan;
    BlockState<B>& S = sm.st;
    const int tid = threadIdx.x;
    const int G = task.end - task.beg;
    const bool pairs = P.mode == kPairs;
    // Dedup targets.  A split heavy root (one root, G == 1) uses its global
    // row for both the pair bits and the found bit; counting happens on
    // insertion so that the slices of one root count each result once.  A
    // resumed spill task does the same with the rows of all its roots.
    const bool resumed = kS && st != nullptr;
    const bool sliced = task.gRow >= 0;   // level 0 holds a slice of the root's segment
    const bool heavy = resumed || sliced;
    // Sort mode appends pair keys instead of setting bits (no bitmap at
    // all); block rows keep the task's rows in the block's own region of a
    // global buffer instead of one row per root of the phase.
    const bool sortMode = pairs && P.pairKeys != nullptr;
    const bool blockRows = pairs && !heavy && !sortMode && P.gBlockWords > 0;
    const bool shared = !heavy && !(pairs && (P.gBitmap || sortMode));
    uint32_t* sbits = reinterpret_cast<uint32_t*>(sm.pool + P.bitmapOff);
    int* const items = sm.pool;
    uint32_t* bm = resumed ? st->rows
                   : heavy ? (P.gHeavy ? P.gHeavy + (long long)task.gRow * P.rowWords : nullptr)
                         : (shared ? sbits : (blockRows ? P.gBitmap + (long long)blockIdx.x * P.gBlockWords : P.gBitmap));
    uint32_t* fb = heavy ? bm : sbits;   // kExist found bits
    // per-phase global rows start at the phase's first root: bm is the row of
    // the task's first one
    if (pairs && !heavy && !shared && !blockRows && !sortMode) bm += ((long long)task.beg - P.gRowBase) * P.rowWords;
    const long long keyRow0 = (long long)task.beg - P.gRowBase;   // sort mode: key row of the task's root 0

    // clear the task's shared dedup bits
    // pair rows are word-aligned: row r occupies words [r * rowWords, (r + 1) * rowWords)
    const int nWords = heavy ? 0 : (shared ? (int)(pairs ? (long long)G * P.rowWords : ((G + 31) >> 5))
                                           : (pairs ? 0 : ((G + 31) >> 5)));
    for (int i = tid; i < nWords; i += B) sbits[i] = 0u;
    if (blockRows && (long long)G * P.rowWords > P.gBlockWords) {   // the task builder keeps tasks this small
        if (tid == 0) {
            S.spill = 0;
            atomicOr(status, 32);
        }
        __syncthreads();   // as on the way out below: the caller's last reads of `next` are done
        return;
    }
    if (blockRows) {
        // the region is 16-byte aligned and a whole number of uint4 long
        uint4* b4 = reinterpret_cast<uint4*>(bm);
        const long long n4 = ((long long)G * P.rowWords + 3) >> 2;
        for (long long i = tid; i < n4; i += B) b4[i] = make_uint4(0u, 0u, 0u, 0u);
        if (tid == 0) mt.add(16 * (unsigned long long)n4);
    }
    // hub and memo items: the task's claim table (roots and slots must fit its fields)
    const bool claims = P.hubSeen && G <= 1024 && ix.nHub <= (1 << 20);
    if (claims)
        for (int i = tid; i < kHubSeen; i += B) P.hubSeen[(long long)blockIdx.x * kHubSeen + i] = 0ull;
    if (tid == 0) {
        S.firstFail = INT_MAX;
        S.safeLevels = 0;
        S.spill = 0;
        S.lookAt = !kS || sp.out < 0 || sortMode || blockRows ? LLONG_MAX : (sp.always ? 0 : clock64() + kSpillEvery);
        S.rows = pairs ? bm : fb;
        S.rowsWords = !heavy && (shared || !pairs) ? (pairs ? G * P.rowWords : (G + 31) >> 5) : 0;
        S.rowsSup = P.supN > 0 && !heavy ? 1 : 0;
        S.base = resumed ? st->level : 0;
        int off = 0;
        for (int l = 0; l <= kMaxBody; ++l) {
            S.curItem[l] = 0;
            S.curOff[l] = 0;
            S.count[l] = 0;
            S.levelOff[l] = off;
            if (l < P.m) off += P.cap * (P.tupleLen[l] + 2);
            else if (P.m == 0 && l == 0) off += P.cap * P.tupleLen[0];
        }
    }
    if constexpr (kS) {   // (its latency hides behind the roots')
        if (tid == B - 1 && sp.out >= 0) S.idle = *reinterpret_cast<const volatile int*>(S.queue) - S.nTasks;
    }
    if (tid >= 32 && tid - 32 < P.m) level_info<B>(sm, ix, tid - 32, pairs, sortMode, sliced, claims, kLeafChunk, kWideChunk);
    __syncthreads();

    const int kBase = resumed ? st->level : 0;   // the search ends when this level is exhausted
    if (resumed) {
        const int lenL = P.tupleLen[kBase], ints = lenL + 2;
        const int n = min(st->recN, P.cap);
        for (int i = tid; i < n * ints; i += B) {
            const int r = i / ints, q = i - r * ints;
            items[S.levelOff[kBase] + i] = sp.recs[sp.in & 1][(long long)(st->recBeg + r) * kSpillRecInts + q];
        }
        if (tid == 0) S.count[kBase] = n;
    } else {
    // ---- level 0: roots (tuple, then the segment of step 1) ----
        const int len0 = P.tupleLen[0];
        const int stride0 = P.m > 0 ? len0 + 2 : len0;
        // as for deeper items: a root whose segment has no value able to
        // take step 2 (keyed on that value) is not stored
        const bool lookTest0 = P.m >= 2 && P.steps[0].kind == kExpand && P.steps[1].kind == kExpand &&
                               P.steps[1].keyRef == len0;
        const int lookBit0 = lookTest0 ? sig_bit(P.steps[1].pred, P.steps[1].dir) : 0;
        // the first step expands the root's own row: its record has all
        const bool ownRow = P.rootKind == kRootRows && P.m > 0 && P.steps[0].kind == kExpand && !P.steps[0].free &&
                            P.steps[0].pred == P.rootPred && P.steps[0].dir == P.rootDir &&
                            P.steps[0].keyRef == kTupleHead;
        for (int i = tid; i < G; i += B) {
            const int r = task.beg + i;
            int tv[kTupleHead + 2];
            tv[0] = i;
            tv[1] = kItemNew;
            int nv = kTupleHead;
            bool ok = true;
            RowHit seg{make_int2(0, 0), make_uint2(0u, 0u), -1, -1};
            if (ownRow) {
                const uint4* p = reinterpret_cast<const uint4*>(ix.rows[P.rootDir] + r);
                const uint4 s = __ldg(p), t = __ldg(p + 1);
                mt.add(32);
                tv[nv++] = (int)s.x;
                seg = RowHit{make_int2((int)s.y, (int)s.z), make_uint2(t.x, t.y), -1, (int)s.w};
            } else if (P.rootKind == kRootRows) {
                tv[nv++] = __ldg(ix.rowKey[P.rootDir] + r);
                mt.add(4);
            } else {
                mt.add(8);
                const int key = __ldg(ix.src[P.rootDir] + r);
                const int v = __ldg(ix.val[P.rootDir] + r);
                if (P.rootKeyEqVal && key != v) ok = false;
                if (P.rootKeyNeVal && key == v) ok = false;
                if (P.rootValConst < 0 && v != P.consts[-1 - P.rootValConst]) ok = false;
                if (P.rootAppendKey) tv[nv++] = key;
                if (P.rootAppendVal) tv[nv++] = v;
            }
            if (ok && nv != len0) { ok = false; atomicOr(status, 2); }
            auto val0 = [&](TermRef ref) -> int { return ref < 0 ? P.consts[-1 - ref] : tv[ref < nv ? ref : 0]; };
            if (ok) ok = pass_filters(P, ix, 0, mt, val0);
            if (ok && P.m > 0) {
                if (!ownRow) seg = step_row(P, ix, 0, mt, val0);
                tv[1] = item_state(P.steps[0], seg.hub);
                if (sliced) {
                    const int b0 = seg.seg.x;
                    seg.seg.x = min(seg.seg.y, b0 + task.sub0);
                    seg.seg.y = min(seg.seg.y, b0 + task.sub1);
                    // (a slice's values are not the whole row's: no hub or memo, and its own signatures)
                    tv[1] = kItemEnum;
                    if (lookTest0 && seg.seg.y > seg.seg.x) {
                        const uint2 w = __ldg(reinterpret_cast<const uint2*>(ix.sufSig[P.steps[0].dir]) + seg.seg.x);
                        seg.sig = w;
                        mt.add(8);
                    }
                }
                ok = seg.seg.y > seg.seg.x;
                if (ok && lookTest0) ok = ((lookBit0 & 32 ? seg.sig.y : seg.sig.x) >> (lookBit0 & 31)) & 1u;
            }
            if (ok) {
                const int slot = atomicAdd(&S.count[0], 1);
                if (slot < P.cap) {
                    int* dst = items + S.levelOff[0] + slot * stride0;
                    for (int q = 0; q < len0; ++q) dst[q] = tv[q];
                    if (P.m > 0) { dst[len0] = seg.seg.x; dst[len0 + 1] = seg.seg.y - seg.seg.x; }
                } else {
                    atomicOr(status, 4);
                }
            }
        }
    }
    __syncthreads();

    unsigned long long myNew = 0;
    if (P.m == 0) {
        for (int i = tid; i < S.count[0] && i < P.cap; i += B) {
            const int root = items[S.levelOff[0] + i * P.tupleLen[0]];
            const uint32_t old = atomicOr(&fb[root >> 5], 1u << (root & 31));
            if (heavy && !(old & (1u << (root & 31)))) myNew++;
        }
    } else {
        // The search position (level k, first window item w0, candidates of
        // that item consumed already) is kept alike in every thread's
        // registers; a level's position goes to shared memory only when the
        // search descends below it.  A round takes two barriers: one
        // publishes the window's prefix sums, one closes the round.  Reads
        // of the shared counters that a later step may reset can only see
        // the reset when the decision they feed is the same either way.
        int k = kBase, w0 = 0, off = 0;
        for (;;) {
            if constexpr (kS) {
                if (S.spill) {   // set before the last round's barrier: all threads are here
                    if (spill_items<B>(sm, task, sp, k, w0, off)) break;
                }
            }
            const int cnt = min(S.count[k], P.cap);
            if (w0 >= cnt) {
                if (k == S.base) break;
                // nobody reads level k's bit again before it is re-entered
                if (tid == 0) S.safeLevels &= ~(1u << k);
                --k;
                w0 = S.curItem[k];
                off = S.curOff[k];
                continue;
            }
            const int nw = min(B, cnt - w0);
            const Level& lv = S.lv[k];
            const int lvf = lv.flags;   // uniform for the round; what only survivors need is read when they do
            const int lenK = lv.len;
            const int strideK = lenK + 2;
            int* const baseK = items + lv.at;
            const bool leaf = (lvf & kLvLeaf) != 0;
            const int pathKind = lvf >> kLvPath;
            bool isHub = false;   // item marked for the hub or memo pass

            // window: the stored neighbour segment of each item
            int myBeg = 0;
            int myLen = 0;
            if (tid < nw) {
                int* it = baseK + (w0 + tid) * strideK;
                bool pruned = false;
                if (!pairs) {
                    pruned = (fb[it[0] >> 5] >> (it[0] & 31)) & 1u;
                    if (heavy) mt.add(4);
                } else if ((lvf & kLvHasRank) && !sortMode) {
                    pruned = (bm[(long long)it[0] * P.rowWords + (it[1] >> 5)] >> (it[1] & 31)) & 1u;
                    if (!shared) mt.add(4);
                }
                if (!pruned) {
                    myBeg = it[lenK];
                    myLen = it[lenK + 1];
                    if (pathKind) {
                        // A round consumes candidates, not items: an item may
                        // wait through many windows.  It is classified in its
                        // first one and the verdict kept in its rank slot
                        // (unused before hO is bound).  Per-round
                        // classification was 25 % of the block time of a
                        // 5-atom biomedical rule (13.2M for 0.33M items).
                        int code = it[1];
                        if (code <= kItemNew) {
                            const int hub = -1 - code;
                            if (hub >= 0 ? pathKind == 5 : pathKind != 5) {
                                code = kItemEnum;
                            } else if (pathKind == 1) {
                                code = kItemHub + hub;   // the segment is a whole hub row
                            } else {
                                const int c = classify_item(P, ix, P.steps[k], it, lenK, pathKind, myBeg, myLen, fb, heavy,
                                                            hub, mt);
                                if (c == -4) myNew += 1;   // a new found bit of a split root
                                code = c == -1 ? kItemEnum : (c >= 0 ? kItemHub + c : kItemDone);
                            }
                            it[1] = code;
                        }
                        if (code >= kItemHub) {
                            isHub = true;
                            myBeg = -2 - (code - kItemHub);   // marks the item for the hub or memo pass; no candidates
                            myLen = 0;
                        } else if (code == kItemDone) {
                            myLen = 0;   // decided by the existence memo
                        }
                    }
                    if (tid == 0 && !isHub) {
                        myBeg += off;
                        myLen = myLen > off ? myLen - off : 0;
                    }
                    myLen = min(myLen, kMaxSeg);
                }
            }
            if (tid < ((nw + 31) & ~31)) {
                sm.wBeg[tid] = myBeg;
                sm.wLen[tid] = myLen;
            }
            if (tid == 0 && !leaf) S.count[k + 1] = 0;
            const bool anyHub = publish_window<B>(myLen, isHub, sm, nw);
            const int total = window_total<B>(sm, nw);
            // Wide round: up to kWideChunk candidates although each survivor
            // takes a slot of the next level.  A survivor that finds it full
            // records its candidate index, and the level resumes from the
            // first such candidate; items made from later candidates are made
            // again then, which changes no count (every dedup structure is a
            // set counted on insertion).  A level that overflowed takes
            // capacity-sized rounds, which cannot overflow, until it is
            // exhausted, so the search always advances.  Sort mode keeps
            // capacity-sized rounds: its key count must not depend on how
            // the threads raced (a launch is staged again with that count).
            const bool wide = (lvf & kLvWide) && !((S.safeLevels >> k) & 1u);
            const int take = min(total, (lvf & kLvWide) && !wide ? P.cap : lv.maxTake);

            // One candidate: its parent item `lo`, edge `e`, new value(s)
            // n0/n1 and (when this step binds hO) the loaded rank.
            auto eval = [&](int lo, int n0, int n1, int rankLoaded, int j) {
                const int* par = baseK + (w0 + lo) * strideK;
                const int root = par[0];
                if (!pairs && ((fb[root >> 5] >> (root & 31)) & 1u)) return;
                if ((lvf & kLvScan) && ((lvf & kLvSameVar) ? (n0 != n1) : (n0 == n1))) return;
                if (n0 != kAnyValue)
                    for (int q = kTupleHead; q < lenK; ++q) {
                        const int x = par[q];
                        if (x == n0 || ((lvf & kLvTwo) && x == n1)) return;
                    }
                auto valN = [&](TermRef ref) -> int {
                    if (ref < 0) return P.consts[-1 - ref];
                    if (ref < lenK) return par[ref];
                    return ref == lenK ? n0 : n1;
                };
                if ((lvf & kLvFilters) && !pass_filters(P, ix, k + 1, mt, valN)) return;
                int rank = par[1];
                if (lvf & kLvHo) {
                    rank = rankLoaded;
                    if (!leaf && !sortMode) {
                        if (!shared) mt.add(4);
                        if ((bm[(long long)root * P.rowWords + (rank >> 5)] >> (rank & 31)) & 1u) return;
                    }
                }
                if (leaf) {
                    if (!pairs) {
                        const uint32_t mask = 1u << (root & 31);
                        const uint32_t old = atomicOr(&fb[root >> 5], mask);
                        if (heavy) { mt.add(8); myNew += (old & mask) ? 0ull : 1ull; }
                    } else if (sortMode) {
                        emit_pair(P, keyRow0 + root, rank);
                        mt.add(8);
                    } else {
                        const uint32_t mask = 1u << (rank & 31);
                        uint32_t* word = bm + (long long)root * P.rowWords + (rank >> 5);
                        if (!shared) {
                            // a global row may be shared by many blocks, and most
                            // candidates find their bit set: a load costs a
                            // contended word less than an atomic
                            mt.add(4);
                            if (__ldcg(word) & mask) return;
                            mt.add(8);
                        }
                        const uint32_t old = atomicOr(word, mask);
                        myNew += (old & mask) ? 0ull : 1ull;
                    }
                } else {
                    const RowHit hit = step_row(P, ix, k + 1, mt, valN);
                    if (hit.seg.y <= hit.seg.x) return;
                    if ((lvf & kLvLook) &&
                        !((((lvf & kLvLookHigh) ? hit.sig.y : hit.sig.x) >> lv.lookShift) & 1u))
                        return;
                    if (!(lvf & (kLvHasRank | kLvHo))) rank = item_state(P.steps[k + 1], hit.hub);
                    const int slot = atomicAdd(&S.count[k + 1], 1);
                    if (slot >= P.cap) {
                        if (wide) atomicMin(&S.firstFail, j);
                        else atomicOr(status, 8);   // a capacity-sized round cannot fill the level
                        return;
                    }
                    const int lenN = lv.nextLen;
                    int* dst = items + lv.nextAt + slot * (lenN + 2);
                    dst[0] = root;
                    dst[1] = rank;
                    for (int q = kTupleHead; q < lenK; ++q) dst[q] = par[q];
                    dst[lenK] = n0;
                    if (lvf & kLvTwo) dst[lenK + 1] = n1;
                    dst[lenN] = hit.seg.x;
                    dst[lenN + 1] = hit.seg.y - hit.seg.x;
                }
            };

            // Candidates j = tid, tid + B, ... one at a time (groups of 2 and 4
            // with their loads issued together measured slower)
            {
                const int* const vals = lv.vals;
                const uint32_t* const sigs = lv.sigs;
                const int sigShift = lv.sigShift;
                WinCursor<B> cur;
                for (int j = tid; j < take; j += B) {
                    cur.seek(sm, nw, j);
                    const int lo = cur.item;
                    const int e = sm.wBeg[lo] + (j - cur.first(sm));
                    uint32_t sw = ~0u;
                    int n1 = 0, rk = 0;
                    if (lvf & kLvSig) { sw = __ldg(sigs + 2 * (long long)e); mt.add(4); }
                    const int n0 = __ldg(vals + e);
                    if (lvf & kLvScan) { n1 = __ldg(ix.val[0] + e); mt.add(8); } else mt.add(4);
                    if (lvf & kLvHo) {   // a row scan's rank is the row's place among the predicate's
                        rk = (lvf & kLvRowScan) ? e - lv.rankBase : __ldg(lv.ranks + e);
                        mt.add(4);
                    }
                    if ((sw >> sigShift) & 1u) eval(lo, n0, n1, rk, j);
                }
            }
            // where the next round at this level starts: the item holding
            // candidate `take` (items before it are consumed), and how much
            // of it is (computed here, not before the candidates, so that it
            // holds no registers across them)
            int cut = nw;
            int cutOff = 0;
            {
                if (take < total) {
                    WinCursor<B> c;
                    c.seek(sm, nw, take);
                    cut = c.item;
                    cutOff = take - c.first(sm) + (c.item == 0 ? off : 0);
                }
            }
            if (anyHub && (lvf & kLvClaims)) {
                // items of a (root, hub row) after enough middle values add nothing
                hub_claims(P.hubSeen + (long long)blockIdx.x * kHubSeen, baseK + w0 * strideK, strideK, cut,
                           P.steps[k].keyRef == kTupleHead + 1 ? kTupleHead + 2 : kTupleHead + 1, sm.wBeg, B,
                           leaf ? 2u : 3u);
                __syncthreads();
            }
            if (anyHub) {
                // hub items of the consumed part of the window: [0, cut)
                const int lane = tid & 31, warp = tid >> 5;
                constexpr int kWarps = B / 32;
                const DevStep stp = P.steps[k];
                const int words = P.rowWords;
                // memo items and domains up to 1,024 words: one warp per item
                // (a round's hub items in parallel); larger rows: the whole
                // block on each item in turn
                const bool perWarp = !leaf || words <= 1024;
                const int nEx = lenK - kTupleHead;
                const int exDir = 1 - stp.dir;
                int ordinal = 0;
                for (int base = 0; base < cut; base += 32) {
                    const int i = base + lane;
                    unsigned bal = __ballot_sync(0xffffffffu, i < cut && sm.wBeg[i] <= -2);
                    while (bal) {
                        const int item = base + __ffs(bal) - 1;
                        bal &= bal - 1;
                        const int mine = ordinal++;
                        if (perWarp && mine % kWarps != warp) continue;
                        const int* par = baseK + (w0 + item) * strideK;
                        if (!leaf) {
                            const int slot = -2 - sm.wBeg[item];
                            const int nEx3 = pathKind == 4
                                ? memo3_exceptions(P, ix, par, lenK, slot, words, S.exRank[warp], lane, mt) : 0;
                            DevStep stB = P.steps[k + 1];
                            if (pathKind == 5) stB.dir = (int8_t)(1 - stB.dir);
                            myNew += memo_item(P, ix, stp, stB, par, lenK, slot,
                                               bm + (long long)par[0] * words, words, S.exRank[warp],
                                               lane, mt, shared, nEx3, pathKind == 5);
                            continue;
                        }
                        // hO must differ from every bound value: their ranks in hO's domain
                        int* ex = S.exRank[warp];
                        if (lane < nEx) {
                            ex[lane] = row_find(ix, stp.pred, exDir, par[kTupleHead + lane], mt).rank;
                        }
                        __syncwarp();
                        const int h = -2 - sm.wBeg[item];
                        const uint32_t* hb = ix.hubBits + __ldg(ix.hubOff + h);
                        uint32_t* dst = bm + (long long)par[0] * words;
                        const int w0b = perWarp ? lane : tid;
                        const int step = perWarp ? 32 : B;
                        for (int w = w0b; w < words; w += step) {
                            uint32_t m = __ldg(hb + w);
                            for (int q = 0; q < nEx; ++q)
                                if ((ex[q] >> 5) == w && ex[q] >= 0) m &= ~(1u << (ex[q] & 31));
                            mt.add(4);
                            if (m && !shared) m &= ~__ldcg(dst + w);
                            if (m) {
                                const uint32_t old = atomicOr(dst + w, m);
                                if (!shared) mt.add(8);
                                myNew += (unsigned long long)__popc(m & ~old);
                            }
                        }
                        __syncwarp();
                    }
                }
            }
            if constexpr (kD) {
                if (tid == 0 && global_ns() > S.deadline) S.stop = 1;
            }
            if constexpr (kS) {
                // blocks past the end of the queue are idle; once a sixteenth
                // of the launch is, the items left here are worth a follow-up
                // launch
                if (tid == 0 && clock64() > S.lookAt) {
                    const int idle = *reinterpret_cast<const volatile int*>(S.queue) - S.nTasks;
                    S.lookAt = sp.always ? 0 : clock64() + kSpillEvery;
                    if (idle * 16 >= (int)gridDim.x || sp.always) S.spill = 1;
                }
            }
            __syncthreads();
            if constexpr (kD) {
                if (S.stop) break;   // set before the barrier, read by every thread after it: all leave together
            }
            if (wide) {
                const int ff = S.firstFail;   // final after the barrier
                if (ff < take) {
                    WinCursor<B> c;
                    c.seek(sm, nw, ff);
                    cut = c.item;
                    cutOff = ff - c.first(sm) + (c.item == 0 ? off : 0);
                    if (tid == 0) S.safeLevels |= 1u << k;
                    // every thread has read the window and firstFail: the
                    // next round may rewrite them
                    __syncthreads();
                    if (tid == 0) S.firstFail = INT_MAX;
                }
            }
            const int nextItem = w0 + cut;
            if (!leaf && S.count[k + 1] > 0) {
                if (tid == 0) {
                    S.curItem[k] = nextItem;
                    S.curOff[k] = cutOff;
                }
                ++k;
                w0 = 0;
                off = 0;
            } else {
                w0 = nextItem;
                off = cutOff;
            }
        }
    }
    __syncthreads();

    // ---- fused support: every pair row of the task is complete here (a
    // split heavy root's row only after the launch: support_rows_kernel) ----
    if (P.supN > 0 && !heavy && !(kS && S.spill)) {
        const int lane = tid & 31;
        for (int j = 0; j < P.supN; ++j) {
            unsigned long long n = fused_support(P, ix, j, task.beg, G, bm, tid >> 5, B / 32, lane, 0, 1, mt);
#pragma unroll
            for (int d = 16; d; d >>= 1) n += __shfl_down_sync(0xffffffffu, n, d);
            if (lane == 0 && n) atomicAdd(results + P.supSlot[j], n);
        }
    }

    // ---- result ----
    unsigned long long mine = 0;
    if (!pairs && !heavy) {
        for (int i = tid; i < ((G + 31) >> 5); i += B) mine += __popc(sbits[i]);
    } else {
        mine = myNew;
    }
    const unsigned long long tot = block_sum<B>(mine, S);
    if (tid == 0 && tot) atomicAdd(results + P.resultSlot, tot);
    if (tid == 0) mt.add(8);
}

// kI: 0 plain, may spill; 5 plain, may not: most small launches, without the
// registers that spilling takes (10 biomedical rules 143 -> 125 us, a dense
// batch 80 -> 74 us, short rules one by one 5.6 -> 5.4 ms); 1 records each
// task's start and end time; 2 also counts the algorithmic bytes; 3 records
// task times under a deadline (served launches: past prof.budgetNs from the
// block's start the block abandons its task at the end of a frontier round,
// skips the rest, and marks the plans that lost a task in prof.incomplete);
// 4 one plan that comes with the launch (InlineLaunch).
template <int B, int kI>
__global__ void __launch_bounds__(B, 1024 / B)
engine_kernel(const __grid_constant__ DevIndex ix, const DevPlan* __restrict__ plans, const DevTask* __restrict__ tasks,
              int nTasks, int* taskCounter, unsigned long long* results, int* status, EngineProfile prof,
              const __grid_constant__ SpillArgs sp, const __grid_constant__ InlineLaunch in) {
    constexpr bool kC = kI == 2;
    constexpr bool kD = kI == 3;
    constexpr bool kS = kI == 0;   // only the plain variant spills: the others time whole tasks
    constexpr bool kIn = kI == 4;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem<B>& sm = *reinterpret_cast<Smem<B>*>(smem_raw);
    Meter<kC> mt;
    if (prof.span && threadIdx.x == 0) atomicMax(prof.span, ~global_ns());
    if constexpr (kD) {
        if (threadIdx.x == 0) sm.st.deadline = global_ns() + prof.budgetNs;
    }
    int loaded = -1;   // the plan in shared memory
    const bool follow = kS && sp.in >= 0;   // a follow-up launch: its tasks are a spill list
    if (follow) {
        nTasks = (int)(sp.ctl->used[sp.in] >> 32);
        taskCounter = &sp.ctl->next[sp.in];
        if (nTasks == 0) return;
    }
    if (threadIdx.x == 0) {
        sm.st.nTasks = nTasks - (int)gridDim.x;   // those the counter deals out
        sm.st.queue = taskCounter;
    }
    // a block's first task is its own number, the others come from the counter
    for (bool first = true;; first = false) {
        if (threadIdx.x == 0) {
            sm.st.task = first ? (int)blockIdx.x : (int)gridDim.x + atomicAdd(taskCounter, 1);
            if constexpr (kD) sm.st.stop = global_ns() > sm.st.deadline ? 1 : 0;
        }
        __syncthreads();
        const int t = sm.st.task;
        if (t >= nTasks) break;
        const SpillTask* st = nullptr;
        DevTask task;
        if (follow) {
            st = sp.tasks[sp.in & 1] + t;
            task = DevTask{st->plan, st->beg, st->beg + st->G, 0, 0, -1};
            if (st->level < 0) st = nullptr;   // roots that no block had begun
        } else if constexpr (kIn) {
            const int b = in.beg + t * in.chunk;
            task = DevTask{0, b, min(in.end, b + in.chunk), 0, 0, -1};
        } else {
            task = tasks[t];
        }
        if constexpr (kD) {
            if (sm.st.stop) {   // past the deadline: the task is skipped and its plan marked
                if (threadIdx.x == 0) atomicOr(prof.incomplete + task.plan, 1);
                __syncthreads();
                continue;
            }
        }
        unsigned long long t0 = 0;
        if constexpr (kI >= 1 && kI <= 3) {
            if (threadIdx.x == 0) {
                mt.add(sizeof(DevTask) + sizeof(DevPlan) + 8);
                t0 = global_ns();
            }
        }
        if (task.plan != loaded) {   // (a plan's tasks often follow one another)
            loaded = task.plan;
            const int* src = reinterpret_cast<const int*>(kIn ? &in.plan : plans + task.plan);
            int* dst = reinterpret_cast<int*>(&sm.plan);
            for (int i = threadIdx.x; i < (int)(sizeof(DevPlan) / 4); i += B) dst[i] = src[i];
            __syncthreads();
        }
        // a task of several groups of roots: one after the other
        const int group = st ? INT_MAX : max(1, sm.plan.groupMax);
        if (kS && threadIdx.x == 0) sm.st.rootsEnd = task.end;   // (read after run_task's first barrier)
        for (DevTask part = task; part.beg < task.end;) {
            part.end = group < task.end - part.beg ? part.beg + group : task.end;
            run_task<B, kC, kD, kS>(sm, ix, part, results, status, mt, sp, st);
            if constexpr (kS) {
                // One thread decides for the block: `spill` and `idle` are
                // written again as soon as a block goes on, so a warp that
                // looked at them itself after the barrier could decide
                // otherwise.  (`spill` is this thread's own; `idle` was
                // written before barriers of run_task.)
                if (threadIdx.x == 0)
                    sm.st.next = sm.st.spill ? kGroupLeave   // (the groups behind it went with it)
                                 : part.end < task.end && sp.out >= 0 &&
                                           (sm.st.idle * 16 >= (int)gridDim.x || sp.always)
                                       ? kGroupGive : kGroupGoOn;
            }
            __syncthreads();
            if constexpr (kD) {
                if (sm.st.stop) break;
            }
            if constexpr (kS) {
                const int next = sm.st.next;   // written again behind the next run_task's barriers
                if (next == kGroupLeave) break;
                if (next == kGroupGive && spill_groups<B>(sm, sp, task.plan, part.end, task.end)) break;
            }
            part.beg = part.end;
        }
        if (kIn && nTasks <= (int)gridDim.x) break;   // every block has had its one task
        if constexpr (kD) {
            if (threadIdx.x == 0 && sm.st.stop) atomicOr(prof.incomplete + task.plan, 1);
        }
        if constexpr (kI >= 1 && kI <= 3) {
            if (threadIdx.x == 0 && prof.taskNs) {
                prof.taskNs[2 * t] = t0;
                prof.taskNs[2 * t + 1] = global_ns();
            }
        }
    }
    if constexpr (kC) {
        unsigned long long b = mt.bytes;
        for (int d = 16; d; d >>= 1) b += __shfl_down_sync(0xffffffffu, b, d);
        if ((threadIdx.x & 31) == 0 && b && prof.bytes) atomicAdd(prof.bytes, b);
    }
    if (prof.span && threadIdx.x == 0) atomicMax(prof.span + 1, global_ns());
    if (kIn && in.publish) {
        __syncthreads();   // the block's results are out
        if (threadIdx.x == 0) {
            int* words = static_cast<int*>(in.ctl);
            __threadfence();
            if (atomicAdd(words + kInlineWords, 1) == (int)gridDim.x - 1) {   // the last block
                __threadfence();
                int4* src = static_cast<int4*>(in.ctl);
                int4* dst = static_cast<int4*>(in.host);
                for (int i = 0; i < kInlineWords / 4; ++i) {
                    dst[i] = __ldcg(src + i);
                    src[i] = make_int4(0, 0, 0, 0);
                }
                words[kInlineWords] = 0;
                __threadfence_system();   // the words before their flag; the cleared ones before the next launch's
                *(static_cast<volatile int*>(in.host) + kInlineWords) = in.seq;
            }
        }
    }
}

template <int B>
static cudaError_t configure_b() {
    const int smem = (int)sizeof(Smem<B>);
    cudaError_t e = cudaFuncSetAttribute(engine_kernel<B, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(engine_kernel<B, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(engine_kernel<B, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(engine_kernel<B, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(engine_kernel<B, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(engine_kernel<B, 5>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    return e;
}

size_t engine_smem_bytes(int block) {
    switch (block) {
        case 128: return sizeof(Smem<128>);
        case 256: return sizeof(Smem<256>);
        default: return sizeof(Smem<512>);
    }
}

__global__ void memo_build_kernel(DevIndex ix, const MemoJob* jobs, int nJobs);

cudaError_t engine_configure() {
    cudaError_t e = configure_b<128>();
    // (its limit, once: a launch that set what it needs itself could be
    // overtaken by another thread's smaller one)
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(memo_build_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMemoSmemRanks * 4);
    if (e == cudaSuccess) e = configure_b<256>();
    if (e == cudaSuccess) e = configure_b<512>();
    return e;
}

template <int B>
static void launch_b(const DevIndex& ix, const DevPlan* plans, const DevTask* tasks, int nTasks, int* taskCounter,
                     unsigned long long* results, int* status, int grid, cudaStream_t stream,
                     const EngineProfile* prof, const SpillArgs& sp, const InlineLaunch& in) {
    const size_t smem = sizeof(Smem<B>);
    const EngineProfile p = prof ? *prof : EngineProfile{};
    if (in.on)
        engine_kernel<B, 4><<<grid, B, smem, stream>>>(ix, plans, tasks, nTasks, taskCounter, results, status, p, sp, in);
    else if (p.bytes)
        engine_kernel<B, 2><<<grid, B, smem, stream>>>(ix, plans, tasks, nTasks, taskCounter, results, status, p, sp, in);
    else if (p.budgetNs && p.incomplete && p.taskNs)
        engine_kernel<B, 3><<<grid, B, smem, stream>>>(ix, plans, tasks, nTasks, taskCounter, results, status, p, sp, in);
    else if (p.taskNs)
        engine_kernel<B, 1><<<grid, B, smem, stream>>>(ix, plans, tasks, nTasks, taskCounter, results, status, p, sp, in);
    else if (!sp.ctl)
        engine_kernel<B, 5><<<grid, B, smem, stream>>>(ix, plans, tasks, nTasks, taskCounter, results, status, p, sp, in);
    else
        engine_kernel<B, 0><<<grid, B, smem, stream>>>(ix, plans, tasks, nTasks, taskCounter, results, status, p, sp, in);
}

// Suffix memos (see memo_item): one block per job (a hub row x of one
// transition); warps take the y in N1(x), lanes the h in N2(y).  The first
// witness of h sets its S1 bit, the second its S2 bit, later ones its S3 bit
// (atomicOr returns the old word).
// Adds one path ending at `rank` to a three-step memo's counts: a 32-bit
// shared counter, or the saturating byte in global memory.
__device__ __forceinline__ void memo3_count_path(uint32_t* smemCnt, uint32_t* cnt, uint32_t* S1, int rank) {
    if (smemCnt) {
        atomicAdd(smemCnt + rank, 1u);
        return;
    }
    uint32_t* cw = cnt + (rank >> 2);
    const int sh = (rank & 3) * 8;
    uint32_t old = *cw;
    while (((old >> sh) & 0xffu) != 0xffu) {
        const uint32_t seen = atomicCAS(cw, old, old + (1u << sh));
        if (seen == old) break;
        old = seen;
    }
    atomicOr(S1 + (rank >> 5), 1u << (rank & 31));
}

__global__ void memo_build_kernel(DevIndex ix, const MemoJob* jobs, int nJobs) {
    extern __shared__ uint32_t memoSmem[];
    if ((int)blockIdx.x >= nJobs) return;
    const MemoJob job = jobs[blockIdx.x];
    uint32_t* S1 = job.bits;
    uint32_t* S2 = S1 + job.words;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nWarps = blockDim.x >> 5;
    if (job.row < 0) {
        // scan memo of (p1, d1): its rows [b0, b1), by their number of values
        // other than the key
        const int base = ix.predRow[job.d1][job.p1];
        for (int r = job.b0 + (int)threadIdx.x; r < job.b1; r += blockDim.x) {
            const int key = ix.rowKey[job.d1][base + r];
            const int e0 = ix.rowBeg[job.d1][base + r], e1 = ix.rowBeg[job.d1][base + r + 1];
            int n = 0;
            for (int e = e0; e < e1 && n < kMemoMaps; ++e) n += __ldg(ix.val[job.d1] + e) != key ? 1 : 0;
            for (int q = 0; q < n; ++q) atomicOr(S1 + q * job.words + (r >> 5), 1u << (r & 31));
        }
        return;
    }
    const int rb = ix.rowBeg[job.d1][job.row], re = ix.rowBeg[job.d1][job.row + 1];
    const int b = rb + job.b0, e = job.b1 < 0 ? re : rb + job.b1;
    Meter<false> mt;
    if (job.p3 >= 0) {
        // three steps: warps take the v2 of the slice, lanes the v3 in
        // N2(v2) and their N3 rows (a long one by the whole warp); every
        // path x -> v2 -> v3 -> h with x, v2, v3, h distinct counts once for
        // h, in shared counters added into the memo's bytes at the end
        const int x = ix.rowKey[job.d1][job.row];
        uint32_t* cnt = S1 + job.words;
        uint32_t* sc = job.wo <= kMemoSmemRanks ? memoSmem : nullptr;
        if (sc) {
            for (int r = threadIdx.x; r < job.wo; r += blockDim.x) sc[r] = 0u;
            __syncthreads();
        }
        for (int i = b + warp; i < e; i += nWarps) {
            const int v2 = __ldg(ix.val[job.d1] + i);
            if (v2 == x) continue;
            const int2 r2 = row_lookup(ix, job.p2, job.d2, v2, mt);
            for (int j0 = r2.x; j0 < r2.y; j0 += 32) {
                const int j = j0 + lane;
                int v3 = -1;
                int2 r3 = make_int2(0, 0);
                if (j < r2.y) {
                    v3 = __ldg(ix.val[job.d2] + j);
                    if (v3 != x && v3 != v2) r3 = row_lookup(ix, job.p3, job.d3, v3, mt);
                }
                const bool longRow = r3.y - r3.x >= 32;
                if (!longRow)
                    for (int t = r3.x; t < r3.y; ++t) {
                        const int h = __ldg(ix.val[job.d3] + t);
                        if (h == x || h == v2 || h == v3) continue;
                        const int rank = __ldg(ix.valRank[job.d3] + t);
                        if (rank >= 0 && rank < job.wo) memo3_count_path(sc, cnt, S1, rank);
                    }
                unsigned big = __ballot_sync(0xffffffffu, longRow);
                while (big) {   // long N3 rows: the whole warp walks each
                    const int src = __ffs(big) - 1;
                    big &= big - 1;
                    const int w3 = __shfl_sync(0xffffffffu, v3, src);
                    const int t0 = __shfl_sync(0xffffffffu, r3.x, src), t1 = __shfl_sync(0xffffffffu, r3.y, src);
                    for (int t = t0 + lane; t < t1; t += 32) {
                        const int h = __ldg(ix.val[job.d3] + t);
                        if (h == x || h == v2 || h == w3) continue;
                        const int rank = __ldg(ix.valRank[job.d3] + t);
                        if (rank >= 0 && rank < job.wo) memo3_count_path(sc, cnt, S1, rank);
                    }
                }
            }
        }
        if (sc) {
            __syncthreads();
            for (int r = threadIdx.x; r < job.wo; r += blockDim.x) {
                const uint32_t add = min(sc[r], 255u);
                if (!add) continue;
                uint32_t* cw = cnt + (r >> 2);
                const int sh = (r & 3) * 8;
                uint32_t old = *cw;
                for (;;) {
                    const uint32_t cur = (old >> sh) & 0xffu;
                    const uint32_t nv = min(cur + add, 255u);
                    if (nv == cur) break;
                    const uint32_t seen = atomicCAS(cw, old, (old & ~(0xffu << sh)) | (nv << sh));
                    if (seen == old) break;
                    old = seen;
                }
                atomicOr(S1 + (r >> 5), 1u << (r & 31));
            }
        }
        return;
    }
    const int x = ix.rowKey[job.d1][job.row];
    for (int i = b + warp; i < e; i += nWarps) {
        const int y = __ldg(ix.val[job.d1] + i);
        if (y == x) continue;   // x is bound wherever the memo is used: never a witness
        const int2 r = row_lookup(ix, job.p2, job.d2, y, mt);
        for (int j = r.x + lane; j < r.y; j += 32) {
            if (__ldg(ix.val[job.d2] + j) == y) continue;
            const int rank = __ldg(ix.valRank[job.d2] + j);
            if (rank < 0 || rank >= (job.words << 5)) continue;
            const uint32_t bit = 1u << (rank & 31);
            const uint32_t old = atomicOr(S1 + (rank >> 5), bit);
            if ((old & bit) && (atomicOr(S2 + (rank >> 5), bit) & bit)) atomicOr(S2 + job.words + (rank >> 5), bit);
        }
    }
}

// Fused support of split heavy roots and of spilled tasks, whose rows are
// complete after the launch.  The first nJobs blocks take one heavy root
// each, their warps sharing its head triples; the others share the spilled
// tasks, a warp per root.
__global__ void support_rows_kernel(const __grid_constant__ DevIndex ix, const DevPlan* plans, const SupJob* jobs,
                                    int nJobs, unsigned long long* results, const __grid_constant__ SpillArgs sp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nWarps = blockDim.x >> 5;
    Meter<false> mt;
    auto add = [&](const DevPlan& P, int j, unsigned long long n) {
        for (int d = 16; d; d >>= 1) n += __shfl_down_sync(0xffffffffu, n, d);
        if (lane == 0 && n) atomicAdd(results + P.supSlot[j], n);
    };
    if ((int)blockIdx.x < nJobs) {
        const SupJob jb = jobs[blockIdx.x];
        const DevPlan& P = plans[jb.plan];
        if (!P.gHeavy) return;
        const uint32_t* row = P.gHeavy + (long long)jb.gRow * P.rowWords;
        for (int j = 0; j < P.supN; ++j)
            add(P, j, fused_support(P, ix, j, jb.root, 1, row, 0, 1, lane, warp, nWarps, mt));
        return;
    }
    const int n = min(sp.ctl->sups, kSpillSups);
    for (int i = (int)blockIdx.x - nJobs; i < n; i += (int)gridDim.x - nJobs) {
        const SpillSup u = sp.sups[i];
        if (u.plan < 0) continue;
        const DevPlan& P = plans[u.plan];
        for (int j = 0; j < P.supN; ++j)
            add(P, j, fused_support(P, ix, j, u.beg, u.G, u.rows, warp, nWarps, lane, 0, 1, mt));
    }
}

cudaError_t support_rows(const DevIndex& ix, const DevPlan* plans, const SupJob* jobs, int nJobs,
                         unsigned long long* results, cudaStream_t stream, const SpillArgs& sp, int spillBlocks) {
    const int grid = nJobs + (sp.ctl ? spillBlocks : 0);
    if (grid <= 0) return cudaSuccess;
    support_rows_kernel<<<grid, 256, 0, stream>>>(ix, plans, jobs, nJobs, results, sp);
    return cudaGetLastError();
}

__global__ void widen_slots_kernel(const __grid_constant__ DevIndex ix, const HashSlot* hash16, long long n,
                                   DevSlot* slots) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const HashSlot s = hash16[i];
    DevSlot d{s.tag, s.key, s.beg, s.end, {0u, 0u}, -1, -1};
    if (s.tag != kEmptyTag) {
        const int dir = (int)(s.tag & 1u), pred = (int)(s.tag >> 1);
        const uint64_t sig = ix.sufSig[dir][s.beg];
        d.sig[0] = (uint32_t)sig;
        d.sig[1] = (uint32_t)(sig >> 32);
        d.rank = ix.srcRank[dir][s.beg];
        d.hub = ix.hubOf[dir][ix.predRow[dir][pred] + d.rank];
    }
    slots[i] = d;
}

__global__ void row_records_kernel(const __grid_constant__ DevIndex ix, int dir, int n, DevRow* rows) {
    const int r = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (r >= n) return;
    const int beg = ix.rowBeg[dir][r];
    const uint64_t sig = ix.sufSig[dir][beg];
    rows[r] = DevRow{ix.rowKey[dir][r], beg, ix.rowBeg[dir][r + 1], ix.hubOf[dir][r],
                     {(uint32_t)sig, (uint32_t)(sig >> 32)}, {0, 0}};
}

cudaError_t build_lookup(const DevIndex& ix, const HashSlot* hash16, long long n, DevSlot* slots, DevRow* const* rows,
                         const int* nRows) {
    if (n > 0) widen_slots_kernel<<<(unsigned)((n + 255) / 256), 256>>>(ix, hash16, n, slots);
    for (int d = 0; d < 2; ++d)
        if (nRows[d] > 0) row_records_kernel<<<(nRows[d] + 255) / 256, 256>>>(ix, d, nRows[d], rows[d]);
    return cudaGetLastError();
}

cudaError_t memo_build(const DevIndex& ix, const MemoJob* jobs, int nJobs, int maxWo, cudaStream_t stream) {
    if (nJobs <= 0) return cudaSuccess;
    const size_t smem = (size_t)std::min(maxWo, kMemoSmemRanks) * 4;
    memo_build_kernel<<<nJobs, 256, smem, stream>>>(ix, jobs, nJobs);
    return cudaGetLastError();
}

// prof (optional): task times when prof->taskNs is set, also byte counts
// when prof->bytes is set (instrumented variants); a launch span when
// prof->span is set (any variant).
cudaError_t engine_launch(const DevIndex& ix, const DevPlan* plans, const DevTask* tasks, int nTasks,
                          int* taskCounter, unsigned long long* results, int* status, int grid, int block,
                          cudaStream_t stream, const EngineProfile* prof, const SpillArgs& sp, const InlineLaunch* in) {
    if (nTasks <= 0 && sp.in < 0) return cudaSuccess;
    static const InlineLaunch none{};
    const InlineLaunch& il = in ? *in : none;
    switch (block) {
        case 128: launch_b<128>(ix, plans, tasks, nTasks, taskCounter, results, status, grid, stream, prof, sp, il); break;
        case 256: launch_b<256>(ix, plans, tasks, nTasks, taskCounter, results, status, grid, stream, prof, sp, il); break;
        case 512: launch_b<512>(ix, plans, tasks, nTasks, taskCounter, results, status, grid, stream, prof, sp, il); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace gr
