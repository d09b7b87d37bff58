// context.cu — graph context, staged launches and the C ABI
// (include/gpu_rules_api.h).
//
// Replaces the reference's GpuContext and entry points
// (GPU_03/gpu_rules_lib.cu:181-574).  Differences that matter to callers:
//  * errors are returned, never exit() (the reference's CUDA_OK calls exit,
//    GPU_03/gpu_common.cuh:8-15);
//  * unknown predicates and constants are resolved without growing the
//    dictionary (they match nothing, as a freshly interned id does);
//  * the body size is always computed (CPU_01 semantics), also when the
//    support is 0.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <chrono>
#include <memory>
#include <mutex>
#include <numeric>
#include <string>
#include <vector>

#include "engine.hpp"
#include "index_io.hpp"
#include "parallel.hpp"

namespace gr {

namespace {
thread_local std::string g_lastError;
}  // namespace

void set_error(const std::string& s) {
    g_lastError = s;
    std::fprintf(stderr, "[gpu_rules] %s\n", s.c_str());
}

namespace {
double host_ms() {
    return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

// The level whose hub or memo items may skip repeats (see kHubSeen), or -1:
// its tuple holds hS and two more values, its step expands from one of those
// two, and it is the leaf (binding hO, testing nothing but injectivity) or
// the level of the two-step memo.
int claim_level(const DevPlan& P) {
    if (P.mode != kPairs) return -1;
    auto shaped = [&](int k) {
        const DevStep& st = P.steps[k];
        return P.tupleLen[k] == kTupleHead + 3 && st.kind == kExpand && st.nNew == 1 &&
               (st.keyRef == kTupleHead + 1 || st.keyRef == kTupleHead + 2);
    };
    const int k = P.m - 1;
    if (k >= 0 && shaped(k) && P.steps[k].hoWhich != 0 && P.chkN[P.m] == 0 && P.usedN[P.m] == 0) return k;
    if (P.memoLevel > 0 && shaped(P.memoLevel - 1)) return P.memoLevel - 1;
    return -1;
}

// Bits that hold the values 0 .. n - 1 (at least one).
int bits_for(uint64_t n) {
    int b = 1;
    while (b < 64 && n > 1 && ((n - 1) >> b) != 0) ++b;
    return b;
}
constexpr unsigned long long kMaxSortKeys = 0xffffffffull;   // the sort's 32-bit positions
}  // namespace

namespace {
// Layout of Staged::dSpill: two lists of tasks and records, support jobs, rows.
size_t spill_part(int part) {
    const size_t sizes[] = {kSpillTasks * sizeof(SpillTask), kSpillTasks * sizeof(SpillTask),
                            (size_t)kSpillRecs * kSpillRecInts * 4, (size_t)kSpillRecs * kSpillRecInts * 4,
                            kSpillSups * sizeof(SpillSup), (size_t)kSpillRowWords * 4};
    size_t at = 0;
    for (int i = 0; i < part; ++i) at += (sizes[i] + 255) & ~size_t(255);
    return at;
}
size_t spill_bytes() { return spill_part(6); }
constexpr double kSpillSkew = 4.0;   // least PhaseTasks::skew among the phases of a launch that may spill
}  // namespace

namespace {
// Orders tasks [b, e) (and their costs) by falling cost x scale(i): a stable
// counting sort by quarter-octaves of the estimate.
template <class Scale>
void longest_first(std::vector<DevTask>& tasks, std::vector<double>& cost, size_t b, size_t e, Scale scale) {
    constexpr int kBuckets = 1024;
    auto bucket = [](double v) {
        if (!(v > 0.0)) return 0;
        int ex;
        const double m = std::frexp(v, &ex);   // v = m * 2^ex, m in [0.5, 1)
        return std::max(1, std::min(kBuckets - 1, 512 + 4 * ex + (int)((m - 0.5) * 8.0)));
    };
    std::vector<uint16_t> bk(e - b);
    std::vector<uint32_t> start(kBuckets + 1, 0);
    for (size_t i = b; i < e; ++i) {
        bk[i - b] = (uint16_t)bucket(cost[i] * scale(i));
        ++start[kBuckets - 1 - bk[i - b]];
    }
    uint32_t acc = 0;
    for (uint32_t& x : start) {
        const uint32_t n = x;
        x = acc;
        acc += n;
    }
    std::vector<DevTask> t2(e - b);
    std::vector<double> c2(e - b);
    for (size_t i = b; i < e; ++i) {
        const size_t at = start[kBuckets - 1 - bk[i - b]]++;
        t2[at] = tasks[i];
        c2[at] = cost[i];
    }
    std::copy(t2.begin(), t2.end(), tasks.begin() + (ptrdiff_t)b);
    std::copy(c2.begin(), c2.end(), cost.begin() + (ptrdiff_t)b);
}
}  // namespace

void Staged::stage(Context& c, const std::vector<const PhasePlan*>& phases, const std::vector<PlanSup>& sups,
                   bool sortTasks, cudaStream_t s, double walkBudget, int walkRule, bool allowSort, bool mayInline) {
    inl.clear();
    nPlans = (int)phases.size();
    nResults = nPlans + extraResults;
    stagedBlock = c.geom.block;
    nTasks = 0;
    bitmapWords = 0;
    blockWords = blockRegions = 0;
    nSort = sortSlotShift = 0;
    keyCap = 0;
    h2dBytes = d2hBytes = 0;
    dedup.assign(nPlans, kDedupShared);
    const unsigned long long hint = keyHint;   // consumed by this staging
    keyHint = 0;
    if (hint > kMaxSortKeys) allowSort = false;
    if (!nPlans) return;

    double tSect = host_ms();
    // ---- how each kPairs plan deduplicates ----
    // Per-phase global rows (one bitmap row per root, cleared before the
    // launch) while all of them fit the budget.  Beyond it, per plan: sort
    // mode when the estimated keys cost fewer bytes than clearing and setting
    // the rows, else block rows, whose memory grows with the launch's blocks
    // instead of the phase's roots.  (A key is priced at 22 times its size, as
    // a full sort in seven passes moves it.  Parting the keys by a hash moves
    // them one to three times, so close to the line keys would be the cheaper
    // choice; where the line should lie now has not been measured.)
    const size_t budgetWords = std::max<size_t>(c.dedupBudget / 4, 1);
    std::vector<size_t> fullWords(nPlans, 0);
    std::vector<double> est(nPlans, -1.0);
    auto estimate = [&](int i) {
        if (est[i] < 0) est[i] = std::max(1.0, c.tasks->work_estimate(*phases[i]));
        return est[i];
    };
    size_t fullTotal = 0;
    // the phases lie in their rules' plans, a few cache lines each: passes over
    // all of them run on host threads
    auto plan = [&](int i) -> const DevPlan& { return phases[i]->plan; };
    // (supports are fused when a batch is prepared, the mode is chosen by each
    // staging: a plan that counts supports needs rows to count them from, so
    // one that is forced to keys keeps its rows in shared memory)
    std::vector<uint8_t> global(nPlans, 0);
    parallel_for((size_t)nPlans, [&](size_t i) {
        const bool fused = !sups.empty() && sups[i].n > 0;
        const bool forced = c.dedupForce != 0 && !(fused && c.dedupForce == kDedupSort);
        global[i] = plan((int)i).mode == kPairs && (phases[i]->needsGlobalBitmap || forced) ? 1 : 0;
    }, 256);
    for (int i = 0; i < nPlans; ++i) {
        if (!global[i]) continue;
        fullWords[i] = (size_t)(phases[i]->rootEnd - phases[i]->rootBeg) * (size_t)std::max(plan(i).rowWords, 1);
        fullTotal += fullWords[i];
        dedup[i] = kDedupRows;
    }
    for (int i = 0; i < nPlans; ++i) {
        if (dedup[i] == kDedupShared) continue;
        if (c.dedupForce) {
            dedup[i] = c.dedupForce;
        } else if (fullTotal > budgetWords) {
            const double e = estimate(i);
            const double rowBytes = 4.0 * (double)fullWords[i] + 8.0 * e;
            const double sortBytes = 8.0 * e * 22.0;
            dedup[i] = (sortBytes < rowBytes && 16.0 * e <= (double)c.dedupBudget) ? kDedupSort : kDedupBlockRows;
        }
        if (dedup[i] == kDedupSort && !allowSort) dedup[i] = kDedupBlockRows;
    }
    // sort keys: [sort index | row | rank], at most 64 bits
    std::vector<int32_t> sortPlans;
    int rankBits = 1, rowBits = 1;
    for (int i = 0; i < nPlans; ++i)
        if (dedup[i] == kDedupSort) {
            sortPlans.push_back(i);
            rankBits = std::max(rankBits, bits_for((uint64_t)std::max(plan(i).wo, 1)));
            rowBits = std::max(rowBits, bits_for((uint64_t)std::max(phases[i]->rootEnd - phases[i]->rootBeg, 1)));
        }
    if (!sortPlans.empty()) {
        const int slotBits = sortPlans.size() > 1 ? bits_for(sortPlans.size()) : 0;
        if (rankBits + rowBits + slotBits > 64) {
            for (int i : sortPlans) dedup[i] = kDedupBlockRows;
            sortPlans.clear();
        } else {
            nSort = (int)sortPlans.size();
            sortSlotShift = rankBits + rowBits;
        }
    }
    if (nSort) {
        // kept so that a run whose keys overflow can be staged again
        inSups = sups;
        inPhases = phases;
        inSortTasks = sortTasks;
        inWalk = walkBudget;
        inWalkRule = walkRule;
        inAllowSort = allowSort;
    } else {
        inSups.clear();
        inPhases.clear();
    }
    // block rows: every resident block owns a region that holds its current
    // task's rows; tasks are cut to the rows a region holds
    std::vector<PhaseLimits> lim(nPlans);
    {
        size_t maxRow = 0;
        for (int i = 0; i < nPlans; ++i)
            if (dedup[i] == kDedupBlockRows) maxRow = std::max(maxRow, (size_t)std::max(plan(i).rowWords, 1));
        if (maxRow) {
            blockRegions = (size_t)std::max(c.grid, 1);
            const size_t regionCap = std::max(maxRow, budgetWords / blockRegions);
            size_t need = 0;
            for (int i = 0; i < nPlans; ++i) {
                if (dedup[i] != kDedupBlockRows) continue;
                const size_t rw = (size_t)std::max(plan(i).rowWords, 1);
                const int32_t g = (int32_t)std::max<size_t>(
                    1, std::min<size_t>(regionCap / rw, (size_t)std::max(1, std::min(plan(i).cap, 512))));
                lim[i].group = g;
                lim[i].maxHeavy = (int32_t)std::min<size_t>(INT_MAX, budgetWords / 4 / rw);
                need = std::max(need, (size_t)g * rw);
            }
            blockWords = (need + 3) & ~size_t(3);
        }
    }
    std::vector<size_t> gOff(nPlans, 0);
    for (int i = 0; i < nPlans; ++i) {
        if (dedup[i] != kDedupRows) continue;
        gOff[i] = bitmapWords;
        bitmapWords += fullWords[i];   // word-aligned rows
    }
    const size_t regionOff = (bitmapWords + 3) & ~size_t(3);   // 16-byte aligned regions
    cudaStream_t as = streamOrdered ? s : nullptr;
    if (bitmapWords || blockWords) dBitmap.ensure((regionOff + blockRegions * blockWords) * 4, as);
    if (nSort) {
        double want = 0;
        for (int i : sortPlans) want += estimate(i);
        const double lo = 65536.0, hi = std::max(lo, (double)c.dedupBudget / 16.0);
        keyCap = (unsigned long long)std::min(hi, std::max(lo, want));
        keyCap = std::min(std::max(keyCap, hint), kMaxSortKeys);
        dSort.ensure(256 + (size_t)keyCap * 16 + pairs_sort_hist_words(keyCap) * 4, as);
        hSort.ensure(8);
    }
    hostSect[0] += host_ms() - tSect;
    tSect = host_ms();
    // suffix memos first: the task builder weighs memoised roots by them
    std::vector<std::array<int, 6>> memoKeys;
    auto memo_key_of = [](const DevPlan& P) -> std::array<int, 6> {
        const DevStep& a = P.steps[P.memoLevel - 1];
        return {a.pred, a.dir, P.memoP2, P.memoD2, -1, 0};
    };
    // scan memos have no first step (p1 = -1)
    auto scan_key_of = [](const DevPlan& P) -> std::array<int, 6> {
        const DevStep& a = P.steps[P.scanLevel - 1];
        return {-1, 0, a.pred, a.dir, -1, 0};
    };
    auto memo3_key_of = [](const DevPlan& P) -> std::array<int, 6> {
        return {P.steps[1].pred, P.steps[1].dir, P.steps[2].pred, P.steps[2].dir, P.steps[3].pred, P.steps[3].dir};
    };
    // which of a plan's memos apply in this staging: bit 0 two-step, 1
    // three-step, 2 scan; and those that are not built yet
    std::vector<uint8_t> memoUse(nPlans, 0), memoNew(nPlans, 0);
    parallel_for((size_t)nPlans, [&](size_t i) {
        if (dedup[i] == kDedupSort) return;   // memos set bitmap words; keys carry every pair
        const DevPlan& P = plan((int)i);
        int use = (P.memoLevel > 0 ? 1 : 0) | (P.memoSteps == 3 && c.memo3 ? 2 : 0) | (P.scanLevel > 0 ? 4 : 0);
        if (use & 1) {
            // the memo leaves x out of x's own neighbours, as injectivity
            // does for a variable; a constant that is its own neighbour stays
            // one, so such a plan enumerates
            const DevStep& a = P.steps[P.memoLevel - 1];
            if (a.keyRef < 0) {
                const int32_t e = P.consts[-1 - a.keyRef];
                if (e >= 0 && c.hix.has_triple(a.pred, e, e)) use &= ~1;
            }
        }
        memoUse[i] = (uint8_t)use;
        if ((use & 1) && !c.memo_known(memo_key_of(P))) memoNew[i] |= 1;
        if ((use & 2) && !c.memo_known(memo3_key_of(P))) memoNew[i] |= 2;
        if ((use & 4) && !c.memo_known(scan_key_of(P))) memoNew[i] |= 4;
    }, 128);
    for (int i = 0; i < nPlans; ++i) {
        if (!memoNew[i]) continue;
        if (memoNew[i] & 4) memoKeys.push_back(scan_key_of(plan(i)));
        if (memoNew[i] & 1) memoKeys.push_back(memo_key_of(plan(i)));
        if (memoNew[i] & 2) memoKeys.push_back(memo3_key_of(plan(i)));
    }
    if (!memoKeys.empty()) c.ensure_memos(memoKeys, s);
    hostSect[1] += host_ms() - tSect;
    tSect = host_ms();
    std::vector<PhaseTasks> pts;
    c.tasks->build(phases, c.grid, true, pts, walkBudget, walkRule, &lim, true);
    hostSect[2] += host_ms() - tSect;
    tSect = host_ms();
    // split heavy roots of plans with fused support: counted after the launch
    std::vector<SupJob> supJobs;
    for (int i = 0; i < nPlans; ++i) {
        if (pts[i].heavyRows == 0 || sups.empty() || sups[i].n == 0) continue;
        std::vector<char> seenRow((size_t)pts[i].heavyRows, 0);
        for (const DevTask& t : pts[i].tasks)
            if (t.gRow >= 0 && !seenRow[(size_t)t.gRow]) {
                seenRow[(size_t)t.gRow] = 1;
                supJobs.push_back(SupJob{i, t.beg, t.gRow, 0});
            }
    }
    nSupJobs = (int)supJobs.size();
    std::vector<size_t> hOff(nPlans, 0);
    heavyWords = 0;
    auto row_words = [&](int i) -> int32_t { return plan(i).mode == kPairs ? (plan(i).wo + 31) / 32 : 1; };
    for (int i = 0; i < nPlans; ++i) {
        hOff[i] = heavyWords;
        if (pts[i].heavyRows && dedup[i] != kDedupSort)
            heavyWords += (size_t)pts[i].heavyRows * row_words(i);   // keys need no rows
    }
    if (heavyWords) dHeavy.ensure(heavyWords * 4, as);
    std::vector<int32_t> claimAt(nPlans, -1);
    if (c.hubClaims)
        parallel_for((size_t)nPlans, [&](size_t i) {
            if (dedup[i] != kDedupSort) claimAt[i] = claim_level(plan((int)i));
        }, 256);
    bool anyClaims = false;
    for (int i = 0; i < nPlans; ++i) anyClaims |= claimAt[i] >= 0;
    if (anyClaims) dHubSeen.ensure((size_t)std::max(c.grid, 1) * kHubSeen * 8, as);
    std::vector<DevTask> tasks;
    std::vector<double> cost;
    {
        size_t nt = 0;
        for (int i = 0; i < nPlans; ++i) nt += pts[i].tasks.size();
        tasks.reserve(nt);
        cost.reserve(nt);
        for (int i = 0; i < nPlans; ++i) {
            tasks.insert(tasks.end(), pts[i].tasks.begin(), pts[i].tasks.end());
            cost.insert(cost.end(), pts[i].cost.begin(), pts[i].cost.end());
        }
    }
    // The device's copy of plan i, written straight into the upload buffer
    // (8,000 plans of 1 KB: copied twice before).
    auto fill = [&](int i, DevPlan& P) {
        P = plan(i);
        P.rowWords = row_words(i);
        if (!(memoUse[i] & 1)) P.memoLevel = 0;
        if (!(memoUse[i] & 2)) P.memoSteps = 0;
        if (memoUse[i] & 4) {
            const SuffixMemo* m = c.memo_for(scan_key_of(P));
            if (m && m->words == P.rowWords) P.scanBits = m->bits;
        }
        if (memoUse[i] & 1) {
            const SuffixMemo* m = c.memo_for(memo_key_of(P));
            if (m && (P.mode != kPairs || m->words == P.rowWords)) {
                P.memoTab = m->tab;
                P.memoBits = m->bits;
                P.memoWords = m->words;
            }
        }
        if (memoUse[i] & 2) {
            const SuffixMemo* m = c.memo_for(memo3_key_of(P));
            if (m && m->words == P.rowWords && m->wo == P.wo) {
                P.memo3Tab = m->tab;
                P.memo3Bits = m->bits;
            }
        }
        if (!sups.empty() && sups[i].n > 0) {
            const auto dom = ho_domain(P);
            P.supN = sups[i].n;
            P.supDomPred = dom.first;
            P.supDomDir = dom.second;
            for (int j = 0; j < P.supN; ++j) {
                P.supPred[j] = sups[i].pred[j];
                P.supSlot[j] = nPlans + sups[i].slot[j];
            }
        }
        P.resultSlot = i;
        P.groupMax = pts[i].group;
        const int dm = dedup[i];
        uint32_t* gb = static_cast<uint32_t*>(dBitmap.p);
        P.gBitmap = dm == kDedupRows ? gb + gOff[i] : (dm == kDedupBlockRows ? gb + regionOff : nullptr);
        P.gRowBase = (dm == kDedupRows || dm == kDedupSort) ? phases[i]->rootBeg : 0;
        P.gBlockWords = dm == kDedupBlockRows ? (int64_t)blockWords : 0;
        P.gHeavy = (pts[i].heavyRows && dm != kDedupSort) ? static_cast<uint32_t*>(dHeavy.p) + hOff[i] : nullptr;
        P.claimLevel = claimAt[i];
        P.hubSeen = claimAt[i] >= 0 ? static_cast<unsigned long long*>(dHubSeen.p) : nullptr;
        if (dm == kDedupSort) {
            const int k = (int)(std::find(sortPlans.begin(), sortPlans.end(), i) - sortPlans.begin());
            char* sb = static_cast<char*>(dSort.p);
            P.keyCursor = reinterpret_cast<unsigned long long*>(sb);
            P.pairKeys = reinterpret_cast<unsigned long long*>(sb + 256);
            P.keyCap = keyCap;
            P.keyBase = (unsigned long long)k << sortSlotShift;
            P.rankBits = rankBits;
        }
    };
    anyFused = !supJobs.empty();
    for (const PlanSup& u : sups) anyFused |= u.n > 0;
    // Spilling pays where a task can outlast the others: not for launches
    // whose estimated work is below about 150 us of the whole GPU, and not for
    // sort mode, whose key count must not depend on it.  (Measured with and
    // without: at 66 us, 25 rules of a dense graph, 219 and 151 us; at 169 us,
    // 200 long rules, 805 and 778 us; at 188 us, 1,329 mined rules, 836 and
    // 924 us; at 4,500 us, 10,000 rules, 5.5 and 6.9 ms.)
    // Nor where no step's rows differ much in length, so that no task can
    // outlast the others by far (200 to 1,600 long rules on a uniform graph:
    // 0.83-5.9 ms with, 0.68-5.3 ms without).
    // What is given away costs several times its work, so sets with much work
    // but no long task lose: a prepared batch spills where that measured faster.
    double workNs = 0, skew = 0;
    for (int i = 0; i < nPlans; ++i) {
        workNs += pts[i].work * pts[i].scale;
        skew = std::max(skew, pts[i].skew);
    }
    spillAlways = c.spill == 2;
    spillable = maySpill && c.spill && nSort == 0 &&
                (spillAlways || (spillMeasured ? spillPays
                                     : skew >= kSpillSkew && workNs > 150e3 * std::max(c.grid, 1)));
    if (dCtl.cap == 0) ctlClean = false;
    dCtl.ensure(kCtlBytes, as);
    if (hCtl.cap == 0) {
        hCtl.ensure(kCtlBytes);
        std::memset(hCtl.p, 0, kCtlBytes);
    }
    hostSect[3] += host_ms() - tSect;
    tSect = host_ms();
    if (mayInline && nPlans <= kMaxPerPlan && !spillable && !bitmapWords && !blockWords && !heavyWords && !nSort &&
        std::all_of(pts.begin(), pts.end(), [](const PhaseTasks& t) { return t.chunk > 0; })) {
        // no upload at all: every launch brings its plan
        inl.resize(nPlans);
        for (int i = 0; i < nPlans; ++i) {
            InlineLaunch& L = inl[i];
            L.on = 1;
            L.beg = phases[i]->rootBeg;
            L.end = phases[i]->rootEnd;
            L.chunk = pts[i].chunk;
            L.publish = i + 1 == nPlans ? 1 : 0;
            L.ctl = dCtl.p;
            L.host = hCtl.p;
            fill(i, L.plan);
        }
        nTasks = (int)tasks.size();
        d2hBytes = 64;
        return;
    }
    if (sortTasks && tasks.size() > 1) {
        // longest (estimated device time) first, so the tail of the launch is short
        longest_first(tasks, cost, 0, tasks.size(), [&](size_t i) { return pts[tasks[i].plan].scale; });
    }
    nTasks = (int)tasks.size();
    planTaskEnd.clear();
    if (!sortTasks) {
        // one launch per plan: each plan's tasks stay contiguous, longest
        // first within the plan
        int32_t acc = 0;
        for (int i = 0; i < nPlans; ++i) {
            const int32_t b = acc, e = acc + (int32_t)pts[i].tasks.size();
            if (pts[i].chunk <= 0) longest_first(tasks, cost, (size_t)b, (size_t)e, [](size_t) { return 1.0; });
            planTaskEnd.push_back(acc = e);
        }
    }
    hostSect[4] += host_ms() - tSect;
    tSect = host_ms();
    size_t planBytes = (size_t)nPlans * sizeof(DevPlan);
    size_t taskBytes = (size_t)nTasks * sizeof(DevTask);
    const size_t sortBytes = ((size_t)nSort * sizeof(int32_t) + 15) & ~size_t(15);
    size_t blob = planBytes + taskBytes + sortBytes + (size_t)nSupJobs * sizeof(SupJob);
    hBlob.ensure(blob);
    parallel_for((size_t)nPlans, [&](size_t i) { fill((int)i, static_cast<DevPlan*>(hBlob.p)[i]); }, 64);
    std::memcpy(static_cast<char*>(hBlob.p) + planBytes, tasks.data(), taskBytes);
    if (nSort) std::memcpy(static_cast<char*>(hBlob.p) + planBytes + taskBytes, sortPlans.data(), nSort * sizeof(int32_t));
    if (nSupJobs)
        std::memcpy(static_cast<char*>(hBlob.p) + planBytes + taskBytes + sortBytes, supJobs.data(),
                    (size_t)nSupJobs * sizeof(SupJob));
    hTasks = std::move(tasks);   // kept for profiles and task-time learning
    hCost = std::move(cost);
    dBlob.ensure(blob, as);
    nResults = nPlans + extraResults;
    dResults.ensure((size_t)nResults * sizeof(unsigned long long), as);
    if (spillable) set_spill(true, s);
    hResults.ensure((size_t)nResults * sizeof(unsigned long long));
    ck(cudaMemcpyAsync(dBlob.p, hBlob.p, blob, cudaMemcpyHostToDevice, s), "H2D plans");
    dPlans = static_cast<const DevPlan*>(dBlob.p);
    dTasks = reinterpret_cast<const DevTask*>(static_cast<const char*>(dBlob.p) + planBytes);
    dSortSlots = nSort ? reinterpret_cast<const int32_t*>(static_cast<const char*>(dBlob.p) + planBytes + taskBytes)
                       : nullptr;
    dSupJobs = nSupJobs ? reinterpret_cast<const SupJob*>(static_cast<const char*>(dBlob.p) + planBytes + taskBytes +
                                                          sortBytes)
                        : nullptr;
    h2dBytes = blob;
    d2hBytes = (size_t)nResults * sizeof(unsigned long long) + 8;
    hostSect[5] += host_ms() - tSect;
}

namespace {
// Two-step memos keep the task builder's key ((p1, d1) and (p2, d2) in 32
// bits each); three-step keys set the top bit and pack 21 bits per step.
uint64_t memo_key(int p1, int d1, int p2, int d2, int p3 = -1, int d3 = 0) {
    if (p3 < 0) return ((uint64_t)(uint32_t)(p1 * 2 + d1) << 32) | (uint32_t)(p2 * 2 + d2);
    return (1ull << 63) | ((uint64_t)(uint32_t)(p1 * 2 + d1) << 42) | ((uint64_t)(uint32_t)(p2 * 2 + d2) << 21) |
           (uint64_t)(uint32_t)(p3 * 2 + d3);
}
}  // namespace

const SuffixMemo* Context::memo_for(const std::array<int, 6>& k) const {
    auto it = memos.find(memo_key(k[0], k[1], k[2], k[3], k[4], k[5]));
    return it == memos.end() ? nullptr : it->second.get();
}

bool Context::memo_known(const std::array<int, 6>& k) const {
    return memos.count(memo_key(k[0], k[1], k[2], k[3], k[4], k[5])) != 0;
}

void Context::ensure_memos(const std::vector<std::array<int, 6>>& keys, cudaStream_t s) {
    const HostIndex& h = hix;
    const int nHub = (int)h.hubOff.size();
    std::vector<std::array<int, 6>> fresh;
    for (const auto& k : keys) {
        const int p1 = k[0], p2 = k[2], p3 = k[4];
        const uint64_t key = memo_key(k[0], k[1], k[2], k[3], k[4], k[5]);
        if (memos.count(key)) continue;
        memos[key] = nullptr;
        const bool scan = p1 < 0;
        if (memoGain < 0 || (nHub == 0 && !scan) || p2 < 0 || p1 >= h.nPred || p2 >= h.nPred || p3 >= h.nPred) continue;
        if (p3 >= 0 && h.nPred >= (1 << 20)) continue;
        fresh.push_back(k);
    }
    if (fresh.empty()) return;
    // the rank domain of a memo: the rows of its last step's predicate in
    // the other direction (a scan memo's: the rows it scans)
    auto domain = [&](const std::array<int, 6>& k) -> int64_t {
        if (k[0] < 0) return h.pred_rows(k[2], k[3]);
        return k[4] >= 0 ? h.pred_rows(k[4], 1 - k[5]) : h.pred_rows(k[2], 1 - k[3]);
    };
    // the hub rows of (p1, d1) worth a memo, per new key, on host threads:
    // a row's candidates are what enumeration would visit from x on (its
    // own values, most of which may fail the next step's signature test,
    // and what they lead to)
    std::vector<std::vector<int32_t>> rowsOf(fresh.size());
    parallel_for(fresh.size(), [&](size_t i) {
        const int p1 = fresh[i][0], d1 = fresh[i][1], p2 = fresh[i][2], d2 = fresh[i][3];
        const int p3 = fresh[i][4], d3 = fresh[i][5];
        if (p1 < 0) {   // scan memos: one slot
            rowsOf[i].push_back(-1);
            return;
        }
        const int words = (int)((domain(fresh[i]) + 31) / 32);
        const double need = memoGain * words;
        // the count only grows: a row stops being summed once it qualifies
        // (a hub row's own values mostly do), and the degree array is made
        // only for a row that needs it
        const int32_t* deg = nullptr;
        for (int32_t r = h.predRow[d1][p1]; r < h.predRow[d1][p1 + 1]; ++r) {
            if (h.hubOf[d1][r] < 0) continue;
            double cand = (double)(h.rowBeg[d1][r + 1] - h.rowBeg[d1][r]);
            for (int32_t e = h.rowBeg[d1][r]; e < h.rowBeg[d1][r + 1] && cand < need; ++e) {
                if (!deg) deg = tasks->degrees(p3 >= 0 ? p3 : p2, p3 >= 0 ? d3 : d2);
                if (p3 < 0) {
                    cand += deg[h.val[d1][e]];
                } else {
                    const auto r2 = h.row_range(p2, d2, h.val[d1][e]);
                    for (int32_t e2 = r2.first; e2 < r2.second; ++e2) cand += 1.0 + deg[h.val[d2][e2]];
                }
            }
            if (cand >= need) rowsOf[i].push_back(r);
        }
    }, 1);
    // per memo slot: kMemoMaps bitmaps (two steps), or S1 and one count per rank
    auto slot_words = [&](const std::array<int, 6>& k) -> size_t {
        const size_t words = (size_t)((domain(k) + 31) / 32);
        return k[4] >= 0 ? words + (size_t)(domain(k) + 3) / 4 : kMemoMaps * words;
    };
    // within the memory budget, in key order: one device allocation holding
    // every new memo's hub table, then every new memo's bits
    const size_t tabBytes = ((size_t)nHub * 4 + 255) & ~size_t(255);
    std::vector<size_t> take, bitOff;
    size_t bitTotal = 0;
    for (size_t i = 0; i < fresh.size(); ++i) {
        const size_t bytes = tabBytes + rowsOf[i].size() * slot_words(fresh[i]) * 4;
        if (rowsOf[i].empty() || memoBytes + bytes > kMemoBudgetBytes) continue;
        memoBytes += bytes;
        take.push_back(i);
        bitOff.push_back(bitTotal);
        bitTotal += rowsOf[i].size() * slot_words(fresh[i]) * 4;
    }
    if (take.empty()) return;
    const size_t tabTotal = tabBytes * take.size();
    // one block per slice of a row's values, so that the paths of a long row
    // spread over the SMs
    constexpr int32_t kSlice = 64, kScanRows = 2048;
    size_t nJobs = 0;
    for (size_t i : take)
        for (int32_t r : rowsOf[i])
            nJobs += r < 0 ? (size_t)((domain(fresh[i]) + kScanRows - 1) / kScanRows)
                           : (size_t)((h.rowBeg[fresh[i][1]][r + 1] - h.rowBeg[fresh[i][1]][r] + kSlice - 1) / kSlice);
    // From the last arena, or a new one; the job list uses the room behind the
    // memos until they are built.  Stream-ordered: cudaMalloc and cudaFree wait
    // for every stream, and a server's launch that met new memos stalled for
    // 10-900 ms in them (p99 latency of 10,000 requests/s 100-730 ms where a
    // stall fell, 2 ms otherwise).
    const size_t need = (tabTotal + bitTotal + 255) & ~size_t(255);
    const size_t jobBytes = nJobs * sizeof(MemoJob);
    if (memoChunks.empty() || memoUsed + need + jobBytes > memoChunks.back()->cap) {
        auto chunk = std::make_unique<DevBuf>();
        size_t cap = std::max(need + jobBytes, kMemoArenaBytes);
        chunk->pooled = cudaMallocAsync(&chunk->p, cap, s) == cudaSuccess;   // never resized
        if (!chunk->pooled) {   // no room for an arena: what these memos need, as long as that fits
            cudaGetLastError();
            cap = need + jobBytes;
            ck(cudaMalloc(&chunk->p, cap), "cudaMalloc(memos)");
        }
        chunk->cap = cap;
        memoChunks.push_back(std::move(chunk));
        memoUsed = 0;
    }
    char* base = static_cast<char*>(memoChunks.back()->p) + memoUsed;
    memoUsed += need;
    MemoJob* const dJobs = reinterpret_cast<MemoJob*>(base + need);
    std::vector<int32_t> tabs(tabTotal / 4, -1);
    std::vector<MemoJob> all;
    std::vector<std::pair<uint64_t, std::unique_ptr<SuffixMemo>>> built;   // known once the device has them
    for (size_t t = 0; t < take.size(); ++t) {
        const size_t i = take[t];
        const int p1 = fresh[i][0], d1 = fresh[i][1], p2 = fresh[i][2], d2 = fresh[i][3];
        const int p3 = fresh[i][4], d3 = fresh[i][5];
        const int wo = (int)domain(fresh[i]);
        const int words = (wo + 31) / 32;
        const size_t stride = slot_words(fresh[i]);
        int32_t* tab = tabs.data() + t * (tabBytes / 4);
        uint32_t* bits = reinterpret_cast<uint32_t*>(base + tabTotal + bitOff[t]);
        auto m = std::make_unique<SuffixMemo>();
        m->rowHasMemo.assign((size_t)h.pred_rows(p1, d1), 0);
        const std::vector<int32_t>& rows = rowsOf[i];
        for (size_t j = 0; j < rows.size(); ++j) {
            if (p1 < 0) {
                for (int32_t b0 = 0; b0 < wo; b0 += kScanRows)
                    all.push_back(MemoJob{p2, d2, p2, d2, -1, words, -1, 0, wo, b0, std::min(wo, b0 + kScanRows), 0, bits});
                continue;
            }
            tab[h.hubOf[d1][rows[j]]] = (int32_t)j;
            m->rowHasMemo[(size_t)(rows[j] - h.predRow[d1][p1])] = 1;
            const int32_t len = h.rowBeg[d1][rows[j] + 1] - h.rowBeg[d1][rows[j]];
            for (int32_t b0 = 0; b0 < len; b0 += kSlice)
                all.push_back(MemoJob{p1, d1, p2, d2, rows[j], words, p3, d3, wo, b0, std::min(len, b0 + kSlice), 0,
                                      bits + j * stride});
        }
        m->tab = reinterpret_cast<const int32_t*>(base + t * tabBytes);
        m->bits = bits;
        m->words = words;
        m->wo = p3 >= 0 ? wo : 0;
        m->slots = (int)rows.size();
        built.emplace_back(memo_key(p1, d1, p2, d2, p3, d3), std::move(m));
    }
    ck(cudaMemcpyAsync(base, tabs.data(), tabTotal, cudaMemcpyHostToDevice, s), "H2D memo tables");
    ck(cudaMemsetAsync(base + tabTotal, 0, bitTotal, s), "clear memo bits");
    ck(cudaMemcpyAsync(dJobs, all.data(), all.size() * sizeof(MemoJob), cudaMemcpyHostToDevice, s), "H2D memo jobs");
    int maxWo = 0;
    for (const MemoJob& j : all)
        if (j.p3 >= 0) maxWo = std::max(maxWo, j.wo);
    ck(memo_build(dix, dJobs, (int)all.size(), maxWo, s), "memo build");
    ck(cudaStreamSynchronize(s), "memo build");   // memos are shared by every stream afterwards
    for (auto& m : built) memos[m.first] = std::move(m.second);
}

// Its buffer is stream-ordered also for staging that is not: cudaMalloc waits
// for every stream, and a call of several chunks takes one buffer (31 MB) each.
// Without room for it launches do not spill.
void Staged::set_spill(bool on, cudaStream_t s) {
    spillable = on;
    if (!on) {
        dSpill.release();
        return;
    }
    try {
        dSpill.ensure(spill_bytes(), s, true);
    } catch (const CudaError&) {
        cudaGetLastError();
        spillable = false;
    }
}

SpillArgs Staged::spill_args(int launch) const {
    SpillArgs a;
    if (!spillable) return a;
    char* p = static_cast<char*>(dSpill.p);
    a.ctl = reinterpret_cast<SpillCtl*>(static_cast<char*>(dCtl.p) + kSpillCtlAt) + launch;
    for (int k = 0; k < 2; ++k) {
        a.tasks[k] = reinterpret_cast<SpillTask*>(p + spill_part(k));
        a.recs[k] = reinterpret_cast<int32_t*>(p + spill_part(2 + k));
    }
    a.sups = reinterpret_cast<SpillSup*>(p + spill_part(4));
    a.rows = reinterpret_cast<uint32_t*>(p + spill_part(5));
    a.out = 0;
    a.always = spillAlways ? 1 : 0;
    return a;
}

// The launches that run what the one before spilled; the last may not spill.
void Staged::enqueue_follow_ups(Context& c, cudaStream_t s, unsigned long long* results, int* status,
                                unsigned long long* span, int launch) {
    if (!spillable) return;
    EngineProfile prof;
    prof.span = span;
    for (int k = 0; k < kFollowUps; ++k) {
        SpillArgs a = spill_args(launch);
        a.in = k;
        a.out = k + 1 < kFollowUps ? k + 1 : -1;
        ck(engine_launch(c.dix, dPlans, dTasks, 0, nullptr, results, status, c.grid, c.geom.block, s, &prof, a),
           "engine follow-up launch");
    }
}

void Staged::enqueue_sort(Context& c, cudaStream_t s, unsigned long long* results, int* status) {
    if (!nSort) return;
    char* base = static_cast<char*>(dSort.p);
    auto* cursor = reinterpret_cast<unsigned long long*>(base);
    auto* keys = reinterpret_cast<unsigned long long*>(base + 256);
    auto* tmp = keys + keyCap;
    auto* hist = reinterpret_cast<uint32_t*>(tmp + keyCap);
    ck(pairs_sort_count(keys, tmp, cursor, keyCap, sortSlotShift, dSortSlots, nSort, results, status,
                        hist, std::max(c.sms, 1) * 8, c.sortSet, s),
       "pair sort");
}

void Staged::restage(Context& c, cudaStream_t s) {
    if (!nSort) return;
    keyHint = *static_cast<const unsigned long long*>(hSort.p);
    const std::vector<const PhasePlan*> ph = inPhases;
    const std::vector<PlanSup> su = inSups;
    stage(c, ph, su, inSortTasks, s, inWalk, inWalkRule, inAllowSort);
}

void Staged::check_geometry(const Context& c) const {
    // plans are laid out for the shared pool of the block size they were
    // staged at; a larger block's pool starts with it, a smaller one's is
    // too short (and its larger grid would outrun the per-block tables)
    if (c.geom.block < stagedBlock)
        throw CudaError("the launch's block size (" + std::to_string(c.geom.block) +
                        " threads) is below the one the plans were staged for (" + std::to_string(stagedBlock) +
                        "); prepare the batch again after changing the block size");
}

// The block size of a launch of `tasks` tasks: larger blocks than the plans'
// while all tasks are resident at once.  They shorten each task, but half as
// many are resident: rules through hub rows with 2,000-4,800 tasks take 182 us
// on 256 threads and 333 us on 512; a rule with 95 tasks 28 and 26 us, a
// dense batch with 293 tasks 191 and 175 us.
static int few_task_block(const Context& c, int tasks) {
    return c.ruleBlock > c.geom.block && tasks <= c.sms * (1024 / c.ruleBlock) ? c.ruleBlock : c.geom.block;
}

void Staged::enqueue(Context& c, cudaStream_t s, int instr, int gridCap, unsigned long long budgetNs) {
    budgeted = false;
    if (!nPlans) return;
    check_geometry(c);
    ctlClean = false;
    ck(cudaMemsetAsync(dResults.p, 0, (size_t)nResults * sizeof(unsigned long long), s), "memset results");
    ck(cudaMemsetAsync(dCtl.p, 0, kCtlBytes, s), "memset ctl");
    if (bitmapWords) ck(cudaMemsetAsync(dBitmap.p, 0, bitmapWords * 4, s), "memset bitmap");
    if (heavyWords) ck(cudaMemsetAsync(dHeavy.p, 0, heavyWords * 4, s), "memset heavy rows");
    if (nSort) ck(cudaMemsetAsync(dSort.p, 0, 8, s), "memset key cursor");
    EngineProfile prof;
    if (instr >= 1) {
        dTaskNs.ensure((size_t)std::max(nTasks, 1) * 16, streamOrdered ? s : nullptr);
        prof.taskNs = static_cast<unsigned long long*>(dTaskNs.p);
    }
    if (instr >= 2) {
        dBytes.ensure(8, streamOrdered ? s : nullptr);
        ck(cudaMemsetAsync(dBytes.p, 0, 8, s), "memset bytes");
        prof.bytes = static_cast<unsigned long long*>(dBytes.p);
    }
    if (budgetNs && instr == 1) {
        dIncomplete.ensure((size_t)nPlans * sizeof(int), streamOrdered ? s : nullptr);
        hIncomplete.ensure((size_t)nPlans * sizeof(int));
        ck(cudaMemsetAsync(dIncomplete.p, 0, (size_t)nPlans * sizeof(int), s), "memset incomplete plans");
        prof.budgetNs = budgetNs;
        prof.incomplete = static_cast<int*>(dIncomplete.p);
        budgeted = true;
    }
    // few tasks: larger blocks (see few_task_block); launches that spill keep
    // the blocks of their follow-ups, timed ones those that costs are learnt for
    const int block = instr || gridCap > 0 || spillable ? c.geom.block : few_task_block(c, nTasks);
    int grid = std::max(1, std::min(nTasks, gridCap > 0 ? std::min(gridCap, c.grid) : c.grid));
    if (blockWords && (size_t)grid > blockRegions) throw CudaError("launch grid exceeds the block-row regions");
    ck(engine_launch(c.dix, dPlans, dTasks, nTasks, static_cast<int*>(dCtl.p),
                     static_cast<unsigned long long*>(dResults.p), static_cast<int*>(dCtl.p) + 1, grid,
                     block, s, instr ? &prof : nullptr, instr ? SpillArgs{} : spill_args()),
       "engine launch");
    if (!instr)
        enqueue_follow_ups(c, s, static_cast<unsigned long long*>(dResults.p), static_cast<int*>(dCtl.p) + 1, nullptr);
    ck(support_rows(c.dix, dPlans, dSupJobs, nSupJobs, static_cast<unsigned long long*>(dResults.p), s,
                    !instr && anyFused ? spill_args() : SpillArgs{}, c.sms),
       "fused support of split roots and spilled tasks");
    enqueue_sort(c, s, static_cast<unsigned long long*>(dResults.p), static_cast<int*>(dCtl.p) + 1);
}

void Staged::enqueue_per_plan(Context& c, cudaStream_t s) {
    if (!nPlans) return;
    check_geometry(c);
    if (!inl.empty()) {
        static_assert(kInlineWords * 4 == 64 && kSpillCtlAt >= kInlineWords * 4 && kCtlBytes > kInlineWords * 4,
                      "the ended blocks are counted behind the published words");
        if (!ctlClean) ck(cudaMemsetAsync(dCtl.p, 0, kCtlBytes, s), "memset ctl");
        ctlClean = false;   // until the launches are known to have ended (wait_published)
        inlSeq = inlSeq % 0x3fffffff + 1;
        for (InlineLaunch& L : inl) L.seq = inlSeq;
        int* ctl = static_cast<int*>(dCtl.p);
        for (int i = 0; i < nPlans; ++i) {
            EngineProfile prof;
            prof.span = reinterpret_cast<unsigned long long*>(static_cast<char*>(dCtl.p) + 16 + 16 * i);
            const int n = (inl[i].end - inl[i].beg + inl[i].chunk - 1) / inl[i].chunk;
            ck(engine_launch(c.dix, nullptr, nullptr, n, ctl + i,
                             reinterpret_cast<unsigned long long*>(static_cast<char*>(dCtl.p) + kPerPlanResults),
                             ctl + 2, std::max(1, std::min(n, c.grid)), c.geom.block, s, &prof, SpillArgs{}, &inl[i]),
               "engine launch");
        }
        return;
    }
    if (nPlans > kMaxPerPlan || (int)planTaskEnd.size() != nPlans) throw CudaError("bad per-plan staging");
    // control words: [0..1] task counters, [2] status (int), per plan two
    // u64 span words at byte 16 + 16 * i and its u64 result at
    // kPerPlanResults + 8 * i; all start at zero
    ctlClean = false;
    ck(cudaMemsetAsync(dCtl.p, 0, kCtlBytes, s), "memset ctl");
    if (bitmapWords) ck(cudaMemsetAsync(dBitmap.p, 0, bitmapWords * 4, s), "memset bitmap");
    if (heavyWords) ck(cudaMemsetAsync(dHeavy.p, 0, heavyWords * 4, s), "memset heavy rows");
    if (nSort) ck(cudaMemsetAsync(dSort.p, 0, 8, s), "memset key cursor");
    int* ctl = static_cast<int*>(dCtl.p);
    auto* results = reinterpret_cast<unsigned long long*>(static_cast<char*>(dCtl.p) + kPerPlanResults);
    for (int i = 0; i < nPlans; ++i) {
        const int32_t b = i ? planTaskEnd[i - 1] : 0, e = planTaskEnd[i];
        EngineProfile prof;
        prof.span = reinterpret_cast<unsigned long long*>(static_cast<char*>(dCtl.p) + 16 + 16 * i);
        const int grid = std::max(1, std::min(e - b, c.grid));
        if (blockWords && (size_t)grid > blockRegions) throw CudaError("launch grid exceeds the block-row regions");
        ck(engine_launch(c.dix, dPlans, dTasks + b, e - b, ctl + i, results, ctl + 2,
                         grid, c.geom.block, s, &prof, spill_args(i)),
           "engine launch");
        // each plan's spilled tasks before the next plan's launch: timed with
        // their own phase, and the lists and rows are free again (the rows of
        // fused supports once those are counted)
        enqueue_follow_ups(c, s, results, ctl + 2, prof.span, i);
        const bool last = i + 1 == nPlans;
        ck(support_rows(c.dix, dPlans, dSupJobs, last ? nSupJobs : 0, results, s,
                        anyFused ? spill_args(i) : SpillArgs{}, c.sms),
           "fused support of split roots and spilled tasks");
    }
    enqueue_sort(c, s, results, ctl + 2);
}

int Staged::max_launch_tasks() const {
    int most = 0;
    for (const InlineLaunch& L : inl) most = std::max(most, (L.end - L.beg + L.chunk - 1) / L.chunk);
    if (inl.empty())
        for (size_t i = 0; i < planTaskEnd.size(); ++i)
            most = std::max(most, planTaskEnd[i] - (i ? planTaskEnd[i - 1] : 0));
    return most;
}

// Waits for the control words of an inline launch: the flag behind them in
// host memory is a few us earlier than the stream's end.  Ends with the
// stream in any case (an error is the following synchronisation's to report).
void Staged::wait_published(cudaStream_t s) {
    if (inl.empty()) return;
    const volatile int* flag = static_cast<const volatile int*>(hCtl.p) + kInlineWords;
    for (unsigned spins = 0;; ++spins) {
        if (*flag == inlSeq) {
            std::atomic_thread_fence(std::memory_order_acquire);
            ctlClean = true;
            return;
        }
        if (spins % 4096 == 4095 && cudaStreamQuery(s) != cudaErrorNotReady) return;
    }
}

void Staged::download_spans(cudaStream_t s) {
    if (!nPlans || !inl.empty()) return;   // (an inline launch writes them itself)
    ck(cudaMemcpyAsync(hCtl.p, dCtl.p, 64, cudaMemcpyDeviceToHost, s), "D2H control words");
    download_cursor(s);
}

void compose(const RulePlan& rp, int64_t sup, int64_t body, double supMs, double confMs, GpuRuleResult* out) {
    *out = GpuRuleResult{};
    out->headSize = (int)clamp_int(rp.headSize);
    out->headSupport = (int)clamp_int(rp.headSupport);
    if (rp.status != kRuleOk) return;
    // FinalRule::setMeasures / setConfidence (CPU_01_nonparallel/FinalRule.cpp:19-41)
    int s = (int)clamp_int(sup), b = (int)clamp_int(body);
    out->support = s;
    out->headCoverage = out->headSize > 0 ? (double)s / (double)out->headSize : 0.0;
    out->bodySize = b;
    out->confidence = b > 0 ? (double)s / (double)b : 0.0;
    out->supportMs = supMs;
    out->confidenceMs = confMs;
}

namespace {

// One phase in its own launch (the plain per-rule form), timed by events.
int64_t run_one_phase(Context& c, const PhasePlan& ph, float* ms) {
    c.one.extraResults = 0;
    c.one.stage(c, {&ph}, {}, false, c.stream, c.ruleWalkBudget, kWalkPays);
    for (int attempt = 0;; ++attempt) {
        ck(cudaEventRecord(c.ev[0], c.stream), "event");
        c.one.enqueue(c, c.stream, 0);
        ck(cudaEventRecord(c.ev[1], c.stream), "event");
        c.one.download(c.stream);
        ck(cudaStreamSynchronize(c.stream), "engine");
        c.one.check_status();
        if (attempt > 0 || !c.one.sort_overflow()) break;
        c.one.restage(c, c.stream);   // the exact key count is known now
    }
    ck(cudaEventElapsedTime(ms, c.ev[0], c.ev[1]), "elapsed");
    return (int64_t)c.one.counts()[0];
}

// Runs fn with the context's launch block size and grid switched to those of
// a launch of `tasks` tasks, restoring them afterwards (also when fn throws).
// Only launches run under it: plans keep the batch geometry, whose shared
// pool is a prefix of the larger block's, so per-rule calls share the
// batch's cached walks and learnt costs (both keyed by plan signature).
template <class Fn>
void with_rule_block(Context& c, int tasks, Fn fn) {
    struct Restore {
        Context& c;
        int block, grid;
        ~Restore() { c.geom.block = block; c.grid = grid; }
    } restore{c, c.geom.block, c.grid};
    c.set_block(few_task_block(c, tasks));
    fn();
}

// Both phases of one rule, each in its own launch timed by its own events,
// issued back to back with one host synchronisation; a fused support takes
// no launch of its own.
int evaluate_parsed(Context& c, const Rule& rule, GpuRuleResult* out) {
    RulePlan rp = plan_rule(rule, c.hix, c.geom, c.fans());
    int64_t sup = rp.support.value, body = rp.body.value;
    float supMs = 0.f, confMs = 0.f;
    const bool runS = rp.status == kRuleOk && rp.support.how == kDevice;
    const bool runB = rp.status == kRuleOk && rp.body.how == kDevice;
    std::vector<PlanSup> sups;
    std::vector<const PhasePlan*> phases;
    // fused support (see prepare): the body-size launch also counts the
    // support, into per-plan result slot 1; the support takes no launch
    const bool fused = runS && runB && fusing(c) && fuses(rp);
    if (runS && !fused) phases.push_back(&rp.support);
    if (runB) phases.push_back(&rp.body);
    if (fused) {
        sups.resize(1);
        sups[0].n = 1;
        sups[0].pred[0] = rp.supFuse;   // (its slot, 0, comes after the one plan's own)
    }
    if (!phases.empty()) {
        // one upload, one launch per phase (each timed on the device), one download
        c.one.stage(c, phases, sups, false, c.stream, c.ruleWalkBudget, kWalkPays, true, true);
        for (int attempt = 0;; ++attempt) {
            with_rule_block(c, c.one.max_launch_tasks(), [&] { c.one.enqueue_per_plan(c, c.stream); });
            c.one.download_spans(c.stream);
            c.one.wait_published(c.stream);
            ck(c.one.inl.empty() || !c.one.ctlClean ? cudaStreamSynchronize(c.stream) : cudaSuccess, "engine");
            if (attempt > 0 || !c.one.sort_overflow()) break;
            c.one.restage(c, c.stream);   // the exact key count is known now
        }
        if (static_cast<const int*>(c.one.hCtl.p)[2] != 0)
            throw CudaError("engine reported internal status " + std::to_string(static_cast<const int*>(c.one.hCtl.p)[2]));
        int k = 0;
        if (runS && !fused) { sup = (int64_t)c.one.per_plan_count(k); supMs = (float)c.one.span_ms(k); ++k; }
        if (runB) { body = (int64_t)c.one.per_plan_count(k); confMs = (float)c.one.span_ms(k); }
        if (fused) sup = (int64_t)c.one.per_plan_count(1);   // counted by the body-size launch (supportMs 0)
    }
    compose(rp, sup, body, supMs, confMs, out);
    return 0;
}

// Counts of one rule restricted to slice `shard` of `nShards` of each device
// phase's roots (slices of about equal estimated work).  Support roots are
// head triples and body-size roots are rows of the seed atom keyed by one of
// the head's variables, so the slices' counts add up to the whole rule's:
// distinct (hS, hO) pairs of different roots never collide.  Which variable,
// and where the roots are cut, follows from the rule and the graph alone:
// each slice may be evaluated by another process.  Static parts count in slice
// 0 only.
void evaluate_shard(Context& c, const Rule& rule, int shard, int nShards, long long* counts) {
    RulePlan rp = plan_rule(rule, c.hix, c.geom, c.samples.get());   // (whatever this process's bothEnds)
    int64_t part[2] = {shard == 0 ? rp.support.value : 0, shard == 0 ? rp.body.value : 0};
    PhasePlan* phs[2] = {&rp.support, &rp.body};
    for (int k = 0; k < 2 && rp.status == kRuleOk; ++k) {
        PhasePlan& ph = *phs[k];
        if (ph.how != kDevice) continue;
        const std::vector<int32_t> cut = c.tasks->split_roots(ph, nShards);
        ph.rootBeg = cut[shard];
        ph.rootEnd = cut[shard + 1];
        part[k] = 0;
        float ms = 0.f;
        if (ph.rootEnd > ph.rootBeg) part[k] = run_one_phase(c, ph, &ms);
    }
    counts[0] = rp.status == kRuleOk ? part[0] : 0;
    counts[1] = rp.headSize;
    counts[2] = rp.headSupport;
    counts[3] = rp.status == kRuleOk ? part[1] : 0;
}

// Parses and plans n rules and stages their device phases.
// oneShot: for one run (the task builder then walks only what pays).
void prepare(Batch& b, Context& c, const char* const* rules, int n, int isJson, bool oneShot = false) {
    const double tStart = host_ms();
    b.c = &c;
    b.n = n;
    b.owner.clear();
    b.shared.clear();
    if (b.exec) { cudaGraphExecDestroy(b.exec); b.exec = nullptr; }
    if (b.graph) { cudaGraphDestroy(b.graph); b.graph = nullptr; }
    if ((int)b.rps.size() < n) b.rps.resize(n);   // every entry is written below
    b.parseStatus.assign(n, 0);
    b.hash.resize(2 * (size_t)n);   // per rule: support and body phase hashes
    uint64_t* const hash = b.hash.data();
    const bool fuse = fusing(c);
    // parsing, planning and hashing only read the graph and the
    // dictionaries: in parallel
    parallel_for((size_t)n, [&](size_t i) {
        RulePlan& rp = b.rps[i];
        if (!rules[i]) { b.parseStatus[i] = -1; return; }
        try {
            Rule r = isJson ? c.parser->parse_json(rules[i]) : c.parser->parse_text(rules[i]);
            rp = plan_rule(r, c.hix, c.geom, c.fans());
            if (rp.status == kRuleOk) {
                // (a fused support is only hashed if its plan turns out to be full)
                if (rp.support.how == kDevice && !(fuse && fuses(rp))) hash[2 * i] = phase_hash(rp.support);
                if (rp.body.how == kDevice) hash[2 * i + 1] = phase_hash(rp.body);
            }
        } catch (const RuleError&) {
            b.parseStatus[i] = -1;
        }
    }, 16);
    // fused support: a rule whose support its body-size plan can count (see
    // RulePlan::supFuse) gets no support plan when that plan keeps its pair
    // rows in shared memory (no global dedup bitmap, no forced mode); the
    // count lands in a result slot after the plans' own
    b.supOf.assign(n, -1);
    std::vector<const PhasePlan*>& phases = b.phases;
    std::vector<PlanSup>& sups = b.sups;
    phases.clear();
    sups.clear();
    phases.reserve(2 * (size_t)n);
    sups.reserve(2 * (size_t)n);
    int nFused = 0;
    // plans by hash, open addressing: {hash, plan}
    size_t slots = 64;
    while (slots < 4 * (size_t)n) slots *= 2;
    b.seen.assign(slots, -1);
    b.seenHash.resize(slots);
    for (int i = 0; i < n; ++i) {
        if (b.parseStatus[i] != 0) continue;
        RulePlan& rp = b.rps[i];
        if (rp.status != kRuleOk) continue;
        int bodyPlan = -1;
        for (int k : {1, 0}) {
            const PhasePlan& ph = k == 0 ? rp.support : rp.body;
            if (ph.how != kDevice || !(c.batchPhases & (1 << k))) continue;
            if (k == 0 && fuse && bodyPlan >= 0 && fuses(rp)) {
                PlanSup& u = sups[(size_t)bodyPlan];
                int j = 0;
                while (j < u.n && u.pred[j] != rp.supFuse) ++j;
                if (j < u.n) {   // one body under one head predicate again
                    b.supOf[i] = u.slot[j];
                    continue;
                }
                if (u.n < kMaxSupFused) {
                    u.pred[u.n] = rp.supFuse;
                    u.slot[u.n] = b.supOf[i] = nFused++;
                    ++u.n;
                    continue;
                }
                hash[2 * (size_t)i] = phase_hash(ph);
            }
            // identical computations (same plan and roots, e.g. one body under
            // several heads) run once; the others share the count
            // keyed by hash, confirmed by the full signature (plans are
            // zero-initialised, so equal signatures mean equal computations)
            const uint64_t h = hash[2 * (size_t)i + k];
            size_t at = (size_t)h & (slots - 1);
            int same = -1;
            for (; b.seen[at] >= 0; at = (at + 1) & (slots - 1))
                if (b.seenHash[at] == h && phase_equal(*phases[(size_t)b.seen[at]], ph)) {
                    same = b.seen[at];
                    break;
                }
            if (same >= 0) {
                b.shared.emplace_back(2 * i + k, same);
                if (k == 1) bodyPlan = same;
                continue;
            }
            b.seen[at] = (int)phases.size();
            b.seenHash[at] = h;
            if (k == 1) bodyPlan = (int)phases.size();
            phases.push_back(&ph);
            sups.emplace_back();
            b.owner.push_back(2 * i + k);
        }
    }
    // fused counts follow the plans' own result slots
    for (int i = 0; i < n; ++i)
        if (b.supOf[i] >= 0) b.supOf[i] += (int)phases.size();
    b.st.extraResults = nFused;
    if (!b.stream) ck(cudaStreamCreateWithFlags(&b.stream, cudaStreamNonBlocking), "cudaStreamCreate");
    if (!b.ev0) ck(cudaEventCreate(&b.ev0), "cudaEventCreate");
    if (!b.ev1) ck(cudaEventCreate(&b.ev1), "cudaEventCreate");
    // a one-shot batch walks a phase only when the walk costs less host time
    // than the phase is expected to take on the device; a prepared batch,
    // replayed many times, walks every phase the budget allows
    const double tPlanned = host_ms();
    b.st.stage(c, phases, sups, true, b.stream, b.walkBudget, oneShot ? kWalkPays : kWalkBudget);
    b.hostPlanMs = tPlanned - tStart;
    b.hostStageMs = host_ms() - tPlanned;
}

// Each rule's support and body size after a run: static values, the plans'
// own counts (shared ones included) and fused support counts.
void phase_counts(const Batch& b, std::vector<int64_t>& sup, std::vector<int64_t>& body) {
    sup.resize(b.n);
    body.resize(b.n);
    for (int i = 0; i < b.n; ++i) { sup[i] = b.rps[i].support.value; body[i] = b.rps[i].body.value; }
    const unsigned long long* cnt = b.st.counts();
    for (size_t k = 0; k < b.owner.size(); ++k) {
        int i = b.owner[k] / 2;
        if (b.owner[k] % 2 == 0) sup[i] = (int64_t)cnt[k];
        else body[i] = (int64_t)cnt[k];
    }
    for (const auto& sh : b.shared) {
        int i = sh.first / 2;
        if (sh.first % 2 == 0) sup[i] = (int64_t)cnt[sh.second];
        else body[i] = (int64_t)cnt[sh.second];
    }
    for (int i = 0; i < b.n && i < (int)b.supOf.size(); ++i)
        if (b.supOf[i] >= 0) sup[i] = (int64_t)cnt[b.supOf[i]];
}

void collect(const Batch& b, GpuRuleResult* out, int* status) {
    std::vector<int64_t> sup, body;
    phase_counts(b, sup, body);
    for (int i = 0; i < b.n; ++i) {
        if (status) status[i] = b.parseStatus[i];
        if (b.parseStatus[i] != 0) { out[i] = GpuRuleResult{}; continue; }
        compose(b.rps[i], sup[i], body[i], 0.0, 0.0, &out[i]);
    }
}

// Runs a prepared batch: optional L2 flush (untimed), then the device work
// between two events, then the result download.
void drop_graph(Batch& b) {
    if (b.exec) { cudaGraphExecDestroy(b.exec); b.exec = nullptr; }
    if (b.graph) { cudaGraphDestroy(b.graph); b.graph = nullptr; }
}

void run_batch(Batch& b, bool useGraph, size_t flushBytes, bool retried = false) {
    Context& c = *b.c;
    if (flushBytes) {
        b.flush.ensure(flushBytes);
        ck(cudaMemsetAsync(b.flush.p, (int)(b.lastMs * 7) & 0xff, flushBytes, b.stream), "flush");
    }
    if (useGraph && !b.exec && b.st.nPlans) {
        ck(cudaStreamBeginCapture(b.stream, cudaStreamCaptureModeThreadLocal), "capture");
        b.st.enqueue(c, b.stream, 0);
        ck(cudaStreamEndCapture(b.stream, &b.graph), "capture end");
        ck(cudaGraphInstantiate(&b.exec, b.graph, 0), "graph instantiate");
    }
    ck(cudaEventRecord(b.ev0, b.stream), "event");
    if (useGraph && b.exec) ck(cudaGraphLaunch(b.exec, b.stream), "graph launch");
    else b.st.enqueue(c, b.stream, 0);
    ck(cudaEventRecord(b.ev1, b.stream), "event");
    b.st.download(b.stream);
    ck(cudaStreamSynchronize(b.stream), "engine");
    b.st.check_status();
    if (!retried && b.st.sort_overflow()) {
        // sort-mode keys outgrew the estimate: stage again with the exact
        // count (the next runs fit) and run once more
        b.st.restage(c, b.stream);
        drop_graph(b);
        run_batch(b, useGraph, flushBytes, true);
        return;
    }
    float ms = 0.f;
    ck(cudaEventElapsedTime(&ms, b.ev0, b.ev1), "elapsed");
    b.lastMs = ms;
}

// Times a prepared batch's launch with and without spilling (the best of two
// runs after one) and keeps the faster way; spilling has to gain 3 %.  50
// rules on a graph with hubs: four sets 0.85-1.56 ms without and 1.10-1.81 ms
// with, two others 2.19 and 1.26 ms without, 1.59 and 1.15 ms with.  10,000
// rules: 3.35 and 3.56 ms without, 3.73 and 3.89 ms with; four other sets
// 6.2-7.2 ms without, 4.4-6.0 ms with.
void tune_spill(Batch& b) {
    Context& c = *b.c;
    if (c.spill != 1 || !b.st.nPlans || b.st.nSort) return;
    float best[2] = {0.f, 0.f};
    b.st.spillPays = false;
    for (int on = 0; on < 2; ++on) {
        b.st.set_spill(on != 0, b.stream);
        if (b.st.spillable != (on != 0)) return;   // no room for the buffer
        for (int run = 0; run < 3; ++run) {
            ck(cudaEventRecord(b.ev0, b.stream), "event");
            b.st.enqueue(c, b.stream, 0);
            ck(cudaEventRecord(b.ev1, b.stream), "event");
            b.st.download(b.stream);
            ck(cudaStreamSynchronize(b.stream), "tune");
            b.st.check_status();
            float ms = 0.f;
            ck(cudaEventElapsedTime(&ms, b.ev0, b.ev1), "elapsed");
            if (run == 1 || (run > 1 && ms < best[on])) best[on] = ms;
        }
    }
    b.st.spillPays = best[1] < 0.97f * best[0];
    if (!b.st.spillPays) b.st.set_spill(false, b.stream);
}

Context* as_ctx(void* p) { return static_cast<Context*>(p); }

}  // namespace
}  // namespace gr

using namespace gr;

namespace {

// The rest of a load, whichever source the index came from: the state built
// on the index, and its upload.
void finish_load(Context* c) {
    // GPU_RULES_MEMO3=0 switches the three-step suffix memos off,
    // GPU_RULES_FUSE_SUPPORT=0 the fused support of batches,
    // GPU_RULES_HUB_CLAIMS=0 the skipping of repeated leaf hub items
    if (const char* m = std::getenv("GPU_RULES_MEMO3")) c->memo3 = std::atoi(m) != 0;
    if (const char* f = std::getenv("GPU_RULES_FUSE_SUPPORT")) c->fuseSupport = std::atoi(f) != 0;
    if (const char* h = std::getenv("GPU_RULES_HUB_CLAIMS")) c->hubClaims = std::atoi(h) != 0;
    // GPU_RULES_SPILL=0: long tasks run to their end on one block; 2: every
    // task spills after its first round
    if (const char* h = std::getenv("GPU_RULES_SPILL")) c->spill = std::max(0, std::min(2, std::atoi(h)));
    // GPU_RULES_HOST_PROFILE=1: one stderr line of host-side times per one-shot batch
    // GPU_RULES_SORT_SET: keys a hash set of sort mode takes before its part of
    // the keys is split (fewer: more splits)
    if (const char* h = std::getenv("GPU_RULES_SORT_SET"))
        c->sortSet = std::max(16, std::min(kSortSetKeys, std::atoi(h)));
    if (const char* h = std::getenv("GPU_RULES_HOST_PROFILE")) c->hostProfile = std::atoi(h) != 0;
    c->tasks.reset(new TaskBuilder(c->hix));
    // GPU_RULES_PLAN_BOTH_ENDS=0: body sizes always from the head subject's end
    const char* ends = std::getenv("GPU_RULES_PLAN_BOTH_ENDS");
    c->bothEnds = !ends || std::atoi(ends) != 0;
    c->samples.reset(new FanSamples(c->hix));
    c->tasks->memoRows = [c](int p1, int d1, int p2, int d2, int p3, int d3,
                             double* cost) -> const std::vector<uint8_t>* {
        auto it = c->memos.find(memo_key(p1, d1, p2, d2, p3, d3));
        if (it == c->memos.end() || !it->second) return nullptr;
        // a memo word costs about a quarter of a candidate; an item itself is
        // a chain of dependent loads on one warp (exception lookups, searches
        // of the hub row for bound values; a three-step item also looks up
        // the rows its root reaches): c3 rule 963 (two steps, 4-word memos)
        // measured ~12 us of block time per root against ~7 ns per candidate
        *cost = it->second->words / 4.0 + (p3 >= 0 ? 512.0 : 256.0);
        return &it->second->rowHasMemo;
    };
    c->parser.reset(new RuleParser(c->ents, c->preds, c->prefixes));
    c->init_device();
    c->upload_index();
}

}  // namespace

extern "C" {

const char* gpu_last_error(void) { return g_lastError.c_str(); }

int gpu_query_vram(size_t* freeBytesOut, size_t* totalBytesOut) {
    size_t f = 0, t = 0;
    if (cudaMemGetInfo(&f, &t) != cudaSuccess) {
        cudaGetLastError();
        return -1;
    }
    if (freeBytesOut) *freeBytesOut = f;
    if (totalBytesOut) *totalBytesOut = t;
    return 0;
}

void* gpu_load_graph(const char* ttlPath) {
    if (!ttlPath) { set_error("gpu_load_graph: null path"); return nullptr; }
    Context* c = nullptr;
    try {
        c = new Context();
        std::vector<int32_t> spo;
        std::string err, text;
        if (!read_file(ttlPath, text, &err)) {
            set_error("Failed to parse TTL: " + std::string(ttlPath) + " (" + err + ")");
            delete c;
            return nullptr;
        }
        // one read of the file: the triples (several threads) and the rule
        // parser's prefix lines come from the same text
        parse_turtle_text_parallel(text, c->ents, c->preds, spo);
        c->prefixes = scan_rule_prefixes_text(text);
        std::string().swap(text);
        // GPU_RULES_MEMO_GAIN overrides the suffix-memo threshold (negative: no memos)
        if (const char* g = std::getenv("GPU_RULES_MEMO_GAIN")) c->memoGain = std::atof(g);
        // GPU_RULES_HUB_MIN_DEGREE overrides the hub-row threshold (0: no hub rows)
        int32_t hubMin = kHubMinDegree;
        if (const char* h = std::getenv("GPU_RULES_HUB_MIN_DEGREE")) hubMin = std::max(0, std::atoi(h));
        // the index is built on the device (GPU_RULES_INDEX_BUILD=host: on host threads)
        const char* where = std::getenv("GPU_RULES_INDEX_BUILD");
        if (where && std::strcmp(where, "host") == 0)
            c->hix = build_index(spo, (int32_t)c->ents.size(), (int32_t)c->preds.size(), hubMin);
        else
            c->hix = build_index_device(spo, (int32_t)c->ents.size(), (int32_t)c->preds.size(), hubMin);
        finish_load(c);
        return c;
    } catch (const std::exception& e) {
        set_error(std::string("gpu_load_graph error: ") + e.what());
        cudaGetLastError();
        delete c;
        return nullptr;
    }
}

void* gpu_load_index(const char* path) {
    if (!path) { set_error("gpu_load_index: null path"); return nullptr; }
    Context* c = nullptr;
    try {
        c = new Context();
        std::string err;
        if (!load_graph_file(path, c->ents, c->preds, c->prefixes, c->hix, &err)) {
            set_error(err);
            delete c;
            return nullptr;
        }
        if (const char* g = std::getenv("GPU_RULES_MEMO_GAIN")) c->memoGain = std::atof(g);
        finish_load(c);
        return c;
    } catch (const std::exception& e) {
        set_error(std::string("gpu_load_index error: ") + e.what());
        cudaGetLastError();
        delete c;
        return nullptr;
    }
}

int gpu_save_index(void* ctx, const char* path) {
    if (!ctx || !path) return -1;
    Context& c = *as_ctx(ctx);
    std::string err;
    if (!save_graph_file(path, c.ents, c.preds, c.prefixes, c.hix, &err)) {
        set_error(err);
        return -1;
    }
    return 0;
}

void gpu_free_graph(void* ctx) {
    if (!ctx) return;
    delete as_ctx(ctx);
}

int gpu_evaluate_rule(void* ctx, const char* ruleText, GpuRuleResult* out) {
    if (!ctx || !ruleText || !out) return -1;
    *out = GpuRuleResult{};
    Context& c = *as_ctx(ctx);
    try {
        cudaSetDevice(c.device);
        Rule r = c.parser->parse_text(ruleText);
        return evaluate_parsed(c, r, out);
    } catch (const std::exception& e) {
        set_error(std::string("gpu_evaluate_rule error: ") + e.what());
        *out = GpuRuleResult{};
        return -1;
    }
}

int gpu_evaluate_rule_json(void* ctx, const char* ruleJson, GpuRuleResult* out) {
    if (!ctx || !ruleJson || !out) return -1;
    *out = GpuRuleResult{};
    Context& c = *as_ctx(ctx);
    try {
        cudaSetDevice(c.device);
        Rule r = c.parser->parse_json(ruleJson);
        return evaluate_parsed(c, r, out);
    } catch (const std::exception& e) {
        set_error(std::string("gpu_evaluate_rule_json error: ") + e.what());
        *out = GpuRuleResult{};
        return -1;
    }
}

int gpu_evaluate_rules_batch(void* ctx, const char* const* rules, int n, int isJson,
                             GpuRuleResult* out, int* status, double* deviceMs) {
    if (!ctx || n < 0 || (n > 0 && (!rules || !out))) return -1;
    Context& c = *as_ctx(ctx);
    if (deviceMs) *deviceMs = 0.0;
    try {
        cudaSetDevice(c.device);
        // Pipelined: chunk k+1 is parsed, planned and staged on the host
        // while chunk k runs on the device (each chunk on its own stream).
        // automatic: up to 6 chunks of at least 1,667 rules (c3, 10,000 rules:
        // 1, 2, 4, 6, 8 and 12 chunks measured 53.6, 36.3, 29.0, 27.8, 30.0
        // and 34.1 ms a call)
        const int K = c.batchChunks > 0 ? std::max(1, std::min(c.batchChunks, std::max(n, 1)))
                                        : std::max(1, std::min(6, (n + 1666) / 1667));
        while ((int)c.pipe.size() < K) c.pipe.push_back(new Batch());
        const double t0 = host_ms();
        double planMs = 0, stageMs = 0;
        for (int k = 0; k < K; ++k) {
            const int lo = (int)((long long)n * k / K), hi = (int)((long long)n * (k + 1) / K);
            Batch& b = *c.pipe[k];
            prepare(b, c, rules + lo, hi - lo, isJson, true);
            planMs += b.hostPlanMs;
            stageMs += b.hostStageMs;
            ck(cudaEventRecord(b.ev0, b.stream), "event");
            b.st.enqueue(c, b.stream, 0);
            ck(cudaEventRecord(b.ev1, b.stream), "event");
            b.st.download(b.stream);
        }
        const double t1 = host_ms();
        float span = 0.f;
        for (int k = 0; k < K; ++k) {
            Batch& b = *c.pipe[k];
            ck(cudaStreamSynchronize(b.stream), "engine");
            b.st.check_status();
            if (b.st.sort_overflow()) {   // run this chunk again with the exact key count
                b.st.restage(c, b.stream);
                ck(cudaEventRecord(b.ev0, b.stream), "event");
                b.st.enqueue(c, b.stream, 0);
                ck(cudaEventRecord(b.ev1, b.stream), "event");
                b.st.download(b.stream);
                ck(cudaStreamSynchronize(b.stream), "engine");
                b.st.check_status();
            }
            float ms = 0.f;
            ck(cudaEventElapsedTime(&ms, c.pipe[0]->ev0, b.ev1), "elapsed");
            span = std::max(span, ms);
            if (c.hostProfile) {
                float own = 0.f, at = 0.f;
                ck(cudaEventElapsedTime(&own, b.ev0, b.ev1), "elapsed");
                ck(cudaEventElapsedTime(&at, c.pipe[0]->ev0, b.ev0), "elapsed");
                std::fprintf(stderr, "[gpu_rules]   chunk %d: %d rules, %d tasks, enqueued at %.2f ms, %.2f ms on the device\n",
                             k, b.n, b.st.nTasks, (double)at, (double)own);
            }
            const int lo = (int)((long long)n * k / K);
            collect(b, out + lo, status ? status + lo : nullptr);
        }
        if (deviceMs) *deviceMs = span;
        if (c.hostProfile) {
            double sect[6] = {0, 0, 0, 0, 0, 0};
            for (int k = 0; k < K; ++k)
                for (int j = 0; j < 6; ++j) {
                    sect[j] += c.pipe[k]->st.hostSect[j];
                    c.pipe[k]->st.hostSect[j] = 0.0;
                }
            std::fprintf(stderr, "[gpu_rules] batch of %d in %d chunks: parse+plan %.2f ms, staging %.2f ms "
                         "(dedup %.2f, memos %.2f, tasks %.2f, plans %.2f, order %.2f, upload %.2f), enqueue loop "
                         "%.2f ms, wait+collect %.2f ms, device span %.2f ms\n",
                         n, K, planMs, stageMs, sect[0], sect[1], sect[2], sect[3], sect[4], sect[5],
                         t1 - t0 - planMs - stageMs, host_ms() - t1, (double)span);
        }
        return 0;
    } catch (const std::exception& e) {
        set_error(std::string("gpu_evaluate_rules_batch error: ") + e.what());
        // no chunk may still be writing into the reused buffers, and the
        // caller sees no partial results
        for (Batch* b : c.pipe)
            if (b && b->stream) cudaStreamSynchronize(b->stream);
        cudaGetLastError();
        for (int i = 0; i < n; ++i) {
            out[i] = GpuRuleResult{};
            if (status) status[i] = -1;
        }
        return -1;
    }
}

void* gpu_batch_prepare(void* ctx, const char* const* rules, int n, int isJson) {
    if (!ctx || n < 0 || (n > 0 && !rules)) return nullptr;
    Context& c = *as_ctx(ctx);
    Batch* b = nullptr;
    try {
        cudaSetDevice(c.device);
        b = new Batch();
        b->walkBudget = 4.0e7;   // prepared once, replayed many times
        b->st.spillMeasured = true;
        prepare(*b, c, rules, n, isJson);
        ck(cudaStreamSynchronize(b->stream), "stage");
        return b;
    } catch (const std::exception& e) {
        set_error(std::string("gpu_batch_prepare error: ") + e.what());
        delete b;
        return nullptr;
    }
}

int gpu_batch_run(void* batch, long long flushBytes, GpuRuleResult* out, int* status, double* deviceMs) {
    if (!batch) return -1;
    Batch& b = *static_cast<Batch*>(batch);
    try {
        cudaSetDevice(b.c->device);
        run_batch(b, true, flushBytes > 0 ? (size_t)flushBytes : 0);
        if (out) collect(b, out, status);
        if (deviceMs) *deviceMs = b.lastMs;
        return 0;
    } catch (const std::exception& e) {
        set_error(std::string("gpu_batch_run error: ") + e.what());
        return -1;
    }
}

int gpu_batch_counts(void* batch, long long* counts, int* status) {
    if (!batch || !counts) return -1;
    const Batch& b = *static_cast<const Batch*>(batch);
    std::vector<int64_t> sup, body;
    phase_counts(b, sup, body);
    for (int i = 0; i < b.n; ++i) {
        const RulePlan& rp = b.rps[i];
        const bool ok = b.parseStatus[i] == 0;
        const bool run = ok && rp.status == kRuleOk;
        counts[4 * i + 0] = run ? sup[i] : 0;
        counts[4 * i + 1] = ok ? rp.headSize : 0;
        counts[4 * i + 2] = ok ? rp.headSupport : 0;
        counts[4 * i + 3] = run ? body[i] : 0;
        if (status) status[i] = b.parseStatus[i];
    }
    return 0;
}

int gpu_evaluate_rule_shard(void* ctx, const char* ruleText, int shard, int nShards, long long* counts) {
    if (!ctx || !ruleText || !counts || nShards < 1 || shard < 0 || shard >= nShards) return -1;
    Context& c = *static_cast<Context*>(ctx);
    try {
        cudaSetDevice(c.device);
        evaluate_shard(c, c.parser->parse_text(ruleText), shard, nShards, counts);
        return 0;
    } catch (const std::exception& e) {
        set_error(std::string("gpu_evaluate_rule_shard error: ") + e.what());
        return -1;
    }
}

int gpu_batch_info(void* batch, long long* plans, long long* tasks, long long* h2dBytes, long long* d2hBytes) {
    if (!batch) return -1;
    Batch& b = *static_cast<Batch*>(batch);
    if (plans) *plans = b.st.nPlans;
    if (tasks) *tasks = b.st.nTasks;
    if (h2dBytes) *h2dBytes = (long long)b.st.h2dBytes;
    if (d2hBytes) *d2hBytes = (long long)b.st.d2hBytes;
    return 0;
}

int gpu_batch_kernels(void* batch) {
    if (!batch) return -1;
    return static_cast<const Batch*>(batch)->st.kernels_per_enqueue();
}

int gpu_batch_dedup(void* batch, int* modes, long long* sortKeys) {
    if (!batch || !modes) return -1;
    const Batch& b = *static_cast<const Batch*>(batch);
    for (int i = 0; i < b.n; ++i) modes[i] = -1;
    // the body-size phase (owner rule * 2 + 1) of each rule whose body size
    // counts pairs on the device
    auto put = [&](int owner, int plan) {
        if (owner % 2 != 1 || plan < 0 || plan >= (int)b.st.dedup.size() || plan >= (int)b.phases.size()) return;
        if (b.phases[plan]->plan.mode == kPairs) modes[owner / 2] = b.st.dedup[plan];
    };
    for (size_t k = 0; k < b.owner.size(); ++k) put(b.owner[k], (int)k);
    for (const auto& sh : b.shared) put(sh.first, sh.second);
    if (sortKeys) *sortKeys = b.st.nSort ? (long long)*static_cast<const unsigned long long*>(b.st.hSort.p) : 0;
    return 0;
}

int gpu_batch_count_bytes(void* batch, unsigned long long* bytes) {
    return gpu_batch_profile(batch, bytes, nullptr, nullptr, 0);
}

int gpu_batch_profile(void* batch, unsigned long long* bytes, unsigned long long* taskNs, int* taskInfo,
                      long long maxTasks) {
    if (!batch) return -1;
    Batch& b = *static_cast<Batch*>(batch);
    try {
        cudaSetDevice(b.c->device);
        if (bytes) *bytes = 0;
        if (!b.st.nPlans) return 0;
        b.st.enqueue(*b.c, b.stream, 2);
        unsigned long long by = 0;
        ck(cudaMemcpyAsync(&by, b.st.dBytes.p, 8, cudaMemcpyDeviceToHost, b.stream), "D2H bytes");
        long long n = std::min<long long>(maxTasks, b.st.nTasks);
        if (taskNs && n > 0)
            ck(cudaMemcpyAsync(taskNs, b.st.dTaskNs.p, (size_t)n * 16, cudaMemcpyDeviceToHost, b.stream), "D2H task times");
        ck(cudaStreamSynchronize(b.stream), "profile");
        if (bytes) *bytes = by;
        if (taskInfo)
            for (long long t = 0; t < n; ++t) {
                const DevTask& tk = b.st.hTasks[t];
                taskInfo[3 * t] = b.owner[tk.plan];
                taskInfo[3 * t + 1] = tk.beg;
                taskInfo[3 * t + 2] = tk.end;
            }
        return 0;
    } catch (const std::exception& e) {
        set_error(std::string("gpu_batch_profile error: ") + e.what());
        return -1;
    }
}

int gpu_batch_autotune(void* batch, int rounds) {
    if (!batch || rounds < 0) return -1;
    Batch& b = *static_cast<Batch*>(batch);
    try {
        Context& c = *b.c;
        cudaSetDevice(c.device);
        for (int r = 0; r < rounds && b.st.nPlans; ++r) {
            b.st.enqueue(c, b.stream, 1);
            std::vector<unsigned long long> ns(2 * (size_t)b.st.nTasks);
            ck(cudaMemcpyAsync(ns.data(), b.st.dTaskNs.p, ns.size() * 8, cudaMemcpyDeviceToHost, b.stream), "D2H task times");
            ck(cudaStreamSynchronize(b.stream), "autotune");
            c.tasks->learn(b.phases, b.st.hTasks, b.st.hCost, ns.data(), c.grid);
            drop_graph(b);
            b.st.stage(c, b.phases, b.sups, true, b.stream, b.walkBudget);
            ck(cudaStreamSynchronize(b.stream), "restage");
        }
        if (rounds > 0) tune_spill(b);
        return 0;
    } catch (const std::exception& e) {
        set_error(std::string("gpu_batch_autotune error: ") + e.what());
        return -1;
    }
}

int gpu_set_option(void* ctx, const char* name, long long value) {
    if (!ctx || !name) return -1;
    Context& c = *as_ctx(ctx);
    std::string n(name);
    if (n == "block") return c.set_block((int)value) ? 0 : -1;
    if (n == "task_target" && value >= 0) { c.tasks->forceTarget = (double)value; return 0; }
    if (n == "walk_threshold" && value >= 0) { c.tasks->walkThreshold = (double)value; return 0; }
    if (n == "serve_lanes" && (value == 0 || value == 1)) { c.serveLanes = (int)value; return 0; }
    if (n == "rule_walk_budget" && value >= 0) { c.ruleWalkBudget = (double)value; return 0; }
    if (n == "batch_chunks" && value >= 0 && value <= 16) { c.batchChunks = (int)value; return 0; }
    if (n == "rule_block" && (value == 0 || value == 128 || value == 256 || value == 512)) {
        c.ruleBlock = (int)value;
        return 0;
    }
    if (n == "serve_heavy_share" && value >= 1 && value <= 16) { c.serveHeavyShare = (int)value; return 0; }
    if (n == "serve_heavy_us" && value >= 0) { c.serveHeavyNs = 1e3 * (double)value; return 0; }
    if (n == "serve_deadline_us" && value >= 0) { c.serveDeadlineNs = 1e3 * (double)value; return 0; }
    if (n == "serve_max_us" && value >= 0) { c.serveMaxNs = 1e3 * (double)value; return 0; }
    if (n == "batch_phases" && value >= 1 && value <= 3) { c.batchPhases = (int)value; return 0; }
    if (n == "dedup_budget" && value >= 4096) { c.dedupBudget = (size_t)value; return 0; }
    if (n == "dedup_mode" && (value == 0 || value == kDedupRows || value == kDedupBlockRows || value == kDedupSort)) {
        c.dedupForce = (int)value;
        return 0;
    }
    return -1;
}

void gpu_batch_free(void* batch) {
    delete static_cast<Batch*>(batch);
}

int gpu_graph_stats(void* ctx, long long* entities, long long* predicates, long long* triples) {
    if (!ctx) return -1;
    Context& c = *as_ctx(ctx);
    if (entities) *entities = (long long)c.hix.nEnt;
    if (predicates) *predicates = (long long)c.hix.nPred;
    if (triples) *triples = (long long)c.hix.nTriples;
    return 0;
}

int gpu_graph_predicate(void* ctx, long long index, char* name, int capacity, long long* triples) {
    if (!ctx) return -1;
    Context& c = *as_ctx(ctx);
    if (index < 0 || index >= (long long)c.preds.size()) return -1;
    const std::string& s = c.preds.names[(size_t)index];
    if (triples) *triples = (long long)c.hix.pred_size((int32_t)index);
    if (name && capacity > 0) {
        const size_t n = std::min(s.size(), (size_t)capacity - 1);
        std::memcpy(name, s.data(), n);
        name[n] = 0;
    }
    return (int)s.size();
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Evaluation without device allocation.
//
// Some callers cannot call cudaMalloc while they evaluate rules: a host
// framework that owns a fixed device-memory budget and forbids allocation at
// request time, a serving loop that must not hit cudaMalloc/cudaFree (both can
// synchronise the whole device and stall concurrent work), or code that runs
// between other libraries' stream-ordered work and must not change the
// device's memory map.  gpu_evaluate_rule_noalloc serves them: it evaluates a
// rule exactly like gpu_evaluate_rule (one launch per phase, same results)
// but takes every per-call device buffer (plan, tasks, task counter, status
// word, result counter and, for very large hO domains, the pair bitmap) from
// the fixed array below instead of allocating.
//
// The array is a file-scope __device__ object of kNoAllocScratchBytes; every
// GPU that loads this library holds it until the process exits.  Host code
// cannot use the array's name as a device address, so the first call on each
// device (with that device current) looks the address up with
// cudaGetSymbolAddress and caches it; make that first call before any stream
// capture.  All calls share the array and it keeps the previous call's
// contents, so each call clears the parts that must start at zero.  Calls
// that overlap on the GPU (from several threads, contexts or streams of the
// same device) race on the array and must be serialised by the caller.
namespace gr {
namespace {
constexpr size_t kNoAllocScratchBytes = 8u << 20;   // 8 MiB
constexpr size_t kNoAllocHeader = 256;               // [0,8) counter+status, [64,72) result
constexpr int kNoAllocMaxDevices = 64;
}  // namespace
}  // namespace gr

static __device__ __align__(256) unsigned char g_noallocScratch[gr::kNoAllocScratchBytes];

namespace gr {
namespace {

std::mutex g_noallocMu;
void* g_noallocAddr[kNoAllocMaxDevices] = {};

// Device address of the scratch array on `dev` (which must be current).
void* noalloc_scratch(int dev) {
    if (dev < 0 || dev >= kNoAllocMaxDevices) throw CudaError("device ordinal out of range");
    std::lock_guard<std::mutex> lk(g_noallocMu);
    if (!g_noallocAddr[dev]) {
        void* p = nullptr;
        ck(cudaGetSymbolAddress(&p, g_noallocScratch), "cudaGetSymbolAddress(scratch)");
        g_noallocAddr[dev] = p;
    }
    return g_noallocAddr[dev];
}

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// A phase's tasks and its place in the scratch array.
struct NoallocPhase {
    std::vector<DevTask> tasks;
    size_t taskOff = 0, bitmapOff = 0, bitmapWords = 0, need = 0;
    NoallocPhase(Context& c, const PhasePlan& ph) {
        if (ph.how != kDevice) return;
        std::vector<PhaseTasks> pts;
        c.tasks->build({&ph}, c.grid, false, pts);
        tasks = std::move(pts[0].tasks);
        taskOff = align256(kNoAllocHeader + sizeof(DevPlan));
        bitmapOff = align256(taskOff + tasks.size() * sizeof(DevTask));
        if (ph.needsGlobalBitmap)
            bitmapWords = (size_t)(ph.rootEnd - ph.rootBeg) * (size_t)std::max(ph.plan.rowWords, 1);
        need = bitmapOff + bitmapWords * 4;
    }
};

int64_t run_phase_noalloc(Context& c, const PhasePlan& ph, const NoallocPhase& np, char* scratch, float* ms) {
    DevPlan plan = ph.plan;
    const std::vector<DevTask>& tasks = np.tasks;
    const size_t planOff = kNoAllocHeader, taskOff = np.taskOff, bitmapOff = np.bitmapOff, bitmapWords = np.bitmapWords;
    if (np.need > kNoAllocScratchBytes)
        throw CudaError("rule needs " + std::to_string(np.need) + " bytes of scratch; the no-allocation limit is " +
                        std::to_string(kNoAllocScratchBytes) + " bytes");
    plan.resultSlot = 0;
    plan.gBitmap = bitmapWords ? reinterpret_cast<uint32_t*>(scratch + bitmapOff) : nullptr;
    plan.gRowBase = bitmapWords ? ph.rootBeg : 0;
    int* ctl = reinterpret_cast<int*>(scratch);
    unsigned long long* result = reinterpret_cast<unsigned long long*>(scratch + 64);
    ck(cudaMemcpyAsync(scratch + planOff, &plan, sizeof(DevPlan), cudaMemcpyHostToDevice, c.stream), "H2D plan");
    if (!tasks.empty())
        ck(cudaMemcpyAsync(scratch + taskOff, tasks.data(), tasks.size() * sizeof(DevTask), cudaMemcpyHostToDevice,
                           c.stream), "H2D tasks");
    ck(cudaMemsetAsync(scratch, 0, kNoAllocHeader, c.stream), "clear header");
    if (bitmapWords) ck(cudaMemsetAsync(scratch + bitmapOff, 0, bitmapWords * 4, c.stream), "clear bitmap");
    ck(cudaEventRecord(c.ev[2], c.stream), "event");
    int grid = std::max(1, std::min((int)tasks.size(), c.grid));
    ck(engine_launch(c.dix, reinterpret_cast<const DevPlan*>(scratch + planOff),
                     reinterpret_cast<const DevTask*>(scratch + taskOff), (int)tasks.size(), ctl, result, ctl + 1,
                     grid, c.geom.block, c.stream, nullptr), "engine launch");
    ck(cudaEventRecord(c.ev[3], c.stream), "event");
    unsigned long long count = 0;
    int st[2] = {0, 0};
    ck(cudaMemcpyAsync(&count, result, sizeof(count), cudaMemcpyDeviceToHost, c.stream), "D2H result");
    ck(cudaMemcpyAsync(st, ctl, sizeof(st), cudaMemcpyDeviceToHost, c.stream), "D2H status");
    ck(cudaStreamSynchronize(c.stream), "engine");
    if (st[1] != 0) throw CudaError("engine reported internal status " + std::to_string(st[1]));
    ck(cudaEventElapsedTime(ms, c.ev[2], c.ev[3]), "elapsed");
    return (int64_t)count;
}

}  // namespace
}  // namespace gr

extern "C" int gpu_evaluate_rule_noalloc(void* ctx, const char* ruleText, GpuRuleResult* out) {
    if (!ctx || !ruleText || !out) return -1;
    *out = GpuRuleResult{};
    Context& c = *as_ctx(ctx);
    try {
        ck(cudaSetDevice(c.device), "cudaSetDevice");
        char* scratch = static_cast<char*>(noalloc_scratch(c.device));
        Rule r = c.parser->parse_text(ruleText);
        RulePlan rp = plan_rule(r, c.hix, c.geom, c.fans());
        NoallocPhase ns(c, rp.support), nb(c, rp.body);
        if (ns.need > kNoAllocScratchBytes || nb.need > kNoAllocScratchBytes) {
            // a plan made for speed may need more memory (a larger hO domain,
            // more tasks): what the array holds depends on the plain one
            rp = plan_rule(r, c.hix, c.geom, nullptr, false);
            ns = NoallocPhase(c, rp.support);
            nb = NoallocPhase(c, rp.body);
        }
        int64_t sup = rp.support.value, body = rp.body.value;
        float supMs = 0.f, confMs = 0.f;
        if (rp.status == kRuleOk && rp.support.how == kDevice) sup = run_phase_noalloc(c, rp.support, ns, scratch, &supMs);
        if (rp.status == kRuleOk && rp.body.how == kDevice) body = run_phase_noalloc(c, rp.body, nb, scratch, &confMs);
        compose(rp, sup, body, supMs, confMs, out);
        return 0;
    } catch (const std::exception& e) {
        set_error(std::string("gpu_evaluate_rule_noalloc error: ") + e.what());
        *out = GpuRuleResult{};
        return -1;
    }
}
