// planner.hpp — rule -> device plans (support phase and body-size phase).
#pragma once
#include <atomic>
#include <cstdint>
#include <memory>
#include <shared_mutex>
#include <unordered_map>
#include <utility>
#include <vector>

#include "common.hpp"
#include "index.hpp"
#include "rules.hpp"

namespace gr {

enum RuleStatus : int32_t {
    kRuleOk = 0,
    kRuleUnsupported = 1,   // more than 8 body atoms, 16 variables or too many constants
};

// How a phase's count is obtained.
enum PhaseHow : int32_t {
    kStatic = 0,      // known on the host (value in `value`)
    kDevice = 1,      // plan + tasks on the device
};

struct PhasePlan {
    PhasePlan() {}                      // (the plan of a static phase stays unset)
    int32_t how = kStatic;
    int64_t value = 0;
    DevPlan plan;
    int32_t rootBeg = 0, rootEnd = 0;   // root range (edges or rows)
    bool needsGlobalBitmap = false;     // kPairs whose hO domain exceeds the shared bitmap
    double estCost = 0.0;               // autotuner estimate (relative units)
};

struct RulePlan {
    int32_t status = kRuleOk;
    int64_t headSize = 0, headSupport = 0;
    PhasePlan support, body;
    // >= 0 when the support is the number of head triples (hS, supFuse, hO),
    // hS != hO, among the body-size phase's (hS, hO) pairs: both head terms
    // are distinct variables and no body atom can ground to the head triple
    // (the support plan has no used-triple test), so a body-size plan that
    // keeps its pair rows can count the support too (fused support).
    int32_t supFuse = -1;
};

// Where a kPairs plan ranks hO: the rows of (pred, dir) in the returned
// pair (the step binding hO looks its value up there).
std::pair<int32_t, int32_t> ho_domain(const DevPlan& P);

// Per predicate and direction (pred * 2 + dir): the mean row length that a
// random edge sees, sum(d^2) / sum(d).
std::vector<double> size_biased_fans(const HostIndex& ix);

// Mean row lengths of predicate transitions, estimated from a few evenly
// spaced edges (or rows) of the first predicate and cached: what the planner
// compares grounding orders by.  Safe to call from several threads.
class FanSamples {
public:
    struct Fan {
        float all = 0.f, capped = 0.f;   // rows above kHubMinDegree edges count as kHubMinDegree in `capped`
    };
    explicit FanSamples(const HostIndex& ix);
    const HostIndex& index() const { return ix_; }
    // size-biased row length of (pred, dir)
    double biased(int32_t pred, int dir) const { return biased_[(size_t)pred * 2 + (size_t)dir]; }
    // transitions sampled so far
    size_t sampled() const { return sampled_; }
    // row length under (p1, d1) of the value an edge of (p0, d0) leads to
    Fan edges(int32_t p0, int d0, int32_t p1, int d1) { return get(p0, d0, p1, d1, true); }
    // row length under (p1, d1) of a row key of (p0, d0)
    Fan rows(int32_t p0, int d0, int32_t p1, int d1) { return get(p0, d0, p1, d1, false); }

private:
    static constexpr int kShards = 64;
    static constexpr int32_t kSamples = 64;
    struct Shard {
        std::shared_mutex mu;
        std::unordered_map<uint64_t, Fan> map;
    };
    const HostIndex& ix_;
    const std::vector<double> biased_;
    std::unique_ptr<Shard[]> shards_;
    std::atomic<size_t> sampled_{0};
    Fan get(int32_t p0, int d0, int32_t p1, int d1, bool perEdge);
};

// Plans both phases.  Semantics follow CPU_01_nonparallel/SupportCounting.cpp:
// support (474-552) with the head triple counted as used, body size
// (563-631) with the seed atom's keys as headS candidates, or from hO's end
// where `fans` (optional) says that costs less.  freeVars false: free
// variables are grounded as any other (no free steps, no row scans).  Without
// both a plan's memory depends on the rule and the predicates' rows alone.
RulePlan plan_rule(const Rule& rule, const HostIndex& ix, const Geom& geom, FanSamples* fans = nullptr,
                   bool freeVars = true);

}  // namespace gr
