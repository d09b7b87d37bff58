// Native check of the task builder's costs as the engine uses it (built and
// run by tests/test_costs_cpu.py): rules planned from either end, tasks of
// several groups of roots.
//   * The tasks cover every root of a phase exactly once; a plain task holds
//     at most 64 groups, a split root's slices partition its first segment.
//   * Times fed to learn() come back: expected_ns() of a phase is the sum of
//     its tasks' times, walked, split or neither.
//   * Phases never run are expected at the rate of those that were: with
//     every task at the same rate, expected_ns() is that rate times the work
//     build() gives the phase.
//   * Where a phase's roots are cut into slices does not depend on the memos
//     or times that the builder knows.
//   * New walks visit no more roots and edges than the budget allows.
//   * A served launch walks only phases expected to hold the whole GPU for
//     longer than the walk takes, and those whose tasks turned out long.
// Usage: costs_check GRAPH.ttl RULES.txt
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <fstream>
#include <limits>
#include <map>
#include <set>
#include <string>
#include <vector>

#include "../../masterthesis_gpu_acceleration_b200/csrc/index.hpp"
#include "../../masterthesis_gpu_acceleration_b200/csrc/planner.hpp"
#include "../../masterthesis_gpu_acceleration_b200/csrc/rules.hpp"
#include "../../masterthesis_gpu_acceleration_b200/csrc/tasks.hpp"
#include "../../masterthesis_gpu_acceleration_b200/csrc/turtle.hpp"

using namespace gr;

namespace {

long check_cover(TaskBuilder& tb, const PhasePlan& ph, const PhaseTasks& pt, int idx, size_t& multi, size_t& split) {
    long bad = 0;
    const int32_t R = ph.rootEnd - ph.rootBeg;
    std::vector<int> cover((size_t)std::max(R, 0), 0);
    std::map<int32_t, int32_t> sliceEnd;   // split root -> end of its last slice
    for (const DevTask& t : pt.tasks) {
        if (t.plan != idx || t.beg < ph.rootBeg || t.end > ph.rootEnd || t.beg >= t.end) { ++bad; continue; }
        if (t.gRow < 0) {
            if (t.end - t.beg > (int64_t)pt.group * 64) ++bad;
            multi += t.end - t.beg > pt.group;
            for (int32_t r = t.beg; r < t.end; ++r) ++cover[(size_t)(r - ph.rootBeg)];
        } else {
            int32_t& at = sliceEnd[t.beg];
            if (t.end != t.beg + 1 || t.gRow >= pt.heavyRows || t.sub0 != at || t.sub1 <= t.sub0) ++bad;
            at = t.sub1;
        }
    }
    for (const auto& kv : sliceEnd) {
        ++cover[(size_t)(kv.first - ph.rootBeg)];
        ++split;
        int32_t vals[2];
        tb.root_vals(ph.plan, kv.first, vals);
        const auto seg = tb.first_segment(ph.plan, kv.first, vals);
        if (kv.second != seg.second - seg.first) ++bad;
    }
    for (int c : cover) bad += c != 1;
    return bad;
}

bool near(double a, double b) { return std::fabs(a - b) <= 1e-9 * std::max(std::fabs(a), std::fabs(b)); }

// All phases in one list, as a launch holds them.
struct Launch {
    std::vector<DevTask> tasks;
    std::vector<double> cost;
    std::vector<unsigned long long> ns;
    std::vector<double> total;   // ns per phase
    explicit Launch(const std::vector<PhaseTasks>& out, double rate) : total(out.size(), 0.0) {
        unsigned long long at = 1000;
        for (size_t i = 0; i < out.size(); ++i)
            for (size_t k = 0; k < out[i].tasks.size(); ++k) {
                // (whole ns; at rate 0 every task takes its own time)
                const auto d = rate > 0 ? (unsigned long long)std::llround(rate * out[i].cost[k])
                                        : 100ull + (unsigned long long)((k * 7919 + i * 104729) % 5000);
                tasks.push_back(out[i].tasks[k]);
                cost.push_back(out[i].cost[k]);
                ns.push_back(at);
                ns.push_back(at + d);
                total[i] += (double)d;
            }
    }
};

}  // namespace

int main(int argc, char** argv) {
    if (argc < 3) return 2;
    std::string text, err;
    if (!read_file(argv[1], text, &err)) { std::fprintf(stderr, "%s\n", err.c_str()); return 2; }
    TermDict ents, preds;
    std::vector<int32_t> spo;
    parse_turtle_text(text, ents, preds, spo);
    HostIndex ix = build_index(spo, (int32_t)ents.size(), (int32_t)preds.size(), kHubMinDegree);
    RuleParser parser(ents, preds, scan_rule_prefixes_text(text));
    std::ifstream in(argv[2]);
    std::string line;
    std::vector<RulePlan> rps;
    Geom geom;
    FanSamples fans(ix);
    while (std::getline(in, line)) {
        if (line.empty()) continue;
        try {
            rps.push_back(plan_rule(parser.parse_text(line), ix, geom, &fans));
        } catch (const RuleError&) {
        }
    }
    // phases of different computations (equal ones share what is learnt)
    std::vector<const PhasePlan*> phases;
    std::set<uint64_t> seen;
    for (const RulePlan& rp : rps) {
        if (rp.status != kRuleOk) continue;
        for (const PhasePlan* ph : {&rp.support, &rp.body})
            if (ph->how == kDevice && seen.insert(phase_hash(*ph)).second) phases.push_back(ph);
    }
    const int blocks = 148 * (1024 / geom.block);
    long bad = 0, badNs = 0, badRate = 0;
    size_t multi = 0, split = 0, unseen = 0;
    for (double threshold : {2.0e5, 0.0}) {   // walked where it pays; every phase
        TaskBuilder tb(ix);
        tb.walkThreshold = threshold;
        if (threshold == 0.0) tb.forceTarget = 20000;
        std::vector<PhaseTasks> out;
        tb.build(phases, blocks, true, out, threshold == 0.0 ? 1e12 : 4.0e7, false, nullptr, true);
        for (size_t i = 0; i < phases.size(); ++i) bad += check_cover(tb, *phases[i], out[i], (int)i, multi, split);
        const Launch run(out, 0.0);
        tb.learn(phases, run.tasks, run.cost, run.ns.data(), blocks);
        for (size_t i = 0; i < phases.size(); ++i) badNs += !near(tb.expected_ns(*phases[i]), run.total[i]);
    }
    {   // every second phase learnt, no walks: the others follow the rate
        constexpr double kRate = 3.0;
        TaskBuilder tb(ix), all(ix);
        tb.walkThreshold = all.walkThreshold = std::numeric_limits<double>::infinity();
        std::vector<const PhasePlan*> half;
        for (size_t i = 0; i < phases.size(); i += 2) half.push_back(phases[i]);
        std::vector<PhaseTasks> out, whole;
        tb.build(half, blocks, true, out, 0.0, false, nullptr, true);
        all.build(phases, blocks, true, whole, 0.0, false, nullptr, true);
        const Launch run(out, kRate);
        tb.learn(half, run.tasks, run.cost, run.ns.data(), blocks);
        for (size_t i = 1; i < phases.size(); i += 2, ++unseen) {
            // (task times are whole ns: half a ns in 3 x 6,000 units at least)
            const double got = tb.expected_ns(*phases[i]), want = kRate * whole[i].work;
            if (std::fabs(got - want) > 1e-4 * want) ++badRate;
        }
    }
    double skew = 0;
    {
        TaskBuilder tb(ix);
        std::vector<PhaseTasks> out;
        tb.build(phases, blocks, true, out, 4.0e6, kWalkPays, nullptr, true);
        for (const PhaseTasks& pt : out) skew = std::max(skew, pt.skew);
    }
    long badCuts = 0;
    {
        TaskBuilder plain(ix), used(ix);
        std::vector<uint8_t> flags((size_t)ix.nEnt, 1);
        used.memoRows = [&](int, int, int, int, int, int, double* cost) { *cost = 256.0; return &flags; };
        used.walkThreshold = 0.0;
        std::vector<PhaseTasks> out;
        used.build(phases, blocks, true, out, 4.0e6, kWalkBudget, nullptr, true);
        const Launch run(out, 0.0);
        used.learn(phases, run.tasks, run.cost, run.ns.data(), blocks);
        for (const PhasePlan* ph : phases) badCuts += plain.split_roots(*ph, 3) != used.split_roots(*ph, 3);
    }
    long badSteps = 0;
    size_t steps = 0;
    for (double budget : {2.0e4, 2.0e5, 4.0e6})
        for (bool memos : {false, true}) {
            TaskBuilder tb(ix);
            tb.walkThreshold = 0.0;
            std::vector<uint8_t> flags((size_t)ix.nEnt, 1);   // (longer than any predicate's rows)
            if (memos)
                tb.memoRows = [&](int, int, int, int, int, int, double* cost) { *cost = 256.0; return &flags; };
            std::vector<PhaseTasks> out;
            tb.build(phases, blocks, true, out, budget, kWalkBudget, nullptr, true);
            badSteps += (double)tb.walk_steps() > budget;
            steps += tb.walk_steps();
        }
    long badServed = 0;
    {
        TaskBuilder tb(ix), all(ix);
        tb.walkThreshold = 0.0;
        all.walkThreshold = std::numeric_limits<double>::infinity();
        std::vector<PhaseTasks> out, whole;
        all.build(phases, blocks, true, whole, 0.0, false, nullptr, true);
        tb.build(phases, blocks, true, out, 1e12, kWalkServed, nullptr, true);
        for (size_t i = 0; i < phases.size(); ++i) {
            // (a walk takes a step per root at least; chunk 0: walked)
            const double least = kWalkNsPerEdge * (phases[i]->rootEnd - phases[i]->rootBeg);
            badServed += out[i].chunk == 0 && whole[i].work < least * blocks;
        }
        const Launch run(out, 1e3);   // every task takes more than the ms below
        tb.learn(phases, run.tasks, run.cost, run.ns.data(), blocks, 1.0, 1.0e6);
        tb.build(phases, blocks, true, out, 0.0, kWalkServed, nullptr, true);
        size_t at = 0;
        for (size_t i = 0; i < phases.size(); ++i) {
            double worst = 0, sum = 0;
            for (; at < run.tasks.size() && run.tasks[at].plan == (int)i; ++at) {
                const double d = (double)(run.ns[2 * at + 1] - run.ns[2 * at]);
                worst = std::max(worst, d);
                sum += d;
            }
            double every = 0;
            for (double t : run.total) every += t;
            badServed += worst > std::max(1.0e6, every / (blocks * 8.0)) && out[i].chunk != 0;
        }
    }
    std::printf("phases %zu multi-group tasks %zu split roots %zu unseen %zu; cover %ld times %ld rates %ld served %ld cuts %ld steps %ld (%zu) sampled %zu skew x1000 %.0f\n",
                phases.size(), multi, split, unseen, bad, badNs, badRate,
                badServed, badCuts, badSteps, steps, fans.sampled(), 1000 * skew);
    return bad + badNs + badRate + badServed + badCuts + badSteps == 0 ? 0 : 1;
}
