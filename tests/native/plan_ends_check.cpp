// The checks of plan_check.cpp for plans as the engine makes them: body sizes
// from the end that the sampled fan-outs favour, at every block size, beside
// the plain plans that calls with a scratch limit fall back to.
// Usage: plan_ends_check GRAPH.ttl RULES.txt
#define main plan_check_main
#include "plan_check.cpp"
#undef main

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
    FanSamples fans(ix);
    long bad = 0, phases = 0, far = 0, scans = 0;
    while (std::getline(in, line)) {
        if (line.empty()) continue;
        for (int block : {128, 256, 512})
            for (bool fast : {true, false}) {
                Geom geom;
                geom.block = block;
                RulePlan rp;
                try {
                    rp = plan_rule(parser.parse_text(line), ix, geom, fast ? &fans : nullptr, fast);
                } catch (const RuleError&) {
                    continue;
                }
                if (rp.status != kRuleOk) continue;
                for (const PhasePlan* ph : {&rp.support, &rp.body}) {
                    if (ph->how != kDevice) continue;
                    ++phases;
                    bad += check_plan(*ph, geom);
                    bool free = ph->plan.supDir == 1;
                    far += free;
                    for (int s = 0; s < ph->plan.m; ++s) {
                        scans += ph->plan.steps[s].kind == kRowScan;
                        free |= ph->plan.steps[s].kind == kRowScan || ph->plan.steps[s].free;
                    }
                    bad += !fast && free;   // the plain plan has none of them
                }
            }
    }
    std::printf("device phases %ld from the far end %ld row scans %ld violations %ld\n", phases, far, scans, bad);
    return bad == 0 ? 0 : 1;
}
