// The planner's group T-form tables (products of more than 8 vectors) against its
// tile T-form tables: both name every chunk of every input tile once.  Compiled
// together with the planner, so that the reach of a segment's offsets, 64 GiB,
// can be set to a size that a test matrix exceeds.
#include "../../hlr_b200/csrc/plan.cpp"

#include <tuple>

using namespace hlrc;

// 0: the tables agree; < 0: the planner's status; > 0: the first check that fails.
// segments: group segments of all passes.
extern "C" int group_plan_check(const hlrc_h_desc* d, uint64_t span, int* segments) {
    if (span) g_knobs.group_span = span;
    hlrc_options o{};
    o.precision = HLRC_PREC_F64;
    o.max_nrhs = 32;
    Plan p;
    const hlrc_status st = plan_h(*d, o, p);
    g_knobs = PlanKnobs{};
    if (st != HLRC_OK) return -int(st);
    *segments = 0;
    bool any = false;
    for (const TTPass& t : p.ttpasses) {
        // (first row in the input vector, element offset, columns) of each chunk
        std::vector<std::tuple<uint32_t, uint64_t, int>> tile, group;
        for (const TTSeg& s : t.segs[FMT_F64])
            for (uint32_t c = s.cb; c < s.ce; ++c) tile.emplace_back(s.v_off, uint64_t(t.chunks[c].byte_off) / sizeof(double), int(t.chunks[c].nc));
        for (const GTSeg& s : t.gsegs) {
            ++*segments;
            uint64_t lo = ~uint64_t(0), hi = 0;
            for (uint32_t c = s.cb; c < s.ce; ++c)
                for (uint32_t a = 0; a < s.ntiles; ++a) {
                    const GTChunk& g = t.gchunks[c];
                    if (g.a[a] == GT_NONE) continue;
                    const uint64_t at = s.base + 2 * uint64_t(g.a[a]);
                    lo = std::min(lo, at);
                    hi = std::max(hi, at);
                    group.emplace_back(t.gtiles[s.tile0 + a].v_off, at, int(g.nc));
                }
            if (span && hi - lo >= span) return 2;
        }
        std::sort(tile.begin(), tile.end());
        std::sort(group.begin(), group.end());
        if (tile != group) return 3;
        any = any || !tile.empty();
        if (std::adjacent_find(group.begin(), group.end()) != group.end()) return 4;
    }
    return any ? 0 : 1;
}
