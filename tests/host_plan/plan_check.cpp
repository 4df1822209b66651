// Plans of random steps as psi_gqa_prepare makes them, checked on the host: how a step is dealt to the decode and the chunk
// kernels, and the books of every order of a chunk plan.  Built together with the library's host_logic.cpp.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <random>
#include <set>
#include <tuple>

#include "host_logic.hpp"

using namespace psi;

#define CHECK(cond)                                                             \
    do {                                                                        \
        if (!(cond)) {                                                          \
            std::fprintf(stderr, "%s:%d: %s\n", __FILE__, __LINE__, #cond);     \
            std::exit(1);                                                       \
        }                                                                       \
    } while (0)

namespace {

constexpr uint32_t kNone = 0xFFFFFFFFu;
uint64_t up(uint64_t a, uint64_t b) { return (a + b - 1) / b; }

struct Step {
    std::vector<uint32_t> slots, positions, cu{0};
    void add(uint32_t slot, uint32_t position, uint32_t run) {
        slots.push_back(slot);
        positions.push_back(position);
        cu.push_back(cu.back() + run);
    }
    RequestRuns runs() const { return plain_runs(slots.data(), positions.data(), cu.data(), static_cast<uint32_t>(slots.size())); }
};

ChunkRule rule_for(uint32_t ctas, uint32_t head_dim, uint32_t kv_heads, bool short_runs = true) {
    ChunkRule rule;
    rule.max_ctas = ctas;
    rule.head_dim = head_dim;
    rule.token_bytes = uint64_t(kv_heads) * head_dim * 4;
    rule.short_runs = short_runs;
    return rule;
}

// Every unit's keys are covered once, in order; pieces of a cut unit hold partial slots eight apart and one group of eight
// counters, nobody else's; every item belongs to one CTA.
void check_books(const PlanGeometry& geo, const RequestRuns& runs, const std::vector<uint32_t>& requests, const ChunkPlan& plan,
                 uint32_t max_ctas, uint32_t slot_base, uint32_t counter_base) {
    std::map<uint32_t, uint32_t> request_at;  // flat token -> request
    uint64_t units = 0;
    const uint32_t tokens_per_item = kMaxRows * kChunkTilesPerItem / geo.heads_per_tile, heads = geo.num_kv_heads * geo.head_tiles;
    for (uint32_t r : requests) {
        units += up(runs.run(r), tokens_per_item) * heads;
        for (uint32_t t = runs.cu_tokens[r]; t < runs.cu_tokens[r + 1]; ++t) request_at[t] = r;
    }
    CHECK(plan.num_ctas() <= max_ctas);
    if (plan.cta_item_begin.empty()) {
        CHECK(plan.items.empty() && units == 0);
        return;
    }
    CHECK(plan.cta_item_begin.front() == 0 && plan.cta_item_begin.back() == plan.items.size());
    CHECK(std::is_sorted(plan.cta_item_begin.begin(), plan.cta_item_begin.end()));
    std::map<std::tuple<uint32_t, uint32_t>, std::vector<DeviceItem>> by_unit;
    for (const DeviceItem& d : plan.items) {
        CHECK(request_at.count(d.flat_begin));
        const uint32_t r = request_at[d.flat_begin];
        CHECK(d.num_tokens >= 1 && d.num_tokens * d.num_heads <= kMaxRows * kChunkTilesPerItem);
        CHECK(d.req_slot == runs.req_slots[r] && d.first_pos == runs.position(r, d.flat_begin) && d.new_begin == runs.token_indices[r]);
        CHECK(((d.flags & kItemOnePosition) != 0) == runs.one_position(r));
        CHECK(d.kv_begin < d.kv_end && d.kv_begin % 16 == 0);
        by_unit[{d.flat_begin, d.head0}].push_back(d);
    }
    CHECK(by_unit.size() == units);
    std::set<uint32_t> slots, counters;
    for (auto& [key, pieces] : by_unit) {
        std::sort(pieces.begin(), pieces.end(), [](const DeviceItem& a, const DeviceItem& b) { return a.kv_begin < b.kv_begin; });
        const uint32_t r = request_at[pieces[0].flat_begin];
        CHECK(pieces.front().kv_begin == 0);
        CHECK(pieces.back().kv_end == runs.context(r, pieces[0].flat_begin + pieces[0].num_tokens));
        for (size_t i = 0; i + 1 < pieces.size(); ++i) CHECK(pieces[i].kv_end == pieces[i + 1].kv_begin && pieces[i].kv_end % 16 == 0);
        if (pieces.size() == 1) {
            CHECK(pieces[0].partial_slot == kNone);
            continue;
        }
        for (uint32_t i = 0; i < pieces.size(); ++i) {
            CHECK(pieces[i].unit_num_items == pieces.size() && pieces[i].unit_first_slot == pieces[0].unit_first_slot);
            CHECK(pieces[i].reduce_unit == pieces[0].reduce_unit);
            CHECK((pieces[i].partial_slot - pieces[i].unit_first_slot) % kChunkTilesPerItem == 0);
            for (uint32_t s = 0; s < kChunkTilesPerItem; ++s) CHECK(slots.insert(pieces[i].partial_slot + s).second);
        }
        for (uint32_t s = 0; s < kChunkTilesPerItem; ++s) CHECK(counters.insert(pieces[0].reduce_unit + s).second);
    }
    CHECK(slots.size() == plan.num_partial_slots && counters.size() == plan.num_counters);
    if (!slots.empty()) CHECK(*slots.begin() == slot_base && *slots.rbegin() == slot_base + plan.num_partial_slots - 1);
    if (!counters.empty()) CHECK(*counters.begin() == counter_base && *counters.rbegin() == counter_base + plan.num_counters - 1);
}

void check_random_plans() {
    std::mt19937 rng(7);
    auto pick = [&](uint32_t lo, uint32_t hi) { return std::uniform_int_distribution<uint32_t>(lo, hi)(rng); };
    const std::pair<uint32_t, uint32_t> profiles[] = {{16, 2}, {24, 4}, {40, 8}, {4, 1}, {34, 2}, {3, 3}};
    size_t orders[3] = {0, 0, 0}, uneven = 0;
    for (int trial = 0; trial < 600; ++trial) {
        const auto [hq, hkv] = profiles[trial % 6];
        const PlanGeometry geo = plan_geometry(hq, hkv);
        const uint32_t max_ctas = trial % 5 == 0 ? 1 : (trial % 5 == 1 ? 7 : 148);
        Step step;
        const uint32_t n = pick(1, trial % 3 == 0 ? 200 : 8), longest_run = trial % 2 ? 700 : 12, longest_ctx = 1u << pick(0, 17);
        for (uint32_t r = 0; r < n; ++r) {
            if (trial % 4 == 2 && r % 2 == 0) {  // rows of a draft block
                const uint32_t rows = pick(1, 9), position = pick(0, longest_ctx);
                for (uint32_t i = 0; i < rows; ++i) step.add(r, position, 1);
            } else {
                step.add(r, pick(0, longest_ctx), pick(0, longest_run));
            }
        }
        MergedRuns merged;
        RequestRuns runs = step.runs();
        if (merge_one_position_runs(runs, merged)) runs = merged.view();
        std::vector<uint32_t> decode, chunk;
        const ChunkRule rule = rule_for(max_ctas, trial % 2 ? 128 : 256, hkv, trial % 7 != 0);
        const bool fine = split_runs(geo, runs, rule, decode, chunk);
        // every request with rows is dealt once; a step with long runs leaves all others to the decode kernel
        std::set<uint32_t> seen;
        for (uint32_t r : decode) CHECK(runs.run(r) > 0 && seen.insert(r).second);
        for (uint32_t r : chunk) CHECK(runs.run(r) > geo.tokens_per_tile && seen.insert(r).second);
        for (uint32_t r = 0; r < runs.size(); ++r) {
            CHECK((runs.run(r) > 0) == (seen.count(r) > 0));
            const bool is_long = up(runs.run(r), geo.tokens_per_tile) >= kChunkMinTiles && !runs.one_position(r);
            const bool in_chunk = std::find(chunk.begin(), chunk.end(), r) != chunk.end();
            if (is_long) CHECK(in_chunk && !fine);
            else if (in_chunk) CHECK(fine && rule.short_runs);
        }
        const WorkPlan plan = build_balanced_plan(geo, runs, decode, max_ctas, 16, 32);
        const uint32_t slot_base = plan.num_partial_slots, counter_base = static_cast<uint32_t>(plan.reduces.size());
        std::vector<ChunkOrder> all = {ChunkOrder::kStream, ChunkOrder::kEqualShares, ChunkOrder::kL2Resident};
        const ChunkOrder shipped = chunk_order(geo, runs, chunk, rule.token_bytes);
        for (ChunkOrder order : all) {
            const ChunkPlan c = build_chunk_plan(geo, runs, chunk, max_ctas, slot_base, counter_base, order, kChunkUnitCostTiles);
            check_books(geo, runs, chunk, c, max_ctas, slot_base, counter_base);
            // what psi_gqa_reserve_replay sets aside for max_tokens = the step's tokens
            const uint64_t heads = uint64_t(geo.num_kv_heads) * geo.head_tiles, units = step.cu.back() * heads;
            const ReplayCapacity cap = replay_capacity(geo, step.cu.back(), max_ctas, true);
            CHECK(cap.reduces == units && plan.reduces.size() <= cap.reduces);
            CHECK(plan.items.size() <= cap.items && c.items.size() <= cap.chunk_items);
            CHECK(uint64_t(slot_base) + c.num_partial_slots <= cap.slots);
            CHECK(plan.num_ctas() <= max_ctas);
            if (order == shipped && !chunk.empty()) ++orders[static_cast<int>(order)];
            if (order == ChunkOrder::kEqualShares && c.num_ctas() > 1 && chunk.size() > 3) {
                uint64_t top = 0, total = 0;
                for (uint32_t cta = 0; cta < c.num_ctas(); ++cta) {
                    uint64_t load = 0;
                    for (uint32_t i = c.cta_item_begin[cta]; i < c.cta_item_begin[cta + 1]; ++i)
                        load += up(c.items[i].kv_end - c.items[i].kv_begin, 16) + kChunkUnitCostTiles;
                    top = std::max(top, load);
                    total += load;
                }
                // shares are equal up to a folded sliver and the start of one cut unit more
                if (top > total / c.num_ctas() + 2 * kChunkMinPieceTiles) ++uneven;
            }
        }
    }
    CHECK(orders[0] > 10 && orders[1] > 10 && orders[2] > 10);
    CHECK(uneven == 0);
}

void check_merging() {
    Step s;
    for (int i = 0; i < 3; ++i) s.add(5, 99, 1);
    s.add(5, 100, 1);  // next position
    s.add(6, 100, 1);  // another slot
    s.add(6, 100, 2);  // not a single row
    for (int i = 0; i < 2; ++i) s.add(6, 100, 1);
    MergedRuns m;
    CHECK(merge_one_position_runs(s.runs(), m));
    const RequestRuns v = m.view();
    CHECK(v.size() == 5);
    const uint32_t runs[] = {3, 1, 1, 2, 2}, slots[] = {5, 5, 6, 6, 6};
    const bool one[] = {true, false, false, false, true};
    for (uint32_t r = 0; r < 5; ++r) CHECK(v.run(r) == runs[r] && v.req_slots[r] == slots[r] && v.one_position(r) == one[r]);
    CHECK(v.context(0, 3) == 100 && v.position(0, 2) == 99 && v.context(3, v.cu_tokens[4]) == 102);
    Step none;
    none.add(1, 7, 1);
    none.add(1, 8, 1);
    none.add(2, 8, 1);
    CHECK(!merge_one_position_runs(none.runs(), m));
}

// Steps timed on either kernel: the decode kernel keeps the ones it is faster on.
void check_routes() {
    struct Timed {
        uint32_t hq, hkv, head_dim, requests, context, run;
        bool chunk;
    };
    const Timed timed[] = {{40, 8, 128, 1, 2000, 4, false}, {40, 8, 128, 1, 2000, 8, false}, {40, 8, 128, 4, 8000, 4, false},
                           {16, 2, 256, 1, 2000, 3, false}, {16, 2, 256, 4, 8000, 8, false}, {16, 2, 256, 16, 1000, 3, false},
                           {24, 4, 256, 1, 2000, 8, false}, {24, 4, 256, 4, 8000, 3, false}, {4, 1, 128, 16, 20000, 8, false},
                           {4, 1, 128, 64, 3000, 6, false}, {40, 8, 128, 16, 8000, 8, true}, {40, 8, 128, 64, 3000, 4, true},
                           {16, 2, 256, 64, 8000, 8, true}, {24, 4, 256, 64, 3000, 8, true}, {24, 4, 256, 16, 8000, 4, true}};
    for (const Timed& t : timed) {
        Step s;
        for (uint32_t r = 0; r < t.requests; ++r) s.add(r, t.context - t.context * (t.requests - 1 - r) / (2 * t.requests), t.run);
        std::vector<uint32_t> decode, chunk;
        const PlanGeometry geo = plan_geometry(t.hq, t.hkv);
        ChunkRule rule = rule_for(148, t.head_dim, t.hkv);
        CHECK(split_runs(geo, s.runs(), rule, decode, chunk) == t.chunk);
        CHECK((chunk.size() == t.requests) == t.chunk);
        rule.handicap = 1u << 20;
        decode.clear(), chunk.clear();
        CHECK(!split_runs(geo, s.runs(), rule, decode, chunk) && chunk.empty());
        s.add(900, 5000, 600);  // a long run beside them
        rule.handicap = 0;
        decode.clear(), chunk.clear();
        CHECK(!split_runs(geo, s.runs(), rule, decode, chunk) && chunk == std::vector<uint32_t>{t.requests});
    }
}

}  // namespace

int main() {
    check_merging();
    check_routes();
    check_random_plans();
    std::puts("plans ok");
    return 0;
}
