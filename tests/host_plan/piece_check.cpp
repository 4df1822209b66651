// build_decode_plan over random and over timed steps: every unit covered once, adjacent items, one item a CTA where the units
// are cut into equal pieces, partial slots and counters, and which of the two plans a timed step gets.
#include <cmath>
#include <cstdio>
#include <map>
#include <random>

#include "host_logic.hpp"

using namespace psi;

#define CHECK(x) do { if (!(x)) { std::printf("%s:%d: %s\n", __FILE__, __LINE__, #x); return 1; } } while (0)

struct Step {
    std::vector<uint32_t> slots, positions, cu{0}, all;
    void add(uint32_t position, uint32_t run) {
        all.push_back(static_cast<uint32_t>(slots.size()));
        slots.push_back(static_cast<uint32_t>(slots.size()));
        positions.push_back(position);
        cu.push_back(cu.back() + run);
    }
    RequestRuns runs() const { return plain_runs(slots.data(), positions.data(), cu.data(), static_cast<uint32_t>(slots.size())); }
};

static uint64_t up(uint64_t a, uint64_t b) { return (a + b - 1) / b; }

static bool pieces(const WorkPlan& p) {
    for (uint32_t c = 0; c < p.num_ctas(); ++c)
        if (p.cta_item_begin[c + 1] - p.cta_item_begin[c] != 1) return false;
    return true;
}

int main() {
    std::mt19937 rng(11);
    auto pick = [&](uint32_t lo, uint32_t hi) { return std::uniform_int_distribution<uint32_t>(lo, hi)(rng); };
    const std::pair<uint32_t, uint32_t> profiles[] = {{16, 2}, {24, 4}, {40, 8}, {4, 1}, {34, 2}, {3, 3}};
    uint32_t cut = 0, shared = 0;
    for (int trial = 0; trial < 2000; ++trial) {
        const PlanGeometry geo = plan_geometry(profiles[trial % 6].first, profiles[trial % 6].second);
        const uint32_t max_ctas = trial % 5 == 0 ? pick(1, 9) : 148, longest = 1u << pick(0, 18), n = pick(0, trial % 3 ? 12 : 60);
        Step s;
        for (uint32_t r = 0; r < n; ++r) s.add(pick(0, longest), trial % 4 ? 1 : pick(0, 6));
        const WorkPlan p = build_decode_plan(geo, s.runs(), s.all, max_ctas, trial % 2 ? 16 : 4, trial % 2 ? 32 : 0);
        const WorkPlan b = build_balanced_plan(geo, s.runs(), s.all, max_ctas, trial % 2 ? 16 : 4, trial % 2 ? 32 : 0);
        CHECK(p.num_ctas() <= max_ctas && p.total_kv_tiles == b.total_kv_tiles && p.tiles.size() == b.tiles.size());
        if (p.total_kv_tiles == 0) { CHECK(p.items.empty()); continue; }
        CHECK(p.cta_item_begin.front() == 0 && p.cta_item_begin.back() == p.items.size());
        for (uint32_t c = 0; c < p.num_ctas(); ++c) CHECK(p.cta_item_begin[c] <= p.cta_item_begin[c + 1]);
        const uint64_t units = uint64_t(p.tiles.size()) * geo.num_kv_heads * geo.head_tiles;
        const ReplayCapacity cap = replay_capacity(geo, s.cu.back(), max_ctas, false);
        CHECK(p.items.size() <= cap.items && p.reduces.size() <= cap.reduces && p.num_partial_slots <= cap.slots);
        uint64_t covered = 0, slot = 0, unit = 0, count = 0, at = 0;
        for (size_t i = 0; i < p.items.size();) {
            size_t j = i;
            uint32_t end = 0;
            for (; j < p.items.size() && p.items[j].tile == p.items[i].tile && p.items[j].head_sel == p.items[i].head_sel; ++j) {
                const WorkItem& it = p.items[j];
                CHECK(it.kv_begin == end && it.kv_begin % 16 == 0 && it.kv_end > it.kv_begin);
                end = it.kv_end;
            }
            const ExecTile& tile = p.tiles[p.items[i].tile];
            CHECK(end == tile.first_pos + (tile.flat_end - tile.flat_begin));
            CHECK(at == uint64_t(p.items[i].tile) * geo.num_kv_heads * geo.head_tiles + p.items[i].head_sel);
            ++at;
            for (size_t k = i; k < j; ++k) {
                if (j - i == 1) CHECK(p.items[k].partial_slot == kU32Max);
                else CHECK(p.items[k].partial_slot == slot++ && p.items[k].reduce_unit == unit && p.items[k].unit_num_items == j - i);
            }
            unit += j - i > 1;
            covered += up(end, 16);
            ++count;
            i = j;
        }
        CHECK(count == units && covered == p.total_kv_tiles && slot == p.num_partial_slots && unit == p.reduces.size());
        (pieces(p) ? cut : shared) += 1;
    }
    CHECK(cut > 200 && shared > 200);

    struct Timed { uint32_t hq, hkv, requests, low, high, min_tiles, start; bool pieces; };
    const Timed timed[] = {{40, 8, 1, 777, 777, 16, 32, true},     {40, 8, 1, 100, 100, 16, 32, true},  {40, 8, 1, 2500, 2500, 16, 32, true},
                           {40, 8, 16, 700, 700, 16, 32, true},    {16, 2, 8, 1000, 1000, 16, 32, true}, {16, 2, 64, 300, 300, 16, 32, true},
                           {24, 8, 16, 1000, 1000, 4, 16, true},   {16, 2, 16, 1000, 1000, 4, 0, true},  {16, 2, 16, 4000, 4000, 16, 32, true},
                           {16, 2, 32, 1000, 8000, 16, 32, false}, {16, 2, 16, 500, 4000, 16, 32, false}, {32, 8, 16, 300, 2000, 4, 0, false},
                           {16, 2, 4, 262144, 262144, 16, 32, false}, {24, 4, 64, 4096, 32768, 16, 32, false}};
    for (const Timed& t : timed) {
        Step s;
        for (uint32_t r = 0; r < t.requests; ++r)  // a geometric spread, as they were timed
            s.add(static_cast<uint32_t>(t.low * std::pow(double(t.high) / t.low, t.requests > 1 ? double(r) / (t.requests - 1) : 0.0)), 1);
        const bool got = pieces(build_decode_plan(plan_geometry(t.hq, t.hkv), s.runs(), s.all, 148, t.min_tiles, t.start));
        if (got != t.pieces) std::printf("%u requests of %u to %u: %s\n", t.requests, t.low, t.high, got ? "pieces" : "shares");
        CHECK(got == t.pieces);
    }
    std::printf("pieces ok\n");
    return 0;
}
