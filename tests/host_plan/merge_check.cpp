// Where the f32 and the odd-profile kernel merge cut units: the bound on a unit's pieces that a replay reservation relies on, over
// random steps, and that a reservation which merges in the launch does so for every plan of one-token requests.  And how long the
// pieces of a step are for each kernel.
#include <algorithm>
#include <cstdio>
#include <random>

#include "host_logic.hpp"

using namespace psi;

#define CHECK(x) do { if (!(x)) { std::printf("%s:%d: %s\n", __FILE__, __LINE__, #x); return 1; } } while (0)

int main() {
    std::mt19937 rng(17);
    auto pick = [&](uint32_t lo, uint32_t hi) { return std::uniform_int_distribution<uint32_t>(lo, hi)(rng); };
    const std::pair<uint32_t, uint32_t> profiles[] = {{16, 2}, {24, 8}, {40, 8}, {4, 1}, {34, 2}, {3, 3}, {16, 1}};
    uint32_t many = 0, merging = 0;
    for (int trial = 0; trial < 3000; ++trial) {
        const PlanGeometry geo = plan_geometry(profiles[trial % 7].first, profiles[trial % 7].second);
        const uint32_t max_ctas = trial % 5 == 0 ? pick(1, 600) : 148, longest = 1u << pick(0, 18), n = pick(1, trial % 3 ? 6 : 40);
        const bool one_token = trial % 2 != 0;
        std::vector<uint32_t> slots, positions, cu{0}, all;
        for (uint32_t r = 0; r < n; ++r) {
            slots.push_back(r);
            all.push_back(r);
            positions.push_back(pick(0, longest));
            cu.push_back(cu.back() + (one_token ? 1 : pick(1, 6)));
        }
        const RequestRuns runs = plain_runs(slots.data(), positions.data(), cu.data(), n);
        for (DecodeKernel kernel : {DecodeKernel::kMmaAny, DecodeKernel::kF32}) {
            const WorkPlan plan = build_decode_plan(geo, runs, all, max_ctas, 4, kernel == DecodeKernel::kF32 ? 0 : 16, piece_model(kernel, trial % 4 ? 128 : 64));
            const uint32_t bound = max_ctas / (geo.num_kv_heads * geo.head_tiles) + 2;
            for (const ReduceUnit& unit : plan.reduces) {
                CHECK(unit.num_items <= bound);
                many += unit.num_items > 8;
            }
            for (uint32_t head_dim : {32u, 96u, 128u, 256u}) {
                bool few = true, short_merges = true;
                for (const ReduceUnit& unit : plan.reduces) {
                    const ExecTile& tile = plan.tiles[plan.items[unit.first_item].tile];
                    const uint32_t rows = (tile.flat_end - tile.flat_begin) * geo.heads_per_tile;
                    const MergeShape shape = merge_shape(unit.num_items, rows, head_dim, 256);
                    CHECK(shape.ways == 1 || shape.ways == 2 || shape.ways == 4);
                    CHECK(uint64_t(shape.trips) * shape.at_once * 256 >= uint64_t(unit.num_items) * rows * head_dim / 4);
                    short_merges = short_merges && shape.trips <= 2;
                    few = few && shape.trips <= 2 && unit.num_items <= 8;
                }
                CHECK(merges_in_launch(geo, plan, head_dim) == few);
                if (one_token && merges_in_launch(geo, max_ctas, head_dim)) {
                    CHECK(short_merges);
                    merging += !plan.reduces.empty();
                }
            }
        }
    }
    CHECK(many > 500 && merging > 500);

    // The longest piece, in KV tiles, of steps timed with either model (0: equal shares).
    struct Timed { uint32_t hq, hkv, requests, tokens; DecodeKernel kernel; uint32_t head_dim, longest; };
    const Timed timed[] = {{16, 2, 1, 300, DecodeKernel::kF32, 256, 4}, {16, 2, 8, 370, DecodeKernel::kF32, 256, 0}, {16, 2, 4, 600, DecodeKernel::kF32, 256, 4},
                           {32, 8, 1, 300, DecodeKernel::kF32, 128, 4}, {32, 8, 8, 370, DecodeKernel::kF32, 128, 12}, {16, 1, 4, 300, DecodeKernel::kF32, 128, 4},
                           {16, 2, 16, 600, DecodeKernel::kMmaAny, 200, 10}, {24, 8, 4, 700, DecodeKernel::kMmaAny, 120, 11}, {24, 8, 8, 370, DecodeKernel::kMmaAny, 96, 24},
                           {16, 2, 1, 300, DecodeKernel::kMmaAny, 48, 19}, {40, 8, 1, 300, DecodeKernel::kCudaCore, 80, 0}, {16, 2, 8, 370, DecodeKernel::kCudaCore, 66, 0}};
    for (const Timed& t : timed) {
        std::vector<uint32_t> slots, positions(t.requests, t.tokens), cu{0}, all;
        for (uint32_t r = 0; r < t.requests; ++r) {
            slots.push_back(r);
            all.push_back(r);
            cu.push_back(r + 1);
        }
        const WorkPlan plan = build_decode_plan(plan_geometry(t.hq, t.hkv), plain_runs(slots.data(), positions.data(), cu.data(), t.requests), all, 148, 4,
                                                t.kernel == DecodeKernel::kMmaAny ? 16 : 0, piece_model(t.kernel, t.head_dim));
        const WorkPlan shares = build_balanced_plan(plan_geometry(t.hq, t.hkv), plain_runs(slots.data(), positions.data(), cu.data(), t.requests), all, 148, 4,
                                                    t.kernel == DecodeKernel::kMmaAny ? 16 : 0);
        uint32_t longest = 0;
        for (const WorkItem& item : plan.items) longest = std::max(longest, (item.kv_end - item.kv_begin + kKvTile - 1) / kKvTile);
        if (plan.cta_item_begin == shares.cta_item_begin &&
            std::equal(plan.items.begin(), plan.items.end(), shares.items.begin(), shares.items.end(),
                       [](const WorkItem& a, const WorkItem& b) { return a.tile == b.tile && a.kv_begin == b.kv_begin && a.kv_end == b.kv_end; }))
            longest = 0;
        if (longest != t.longest) std::printf("%u x %u, %u/%u heads: %u\n", t.requests, t.tokens, t.hq, t.hkv, longest);
        CHECK(longest == t.longest);
    }
    // Item lengths: a step of equal pieces has no CTA of several items; one long request among short ones has a long mean and a
    // CTA of short items, which is what the kernels with more warps look at.
    for (const bool unequal : {false, true}) {
        std::vector<uint32_t> slots, positions, cu{0}, all;
        for (uint32_t r = 0; r < (unequal ? 40u : 4u); ++r) {
            slots.push_back(r);
            all.push_back(r);
            positions.push_back(!unequal ? 1000 : r < 4 ? 60000 : 60);
            cu.push_back(r + 1);
        }
        const WorkPlan plan = build_decode_plan(plan_geometry(32, 8), plain_runs(slots.data(), positions.data(), cu.data(), cu.back()), all, 148, 4, 0, kSlowRoundPieces);
        const ItemLengths lengths = item_lengths(plan);
        CHECK(lengths.mean == plan.total_kv_tiles / plan.items.size());
        if (unequal) CHECK(lengths.mean >= 64 && lengths.least < 16);
        else CHECK(lengths.least == kU32Max);
    }
    CHECK(item_lengths(WorkPlan{}).mean == 0);
    std::printf("merges ok\n");
    return 0;
}
