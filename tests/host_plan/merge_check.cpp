// Where the f32 and the odd-profile kernel merge cut units: the bound on a unit's pieces that a replay reservation relies on, over
// random steps, and that a reservation which merges in the launch does so for every plan of one-token requests.
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
            const WorkPlan plan = build_decode_plan(geo, runs, all, max_ctas, 4, kernel == DecodeKernel::kF32 ? 0 : 16, kernel);
            const uint32_t bound = max_ctas / (geo.num_kv_heads * geo.head_tiles) + 2;
            for (const ReduceUnit& unit : plan.reduces) {
                CHECK(unit.num_items <= bound);
                many += unit.num_items > 8;
            }
            for (uint32_t head_dim : {32u, 96u, 128u, 256u}) {
                bool few = true;
                for (const ReduceUnit& unit : plan.reduces) {
                    const ExecTile& tile = plan.tiles[plan.items[unit.first_item].tile];
                    const uint32_t rows = (tile.flat_end - tile.flat_begin) * geo.heads_per_tile;
                    const MergeShape shape = merge_shape(unit.num_items, rows, head_dim, 256);
                    CHECK(shape.ways == 1 || shape.ways == 2 || shape.ways == 4);
                    CHECK(uint64_t(shape.trips) * shape.at_once * 256 >= uint64_t(unit.num_items) * rows * head_dim / 4);
                    few = few && shape.trips <= 2;
                }
                CHECK(merges_in_launch(geo, plan, head_dim) == few);
                if (one_token && merges_in_launch(geo, max_ctas, head_dim)) {
                    CHECK(few);
                    merging += !plan.reduces.empty();
                }
            }
        }
    }
    CHECK(many > 500 && merging > 500);
    std::printf("merges ok\n");
    return 0;
}
