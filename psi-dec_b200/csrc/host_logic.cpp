#include "host_logic.hpp"

#include <algorithm>
#include <cmath>
#include <limits>
#include <queue>

namespace psi {

namespace {
uint64_t div_ceil(uint64_t a, uint64_t b) { return (a + b - 1) / b; }
uint32_t sat_u32(uint64_t v) { return v > kU32Max ? kU32Max : static_cast<uint32_t>(v); }
}  // namespace

// -------------------------------------------------------------------------------------------------------------------
// Replay buckets.  Base list up to 64, then four equal steps per octave, plus `boundary - 1` for each topology
// boundary and the terminal capacity (crates/inference-executor-core/src/replay.rs:25-44,69-90).
// -------------------------------------------------------------------------------------------------------------------
BucketPolicy::BucketPolicy(uint32_t max_capacity, const std::vector<uint32_t>& topology_boundaries)
    : max_capacity_(max_capacity) {
    require(max_capacity > 0, "replay bucket capacity must be positive");
    for (uint32_t b : {1u, 2u, 4u, 6u, 8u, 12u, 16u, 20u, 24u, 32u, 40u, 48u, 56u, 64u}) {
        if (b <= max_capacity) buckets_.push_back(b);
    }
    bool open = true;
    for (uint32_t octave = 64; open && octave < max_capacity; octave = sat_u32(uint64_t(octave) * 2)) {
        for (uint32_t quarter = 1; quarter <= 4; ++quarter) {
            uint32_t candidate = sat_u32(uint64_t(octave) + uint64_t(octave / 4) * quarter);
            if (candidate >= max_capacity) {
                open = false;
                break;
            }
            buckets_.push_back(candidate);
        }
    }
    for (uint32_t boundary : topology_boundaries) {
        require(boundary > 0, "replay topology boundary must be positive");
        if (boundary > 1 && boundary <= max_capacity) buckets_.push_back(boundary - 1);
    }
    buckets_.push_back(max_capacity);
    std::sort(buckets_.begin(), buckets_.end());
    buckets_.erase(std::unique(buckets_.begin(), buckets_.end()), buckets_.end());
}

uint32_t BucketPolicy::capacity(uint32_t active) const {
    require(active > 0, "replay bucket requires active work");
    require(active <= max_capacity_, "replay active work exceeds capacity");
    return *std::lower_bound(buckets_.begin(), buckets_.end(), active);
}

// -------------------------------------------------------------------------------------------------------------------
// Variant selector (crates/inference-backend-metal/src/components/gqa_split_kv.rs:29-157).
// -------------------------------------------------------------------------------------------------------------------
SplitKvSelector::SplitKvSelector(uint32_t io_dtype, uint32_t page_bytes, uint32_t num_q_heads, uint32_t num_kv_heads,
                                 uint32_t head_dim, bool dspark_history) {
    require(io_dtype == PSI_DTYPE_F32 || io_dtype == PSI_DTYPE_BF16, "GQA SplitKV io_dtype must be f32 or bf16");
    require(page_bytes > 0 && num_q_heads > 0 && num_kv_heads > 0 && head_dim > 0, "GQA SplitKV config must be positive");
    require(num_q_heads % num_kv_heads == 0, "GQA q heads must be a multiple of kv heads");
    uint64_t per_token = uint64_t(num_kv_heads) * head_dim * 2u * dtype_bytes(io_dtype);
    require(per_token <= kU32Max, "GQA K/V bytes per token must fit u32");
    require(page_bytes % per_token == 0, "GQA page_bytes must be divisible by the K/V bytes per token");
    tokens_per_page_ = page_bytes / static_cast<uint32_t>(per_token);
    group_ = num_q_heads / num_kv_heads;
    bool profile = (head_dim == 128 && tokens_per_page_ == 8) ||
                   (head_dim == 256 && (tokens_per_page_ == 8 || tokens_per_page_ == 16));
    supports_tiled_ = !dspark_history && io_dtype == PSI_DTYPE_BF16 && profile && group_ <= 8;
    full_group_for_tiled_ = !dspark_history && head_dim == 128 && tokens_per_page_ == 8;
    uint32_t bounded = std::max(32u, std::min(head_dim, 256u));
    single_threads_ = 1;
    while (single_threads_ < bounded) single_threads_ <<= 1;
}

psi_split_kv_variant SplitKvSelector::select(uint32_t num_tokens, uint32_t num_q_token_tiles) const {
    require(num_tokens > 0, "GQA SplitKV selection requires tokens");
    require(num_q_token_tiles > 0 && num_q_token_tiles <= num_tokens, "GQA SplitKV q-token-tile count out of range");
    const uint32_t max_head_tile = 256 / (tiled_q_token_tile_size() / 8 * 32);
    psi_split_kv_variant v{};
    if (!supports_tiled_ || uint64_t(num_tokens) < 2ull * num_q_token_tiles) {
        v.tiled_q = 0;
        v.kv_token_tile_size = single_threads_;
        v.num_threads_per_threadblock = single_threads_;
        v.q_head_tile_size = std::min(group_, max_head_tile);
        return v;
    }
    bool halve = !full_group_for_tiled_ && uint64_t(num_tokens) < 4ull * num_q_token_tiles;
    v.tiled_q = 1;
    v.q_token_tile_size = tiled_q_token_tile_size();
    v.kv_token_tile_size = 16;
    v.q_head_tile_size = std::min(halve ? (group_ + 1) / 2 : group_, max_head_tile);
    return v;
}

// -------------------------------------------------------------------------------------------------------------------
// Reference-format metadata (crates/inference-executor-metal/src/attn/gqa/batch_metadata.rs:192-523).
// -------------------------------------------------------------------------------------------------------------------
ReferenceMetadata::ReferenceMetadata(uint32_t max_tokens)
    : req_slots(max_tokens, 0), flat_token_indices(max_tokens, 0), q_token_tiles(size_t(max_tokens) * 2, 0),
      kv_splits(size_t(max_tokens) * 3, 0), cu_kv_splits(size_t(max_tokens) + 1, 0) {
    require(max_tokens > 0, "GQA batch metadata requires tokens");
}

namespace {

struct SplitCandidateTile {
    uint32_t flat_begin, flat_end, context_len;
    uint64_t kv_tiles;
    uint64_t splits = 1;
};

// Greedy refinement shared by both reference planners: while budget remains, give one more split to the tile whose
// splits are currently the longest (first such tile wins ties), batch_metadata.rs:370-386,466-488.
void refine_splits(std::vector<SplitCandidateTile>& tiles, uint64_t used, uint64_t budget, bool charge_tokens) {
    while (used < budget) {
        int64_t best = -1;
        uint64_t best_len = 0;
        for (size_t i = 0; i < tiles.size(); ++i) {
            const auto& t = tiles[i];
            uint64_t cost = charge_tokens ? t.flat_end - t.flat_begin : 1;
            if (used + cost > budget || t.splits >= t.kv_tiles) continue;
            uint64_t len = div_ceil(t.kv_tiles, t.splits);
            if (best < 0 || len > best_len) {
                best = static_cast<int64_t>(i);
                best_len = len;
            }
        }
        if (best < 0) break;
        used += charge_tokens ? tiles[best].flat_end - tiles[best].flat_begin : 1;
        tiles[best].splits += 1;
    }
}

}  // namespace

uint32_t ReferenceMetadata::expand_tokens(const uint32_t* req_slots_by_req, const uint32_t* token_indices,
                                          const uint32_t* cu_tokens, uint32_t num_reqs) {
    require(num_reqs > 0, "GQA batch metadata requires tokens");
    require(cu_tokens[0] == 0, "GQA batch cu_tokens must start at zero");
    for (uint32_t r = 0; r < num_reqs; ++r) {
        require(cu_tokens[r] <= cu_tokens[r + 1], "GQA batch cu_tokens must be nondecreasing");
        require(uint64_t(token_indices[r]) + (cu_tokens[r + 1] - cu_tokens[r]) <= kU32Max,
                "GQA request context length must fit u32");
    }
    const uint32_t num_tokens = cu_tokens[num_reqs];
    require(num_tokens > 0, "GQA batch metadata requires tokens");
    require(num_tokens <= max_tokens(), "GQA batch exceeds the metadata token capacity");
    for (uint32_t r = 0, t = 0; r < num_reqs; ++r) {
        for (uint32_t i = 0; i < cu_tokens[r + 1] - cu_tokens[r]; ++i, ++t) {
            req_slots[t] = req_slots_by_req[r];
            flat_token_indices[t] = token_indices[r] + i;
        }
    }
    return num_tokens;
}

psi_replay_shape ReferenceMetadata::update(const uint32_t* req_slots_by_req, const uint32_t* token_indices,
                                           const uint32_t* cu_tokens, uint32_t num_reqs,
                                           const psi_split_kv_variant& variant, uint32_t capacity_mode,
                                           const std::vector<uint32_t>& token_topology_boundaries,
                                           uint32_t caller_num_total_tokens) {
    require(num_reqs > 0, "GQA batch metadata requires tokens");
    require(cu_tokens[0] == 0, "GQA batch cu_tokens must start at zero");
    for (uint32_t r = 0; r < num_reqs; ++r) {
        require(cu_tokens[r] <= cu_tokens[r + 1], "GQA batch cu_tokens must be nondecreasing");
        require(uint64_t(token_indices[r]) + (cu_tokens[r + 1] - cu_tokens[r]) <= kU32Max,
                "GQA request context length must fit u32");
    }
    const uint32_t num_tokens = cu_tokens[num_reqs];
    require(num_tokens > 0, "GQA batch metadata requires tokens");
    require(num_tokens <= max_tokens(), "GQA batch exceeds the metadata token capacity");
    if (capacity_mode == PSI_CAPACITY_CALLER_TOKENS) {
        require(num_tokens <= caller_num_total_tokens,
                "GQA active token count must not exceed the caller-owned token capacity");
        require(caller_num_total_tokens <= max_tokens(),
                "GQA caller-owned token capacity must not exceed the metadata capacity");
    }
    for (uint32_t r = 0, t = 0; r < num_reqs; ++r) {
        for (uint32_t i = 0; i < cu_tokens[r + 1] - cu_tokens[r]; ++i, ++t) {
            req_slots[t] = req_slots_by_req[r];
            flat_token_indices[t] = token_indices[r] + i;
        }
    }

    const bool tiled = variant.tiled_q != 0;
    require(variant.kv_token_tile_size > 0, "GQA KV-token tile size must be positive");
    std::vector<SplitCandidateTile> tiles;
    if (!tiled) {
        tiles.reserve(num_tokens);
        for (uint32_t t = 0; t < num_tokens; ++t) {
            uint32_t ctx = flat_token_indices[t] + 1;
            tiles.push_back({t, t + 1, ctx, div_ceil(ctx, variant.kv_token_tile_size)});
        }
        refine_splits(tiles, num_tokens, max_tokens(), /*charge_tokens=*/false);
    } else {
        require(variant.q_token_tile_size > 0, "GQA Q-token tile size must be positive");
        for (uint32_t r = 0; r < num_reqs; ++r) {
            for (uint32_t begin = cu_tokens[r]; begin < cu_tokens[r + 1];) {
                uint32_t end = std::min(cu_tokens[r + 1], begin + variant.q_token_tile_size);
                uint32_t ctx = token_indices[r] + (end - cu_tokens[r]);
                tiles.push_back({begin, end, ctx, div_ceil(ctx, variant.kv_token_tile_size)});
                begin = end;
            }
        }
        refine_splits(tiles, num_tokens, max_tokens(), /*charge_tokens=*/true);
    }

    std::vector<uint32_t> splits, cu{0};
    for (size_t i = 0; i < tiles.size(); ++i) {
        const auto& t = tiles[i];
        for (uint64_t s = 0; s < t.splits; ++s) {
            uint64_t begin = t.kv_tiles * s / t.splits * variant.kv_token_tile_size;
            uint64_t end = t.kv_tiles * (s + 1) / t.splits * variant.kv_token_tile_size;
            require(begin <= kU32Max, "GQA map KV split KV-token begin must fit u32");
            splits.push_back(static_cast<uint32_t>(i));
            splits.push_back(static_cast<uint32_t>(begin));
            splits.push_back(static_cast<uint32_t>(std::min<uint64_t>(end, t.context_len)));
        }
        cu.push_back(static_cast<uint32_t>(splits.size() / 3));
    }
    const uint32_t num_tiles = static_cast<uint32_t>(tiles.size());
    const uint32_t num_splits = static_cast<uint32_t>(splits.size() / 3);

    uint32_t total_tokens = num_tokens, total_tiles = num_tiles, total_splits = 0;
    if (capacity_mode == PSI_CAPACITY_EXACT) {
        uint64_t pow2 = 1;
        while (pow2 < num_splits) pow2 <<= 1;
        total_splits = static_cast<uint32_t>(std::min<uint64_t>(pow2, max_tokens()));
    } else {
        BucketPolicy plain(max_tokens(), {});
        total_tiles = plain.capacity(num_tiles);
        total_splits = plain.capacity(num_splits);
        total_tokens = capacity_mode == PSI_CAPACITY_BUCKETED
                           ? BucketPolicy(max_tokens(), token_topology_boundaries).capacity(num_tokens)
                           : caller_num_total_tokens;
    }
    require(total_splits >= num_splits, "GQA KV split capacity is below the active split count");

    if (tiled) {
        for (uint32_t i = 0; i < num_tiles; ++i) {
            q_token_tiles[size_t(i) * 2] = tiles[i].flat_begin;
            q_token_tiles[size_t(i) * 2 + 1] = tiles[i].flat_end;
        }
    }
    std::copy(splits.begin(), splits.end(), kv_splits.begin());
    std::fill(kv_splits.begin() + splits.size(), kv_splits.begin() + size_t(total_splits) * 3, kU32Max);
    std::copy(cu.begin(), cu.end(), cu_kv_splits.begin());

    psi_replay_shape shape{};
    shape.num_tokens = num_tokens;
    shape.num_total_tokens = total_tokens;
    shape.num_q_token_tiles = num_tiles;
    shape.num_total_q_token_tiles = total_tiles;
    shape.num_sdpa_map_task_templates = num_splits;
    shape.num_total_sdpa_map_task_templates = total_splits;
    shape.reduce_sdpa_partial_outputs = (tiled || num_splits > num_tokens) ? 1u : 0u;
    return shape;
}

// -------------------------------------------------------------------------------------------------------------------
// Device work plans.
// -------------------------------------------------------------------------------------------------------------------
PlanGeometry plan_geometry(uint32_t num_q_heads, uint32_t num_kv_heads) {
    PlanGeometry g{};
    g.group = num_q_heads / num_kv_heads;
    g.heads_per_tile = std::min(g.group, kMaxRows);
    g.head_tiles = static_cast<uint32_t>(div_ceil(g.group, g.heads_per_tile));
    g.tokens_per_tile = std::max(1u, kMaxRows / g.heads_per_tile);
    g.num_kv_heads = num_kv_heads;
    return g;
}

bool merge_one_position_runs(const RequestRuns& runs, MergedRuns& merged) {
    auto same = [&](uint32_t a, uint32_t b) {
        return runs.run(a) == 1 && runs.run(b) == 1 && runs.req_slots[a] == runs.req_slots[b] &&
               runs.token_indices[a] == runs.token_indices[b];
    };
    const uint32_t n = runs.size();
    bool any = false;
    for (uint32_t r = 1; r < n && !any; ++r) any = same(r - 1, r);
    if (!any) return false;
    merged = MergedRuns{};
    merged.cu_tokens.push_back(0);
    for (uint32_t r = 0; r < n;) {
        uint32_t end = r + 1;
        while (end < n && same(r, end)) ++end;
        merged.req_slots.push_back(runs.req_slots[r]);
        merged.token_indices.push_back(runs.token_indices[r]);
        merged.cu_tokens.push_back(runs.cu_tokens[end]);
        merged.one_position.push_back(end - r > 1 ? 1 : 0);
        r = end;
    }
    return true;
}

namespace {

// Closes the plan: assigns partial slots to every item whose (tile, head_sel) unit is shared with another item and
// lists those units for the reduce pass.  Items of one unit must be adjacent.
void finish_plan(WorkPlan& plan) {
    plan.num_partial_slots = 0;
    plan.reduces.clear();
    size_t i = 0;
    while (i < plan.items.size()) {
        size_t j = i + 1;
        while (j < plan.items.size() && plan.items[j].tile == plan.items[i].tile &&
               plan.items[j].head_sel == plan.items[i].head_sel) {
            ++j;
        }
        if (j - i == 1) {
            plan.items[i].partial_slot = kU32Max;
        } else {
            const uint32_t unit = static_cast<uint32_t>(plan.reduces.size());
            const uint32_t first_slot = plan.num_partial_slots;
            plan.reduces.push_back({static_cast<uint32_t>(i), static_cast<uint32_t>(j - i)});
            for (size_t k = i; k < j; ++k) {
                plan.items[k].partial_slot = plan.num_partial_slots++;
                plan.items[k].reduce_unit = unit;
                plan.items[k].unit_first_slot = first_slot;
                plan.items[k].unit_num_items = static_cast<uint32_t>(j - i);
            }
        }
        i = j;
    }
}

// Lists the query tiles of `requests` and their contexts; the KV tiles of all units.
uint64_t list_tiles(const PlanGeometry& geo, const RequestRuns& runs, const std::vector<uint32_t>& requests, WorkPlan& plan,
                    std::vector<uint32_t>& tile_ctx) {
    for (uint32_t r : requests) {
        for (uint32_t begin = runs.cu_tokens[r]; begin < runs.cu_tokens[r + 1];) {
            uint32_t end = std::min(runs.cu_tokens[r + 1], begin + geo.tokens_per_tile);
            plan.tiles.push_back({begin, end, runs.req_slots[r], runs.position(r, begin), runs.token_indices[r],
                                  runs.cu_tokens[r], runs.one_position(r)});
            tile_ctx.push_back(runs.context(r, end));
            begin = end;
        }
    }
    uint64_t total = 0;
    for (uint32_t ctx : tile_ctx) total += div_ceil(ctx, kKvTile) * geo.num_kv_heads * geo.head_tiles;
    return plan.total_kv_tiles = total;
}

// Cuts the units of the plan's query tiles into equal shares (build_balanced_plan).
void share_out(WorkPlan& plan, const std::vector<uint32_t>& tile_ctx, uint32_t heads, uint32_t max_ctas,
               uint32_t min_kv_tiles_per_cta, uint32_t item_start_cost) {
    const uint64_t total = plan.total_kv_tiles;
    uint64_t wanted = std::max<uint64_t>(1, total / std::max(1u, min_kv_tiles_per_cta));
    const uint64_t num_ctas = std::min<uint64_t>(std::max(1u, max_ctas), wanted);
    // Every unit is laid out as `start_cost` virtual tiles (what opening a new item costs a CTA: pipeline drain,
    // merge, first-load latency) followed by its KV tiles; share c covers positions [span*c/n, span*(c+1)/n) of that
    // line, so CTAs that open several items get correspondingly fewer KV tiles.
    const uint64_t start_cost = item_start_cost;
    const uint64_t span = total + start_cost * plan.tiles.size() * heads;
    uint64_t cursor = 0;  // position of the current unit's first (virtual) tile
    uint32_t cta = 0;
    plan.cta_item_begin.assign(1, 0);
    auto share_end = [&](uint64_t c) { return span * (c + 1) / num_ctas; };
    for (uint32_t tile = 0; tile < plan.tiles.size(); ++tile) {
        const uint64_t unit_tiles = div_ceil(tile_ctx[tile], kKvTile);
        const uint64_t unit_span = start_cost + unit_tiles;
        for (uint32_t h = 0; h < heads; ++h) {
            uint64_t done = 0;
            while (done < unit_span) {
                while (cursor + done >= share_end(cta)) {
                    ++cta;
                    plan.cta_item_begin.push_back(static_cast<uint32_t>(plan.items.size()));
                }
                const uint64_t take = std::min(unit_span - done, share_end(cta) - (cursor + done));
                const uint64_t real_begin = std::max(done, start_cost) - start_cost;
                const uint64_t real_end = std::max(done + take, start_cost) - start_cost;
                if (real_end > real_begin) {
                    WorkItem item{};
                    item.tile = tile;
                    item.head_sel = h;
                    item.kv_begin = static_cast<uint32_t>(real_begin * kKvTile);
                    item.kv_end = static_cast<uint32_t>(std::min<uint64_t>(real_end * kKvTile, tile_ctx[tile]));
                    plan.items.push_back(item);
                }
                done += take;
            }
            cursor += unit_span;
        }
    }
    while (plan.cta_item_begin.size() < num_ctas + 1) plan.cta_item_begin.push_back(static_cast<uint32_t>(plan.items.size()));
    finish_plan(plan);
}

}  // namespace

WorkPlan build_decode_plan(const PlanGeometry& geo, const RequestRuns& runs, const std::vector<uint32_t>& requests,
                           uint32_t max_ctas, uint32_t min_kv_tiles_per_cta, uint32_t item_start_cost, const PieceModel& model) {
    WorkPlan plan;
    std::vector<uint32_t> tile_ctx;
    const uint64_t total = list_tiles(geo, runs, requests, plan, tile_ctx);
    const uint32_t heads = geo.num_kv_heads * geo.head_tiles;
    const uint64_t units = uint64_t(plan.tiles.size()) * heads;
    const uint32_t round = model.round_tiles;
    uint64_t pick = 0;
    if (model.round_tiles != 0 && total != 0 && units <= max_ctas) {
        // What an equal share costs, in KV tiles: whole rounds of the share itself (of as many CTAs as that plan would take) with
        // a start for every unit, and a merge of pieces.
        const uint64_t ctas = std::min<uint64_t>(max_ctas, std::max<uint64_t>(1, total / std::max(1u, min_kv_tiles_per_cta)));
        const uint64_t share = (total + std::max(item_start_cost, kPieceStartTiles) * units) / ctas;
        const uint64_t shares = div_ceil(share, round) * round + model.merge_tiles + model.group_tiles;
        const uint64_t longest = div_ceil(*std::max_element(tile_ctx.begin(), tile_ctx.end()), kKvTile);
        uint64_t best = shares + 1;
        // (a bound between two multiples of the round cuts the units as the smaller one does; one that is not below `best`
        // leaves some unit a piece as long)
        const uint64_t least = div_ceil(div_ceil(total, max_ctas), round) * round;
        for (uint64_t bound = least; bound < best; bound += round) {
            // (most bounds fail by the number of pieces: one 32-bit division a query tile, and no more than that)
            const uint32_t cap = static_cast<uint32_t>(bound), room = max_ctas / heads;
            uint32_t pieces = 0;
            for (size_t t = 0; t < tile_ctx.size() && pieces <= room; ++t) pieces += ((tile_ctx[t] - 1) / kKvTile + cap) / cap;
            if (pieces <= room) {
                uint64_t cost = 0;
                for (uint32_t ctx : tile_ctx) {
                    const uint32_t tiles = (ctx - 1) / kKvTile + 1, n = (tiles + cap - 1) / cap;
                    const uint32_t rounds = ((tiles + n - 1) / n + round - 1) / round;
                    cost = std::max<uint64_t>(cost, rounds * round + (n > 1 ? model.merge_tiles + model.group_tiles * ((n + 3) / 4) : 0));
                }
                if (cost < best) best = cost, pick = bound;
            }
            if (bound >= longest) break;
        }
    }
    if (pick == 0) {
        if (total != 0) share_out(plan, tile_ctx, heads, max_ctas, min_kv_tiles_per_cta, item_start_cost);
        return plan;
    }
    plan.items.reserve(max_ctas);
    plan.cta_item_begin.assign(1, 0);
    for (uint32_t tile = 0; tile < plan.tiles.size(); ++tile) {
        const uint64_t tiles = div_ceil(tile_ctx[tile], kKvTile), n = div_ceil(tiles, pick);
        for (uint32_t h = 0; h < heads; ++h) {
            for (uint64_t k = 0; k < n; ++k) {
                WorkItem item{};
                item.tile = tile;
                item.head_sel = h;
                item.kv_begin = static_cast<uint32_t>(tiles * k / n * kKvTile);
                item.kv_end = static_cast<uint32_t>(std::min<uint64_t>(tiles * (k + 1) / n * kKvTile, tile_ctx[tile]));
                plan.items.push_back(item);
                plan.cta_item_begin.push_back(static_cast<uint32_t>(plan.items.size()));
            }
        }
    }
    finish_plan(plan);
    return plan;
}

ItemLengths item_lengths(const WorkPlan& plan) {
    ItemLengths lengths{0, kU32Max};
    if (plan.items.empty()) return lengths;
    lengths.mean = static_cast<uint32_t>(std::min<uint64_t>(plan.total_kv_tiles / plan.items.size(), kU32Max));
    for (uint32_t c = 0; c < plan.num_ctas(); ++c) {
        const uint32_t begin = plan.cta_item_begin[c], end = plan.cta_item_begin[c + 1];
        if (end - begin < 2) continue;
        uint64_t tiles = 0;
        for (uint32_t i = begin; i < end; ++i) tiles += div_ceil(plan.items[i].kv_end - plan.items[i].kv_begin, kKvTile);
        lengths.least = static_cast<uint32_t>(std::min<uint64_t>(tiles / (end - begin), lengths.least));
    }
    return lengths;
}

bool merges_in_launch(const PlanGeometry& geo, const WorkPlan& plan, uint32_t head_dim) {
    for (const ReduceUnit& unit : plan.reduces) {
        const ExecTile& tile = plan.tiles[plan.items[unit.first_item].tile];
        if (unit.num_items > 8 || merge_shape(unit.num_items, (tile.flat_end - tile.flat_begin) * geo.heads_per_tile, head_dim, 256).trips > 2)
            return false;
    }
    return true;
}

bool merges_in_launch(const PlanGeometry& geo, uint32_t max_ctas, uint32_t head_dim) {
    return merge_shape(max_ctas / (geo.num_kv_heads * geo.head_tiles) + 2, geo.heads_per_tile, head_dim, 256).trips <= 2;
}

WorkPlan build_balanced_plan(const PlanGeometry& geo, const uint32_t* req_slots, const uint32_t* token_indices,
                             const uint32_t* cu_tokens, uint32_t num_reqs, uint32_t max_ctas,
                             uint32_t min_kv_tiles_per_cta, uint32_t item_start_cost) {
    std::vector<uint32_t> all(num_reqs);
    for (uint32_t r = 0; r < num_reqs; ++r) all[r] = r;
    return build_balanced_plan(geo, plain_runs(req_slots, token_indices, cu_tokens, num_reqs), all, max_ctas,
                               min_kv_tiles_per_cta, item_start_cost);
}

WorkPlan build_balanced_plan(const PlanGeometry& geo, const RequestRuns& runs, const std::vector<uint32_t>& requests,
                             uint32_t max_ctas, uint32_t min_kv_tiles_per_cta, uint32_t item_start_cost) {
    WorkPlan plan;
    std::vector<uint32_t> tile_ctx;
    const uint64_t total = list_tiles(geo, runs, requests, plan, tile_ctx);
    const uint32_t heads = geo.num_kv_heads * geo.head_tiles;
    if (total != 0) share_out(plan, tile_ctx, heads, max_ctas, min_kv_tiles_per_cta, item_start_cost);
    return plan;
}

WorkPlan build_reference_plan(const PlanGeometry& geo, const ReferenceMetadata& md, const psi_replay_shape& shape,
                              bool tiled_q, const uint32_t* token_indices, const uint32_t* cu_tokens,
                              uint32_t num_reqs) {
    WorkPlan plan;
    const uint32_t heads = geo.num_kv_heads * geo.head_tiles;
    uint32_t req = 0;  // reference q tiles come in flat-token order, so the owning request only moves forward
    for (uint32_t rt = 0; rt < shape.num_q_token_tiles; ++rt) {
        const uint32_t flat_begin = tiled_q ? md.q_token_tiles[size_t(rt) * 2] : rt;
        const uint32_t flat_end = tiled_q ? md.q_token_tiles[size_t(rt) * 2 + 1] : rt + 1;
        const uint32_t s_begin = md.cu_kv_splits[rt], s_end = md.cu_kv_splits[rt + 1];
        for (uint32_t begin = flat_begin; begin < flat_end;) {
            const uint32_t end = std::min(flat_end, begin + geo.tokens_per_tile);
            const uint32_t tile = static_cast<uint32_t>(plan.tiles.size());
            while (req + 1 < num_reqs && begin >= cu_tokens[req + 1]) ++req;
            plan.tiles.push_back({begin, end, md.req_slots[begin], md.flat_token_indices[begin], token_indices[req],
                                  cu_tokens[req], false});
            const uint32_t ctx = md.flat_token_indices[end - 1] + 1;  // keys the sub-tile's last token sees
            for (uint32_t h = 0; h < heads; ++h) {
                for (uint32_t s = s_begin; s < s_end; ++s) {
                    const uint32_t kv_begin = md.kv_splits[size_t(s) * 3 + 1];
                    const uint32_t kv_end = std::min(md.kv_splits[size_t(s) * 3 + 2], ctx);
                    if (kv_begin >= kv_end && s != s_begin) continue;  // the split lies beyond this sub-tile's context
                    WorkItem item{};
                    item.tile = tile;
                    item.head_sel = h;
                    item.kv_begin = kv_begin;
                    item.kv_end = std::max(kv_end, kv_begin);
                    plan.items.push_back(item);
                    plan.total_kv_tiles += div_ceil(item.kv_end - item.kv_begin, kKvTile);
                }
            }
            begin = end;
        }
    }
    plan.cta_item_begin.resize(plan.items.size() + 1);
    for (size_t i = 0; i <= plan.items.size(); ++i) plan.cta_item_begin[i] = static_cast<uint32_t>(i);
    finish_plan(plan);
    return plan;
}

namespace {

// Query rows of one chunk item are packed (token, head) pairs: as many whole tokens as its rows hold.
uint32_t tokens_per_chunk_item(const PlanGeometry& geo) { return kMaxRows * kChunkTilesPerItem / geo.heads_per_tile; }

// Whole units, longest first, where none is long against a CTA's share or worth a cut.
bool whole_units(uint64_t longest, uint64_t fair_share) {
    return longest <= std::max<uint64_t>(fair_share / 2, kChunkWholeTokens / kKvTile);
}

}  // namespace

ChunkOrder chunk_order(const PlanGeometry& geo, const RequestRuns& runs, const std::vector<uint32_t>& requests, uint64_t token_bytes) {
    // K/V the runs touch: below a third of the L2 the order of the work cannot cost HBM traffic, and balance beats stream
    // order; so does it where every run fits one super-tile and nothing is read twice in whatever order
    uint64_t kv_bytes = 0;
    bool one_pass = true;
    for (uint32_t r : requests) {
        one_pass = one_pass && runs.run(r) * geo.heads_per_tile <= kMaxRows * kChunkTilesPerItem;
        kv_bytes += uint64_t(runs.context(r, runs.cu_tokens[r + 1])) * token_bytes;
    }
    return kv_bytes <= (40ull << 20) ? ChunkOrder::kL2Resident : (one_pass ? ChunkOrder::kEqualShares : ChunkOrder::kStream);
}

bool split_runs(const PlanGeometry& geo, const RequestRuns& runs, const ChunkRule& rule, std::vector<uint32_t>& decode_reqs,
                std::vector<uint32_t>& chunk_reqs) {
    const uint64_t heads = uint64_t(geo.num_kv_heads) * geo.head_tiles;
    // (most runs of most steps are one tile: no division for those)
    auto tiles_of = [&](uint32_t r) {
        const uint32_t run = runs.run(r);
        return run <= geo.tokens_per_tile ? std::min(run, 1u) : (run + geo.tokens_per_tile - 1) / geo.tokens_per_tile;
    };
    bool any_long = false;
    std::vector<uint32_t> several;                             // runs of several tiles, none of them a long one
    uint64_t once = 0, per_tile = 0, units = 0, longest = 0;   // KV tiles of `several`: read once, read per query tile
    for (uint32_t r = 0; r < runs.size(); ++r) {
        const uint64_t tiles = tiles_of(r);
        any_long = any_long || (tiles >= kChunkMinTiles && !runs.one_position(r));
        if (tiles < 2) continue;
        const uint64_t keys = div_ceil(runs.context(r, runs.cu_tokens[r + 1]), kKvTile);
        const uint64_t passes = div_ceil(runs.run(r), tokens_per_chunk_item(geo));
        several.push_back(r);
        once += keys * passes * heads;
        per_tile += keys * tiles * heads;
        units += passes * heads;
        longest = std::max(longest, keys);
    }
    bool take = false;
    if (rule.short_runs && !any_long && units > 0) {
        // KV tiles a CTA works off on either kernel, and the pieces of a cut unit.  Measured with 2 to 9 rows a request, 1 to
        // 64 requests of 100 to 30,000 tokens, 40/8, 32/8 and 4/1 heads x 128, 16/2 and 24/4 x 256, fused and after the front
        // stage: a tile saved is worth 0.11 us at head_dim 128 and 0.2 at 256, a piece costs 1.2 us and the kernel itself 5.
        // Of 800 such steps none is slower by more than 0.1 us than on the decode kernel, and 96 % of what taking
        // every step at its best would gain is left.  (Four tokens on 2,000 keys, 40/8 x 128: 20 us a layer against 42;
        // 64 requests of 1,500 to 3,000 tokens, eight rows, 24/4 x 256: 350 us against 124.)
        const uint64_t ctas = std::max<uint64_t>(1, std::min<uint64_t>({rule.max_ctas, kChunkMaxPieces * units, once / 4}));
        const bool whole = chunk_order(geo, runs, several, rule.token_bytes) == ChunkOrder::kL2Resident &&
                           whole_units(longest, (once + kChunkUnitCostTiles * units) / ctas);
        const double share = whole ? std::max<double>(longest, double(once) / rule.max_ctas) : double(once) / ctas;
        const double pieces = whole ? 0.0 : double(ctas) / units;
        const double saved = (double(per_tile) / rule.max_ctas - share) * (rule.head_dim / 128.0) * 0.9;
        take = saved > 45.0 + 11.0 * pieces + double(rule.handicap);
    }
    for (uint32_t r = 0; r < runs.size(); ++r) {
        const uint32_t tiles = tiles_of(r);
        if (tiles == 0) continue;
        const bool chunk = take ? tiles >= 2 : (tiles >= kChunkMinTiles && !runs.one_position(r));
        (chunk ? chunk_reqs : decode_reqs).push_back(r);
    }
    return take;
}

ChunkPlan build_chunk_plan(const PlanGeometry& geo, const RequestRuns& runs, const std::vector<uint32_t>& requests, uint32_t max_ctas,
                           uint32_t slot_base, uint32_t counter_base, ChunkOrder order, uint32_t unit_start_cost) {
    ChunkPlan plan;
    // Units in stream order: all super-tiles of one (request, KV head) follow one another, so that CTAs working on
    // neighbouring units at the same time read the same K/V pages (once from HBM, then from L2).
    struct Unit {
        uint32_t req, flat_begin, flat_end, ctx_end, head;
    };
    std::vector<Unit> units;
    const uint32_t tokens_per_item = tokens_per_chunk_item(geo);
    const uint32_t heads = geo.num_kv_heads * geo.head_tiles;
    uint64_t total = 0, longest = 0;
    // longest requests first: the work dealt last, which decides how far the last CTA trails, is the cheapest
    std::vector<uint32_t> by_length(requests);
    std::stable_sort(by_length.begin(), by_length.end(), [&](uint32_t a, uint32_t b) {
        return runs.context(a, runs.cu_tokens[a + 1]) > runs.context(b, runs.cu_tokens[b + 1]);
    });
    for (uint32_t r : by_length) {
        for (uint32_t h = 0; h < heads; ++h) {
            for (uint32_t begin = runs.cu_tokens[r]; begin < runs.cu_tokens[r + 1];) {
                const uint32_t end = std::min(runs.cu_tokens[r + 1], begin + tokens_per_item);
                units.push_back({r, begin, end, runs.context(r, end), h});
                total += div_ceil(units.back().ctx_end, kKvTile);
                longest = std::max(longest, div_ceil(units.back().ctx_end, kKvTile));
                begin = end;
            }
        }
    }
    plan.total_kv_tiles = total;
    if (total == 0) return plan;
    uint64_t num_ctas = std::min<uint64_t>(std::max(1u, max_ctas), std::max<uint64_t>(1, total / 4));
    if (order != ChunkOrder::kStream) num_ctas = std::min<uint64_t>(num_ctas, uint64_t(kChunkMaxPieces) * units.size());
    auto make_item = [&](const Unit& u, uint64_t tile_begin, uint64_t tile_end) {
        const uint32_t head_tile = u.head % geo.head_tiles;
        DeviceItem d{};
        d.kv_begin = static_cast<uint32_t>(tile_begin * kKvTile);
        d.kv_end = static_cast<uint32_t>(std::min<uint64_t>(tile_end * kKvTile, u.ctx_end));
        d.partial_slot = kU32Max;
        d.flat_begin = u.flat_begin;
        d.num_tokens = u.flat_end - u.flat_begin;
        d.req_slot = runs.req_slots[u.req];
        d.kv_head = u.head / geo.head_tiles;
        d.head0 = d.kv_head * geo.group + head_tile * geo.heads_per_tile;
        d.num_heads = std::min(geo.heads_per_tile, geo.group - head_tile * geo.heads_per_tile);
        d.first_pos = runs.position(u.req, u.flat_begin);
        d.new_begin = runs.token_indices[u.req];
        d.flat_req_begin = runs.cu_tokens[u.req];
        d.flags = (head_tile == 0 ? kItemWritesKv : 0u) | (runs.one_position(u.req) ? kItemOnePosition : 0u);
        return d;
    };
    // `n` consecutive items starting at `first` are the pieces of one unit cut across CTAs: partial slots 8 apart,
    // eight arrival counters
    auto share_unit = [&](std::vector<DeviceItem*>& pieces) {
        const uint32_t n = static_cast<uint32_t>(pieces.size());
        if (n <= 1) return;
        const uint32_t first_slot = slot_base + plan.num_partial_slots;
        for (uint32_t k = 0; k < n; ++k) {
            pieces[k]->partial_slot = first_slot + k * kChunkTilesPerItem;
            pieces[k]->reduce_unit = counter_base + plan.num_counters;
            pieces[k]->unit_first_slot = first_slot;
            pieces[k]->unit_num_items = n;
        }
        plan.num_partial_slots += n * kChunkTilesPerItem;
        plan.num_counters += kChunkTilesPerItem;
    };
    const bool l2_resident = order == ChunkOrder::kL2Resident;
    const uint64_t fair_share = (total + uint64_t(unit_start_cost) * units.size()) / num_ctas;
    if (l2_resident && whole_units(longest, fair_share)) {
        // Whole units, longest first, each to the CTA with the least work so far.  Nothing is cut: a cut saves half a
        // unit's tiles on one CTA and costs two partial writes, a fence and a merge, about kChunkMinPieceTiles of them,
        // so it pays only for units of more than twice that which are also long against a CTA's share.
        std::stable_sort(units.begin(), units.end(), [](const Unit& a, const Unit& b) { return a.ctx_end > b.ctx_end; });
        std::priority_queue<std::pair<uint64_t, uint32_t>, std::vector<std::pair<uint64_t, uint32_t>>, std::greater<>> free_first;
        for (uint32_t c = 0; c < num_ctas; ++c) free_first.push({0, c});
        std::vector<std::vector<DeviceItem>> per_cta(num_ctas);
        for (const Unit& u : units) {
            auto [load, c] = free_first.top();
            free_first.pop();
            const uint64_t tiles = div_ceil(u.ctx_end, kKvTile);
            per_cta[c].push_back(make_item(u, 0, tiles));
            free_first.push({load + tiles + unit_start_cost, c});
        }
        plan.cta_item_begin.assign(1, 0);
        for (const auto& list : per_cta) {
            plan.items.insert(plan.items.end(), list.begin(), list.end());
            plan.cta_item_begin.push_back(static_cast<uint32_t>(plan.items.size()));
        }
        return plan;
    }
    if (l2_resident || order == ChunkOrder::kEqualShares) {
        // A working set that stays in L2 whatever the order: contiguous shares of equal cost, units cut where a share
        // ends (two or three pieces per cut unit instead of many), slivers below a quarter of the minimum piece folded
        // into their neighbour.  Every item, a piece as well as a whole unit, costs its KV tiles plus `unit_start_cost`, so
        // that a share of several short ones is not longer than a single long one.
        const uint64_t sliver = kChunkMinPieceTiles / 4;
        // Cuts the units at the ends of `num_ctas` shares of `span`; the cost of all items.
        auto cut = [&](uint64_t span, auto&& item) {
            auto share_end = [&](uint64_t c) { return span * (c + 1) / num_ctas; };
            uint64_t cursor = 0, end = share_end(0);
            uint32_t cta = 0;
            for (size_t k = 0; k < units.size(); ++k) {
                const uint64_t unit_tiles = div_ceil(units[k].ctx_end, kKvTile);
                uint64_t done = 0;
                while (done < unit_tiles) {
                    cursor += unit_start_cost;
                    while (cta + 1 < num_ctas && cursor + (done == 0 ? sliver : 0) >= end) end = share_end(++cta);
                    uint64_t take = std::min(unit_tiles - done, end > cursor ? end - cursor : 1);
                    if (cta + 1 >= num_ctas || unit_tiles - done - take < sliver) take = unit_tiles - done;
                    item(k, cta, done, done + take);
                    done += take;
                    cursor += take;
                }
            }
            return cursor;
        };
        // How many units are cut depends on where the shares end: the smallest shares that hold all items, to within a
        // quarter of an item's cost a share.
        uint64_t span = total + uint64_t(unit_start_cost) * (units.size() + num_ctas);
        if (unit_start_cost == 0) span = total;
        for (uint64_t low = total + uint64_t(unit_start_cost) * units.size(); unit_start_cost > 0 && span - low > num_ctas * unit_start_cost / 4;) {
            const uint64_t middle = (low + span) / 2;
            if (cut(middle, [](size_t, uint32_t, uint64_t, uint64_t) {}) <= middle) span = middle;
            else low = middle;
        }
        plan.items.reserve(units.size() + num_ctas);
        std::vector<uint32_t> owner;  // CTA of every item, in item order
        std::vector<std::pair<size_t, size_t>> unit_items(units.size());  // [first, last) item of every unit
        cut(span, [&](size_t k, uint32_t cta, uint64_t begin, uint64_t end) {
            if (begin == 0) unit_items[k].first = plan.items.size();
            plan.items.push_back(make_item(units[k], begin, end));
            owner.push_back(cta);
            unit_items[k].second = plan.items.size();
        });
        for (const auto& range : unit_items) {
            std::vector<DeviceItem*> pieces;
            for (size_t i = range.first; i < range.second; ++i) pieces.push_back(&plan.items[i]);
            share_unit(pieces);
        }
        plan.cta_item_begin.assign(num_ctas + 1, static_cast<uint32_t>(plan.items.size()));
        plan.cta_item_begin[0] = 0;
        for (size_t i = plan.items.size(); i-- > 0;) plan.cta_item_begin[owner[i]] = static_cast<uint32_t>(i);
        for (uint64_t c = num_ctas; c-- > 1;)  // CTAs without items start where the next one does
            plan.cta_item_begin[c] = std::min(plan.cta_item_begin[c], plan.cta_item_begin[c + 1]);
        return plan;
    }
    // A unit longer than half a CTA's fair share is cut along its KV range into equal pieces (partial slots, merged
    // by the last arriver), which bounds how far the last CTA can trail the others; shorter units stay whole, since
    // every piece costs a partial write and a fence, and the merge reads all of them.
    const uint64_t piece_cap = std::max<uint64_t>(kChunkMinPieceTiles, div_ceil(total, num_ctas * 2));

    // Pieces are dealt in order to whichever CTA is free first under the cost model (KV tiles + a fixed start
    // cost): the static equivalent of CTAs pulling work from a queue.
    struct Slot {
        uint64_t load;
        uint32_t cta;
        bool operator>(const Slot& o) const { return load != o.load ? load > o.load : cta > o.cta; }
    };
    std::priority_queue<Slot, std::vector<Slot>, std::greater<Slot>> free_first;
    for (uint32_t c = 0; c < num_ctas; ++c) free_first.push({0, c});
    std::vector<std::vector<DeviceItem>> per_cta(num_ctas);
    for (const Unit& u : units) {
        const uint64_t unit_tiles = div_ceil(u.ctx_end, kKvTile);
        const uint32_t n = static_cast<uint32_t>(div_ceil(unit_tiles, piece_cap));
        const uint32_t first_slot = slot_base + plan.num_partial_slots;
        for (uint32_t k = 0; k < n; ++k) {
            const uint64_t tile_begin = unit_tiles * k / n, tile_end = unit_tiles * (k + 1) / n;
            DeviceItem d = make_item(u, tile_begin, tile_end);
            if (n > 1) {  // the unit is shared between CTAs: partial slots 8 apart, eight arrival counters
                d.partial_slot = first_slot + k * kChunkTilesPerItem;
                d.reduce_unit = counter_base + plan.num_counters;
                d.unit_first_slot = first_slot;
                d.unit_num_items = n;
            }
            Slot slot = free_first.top();
            free_first.pop();
            per_cta[slot.cta].push_back(d);
            slot.load += (tile_end - tile_begin) + kChunkStartCostTiles;
            free_first.push(slot);
        }
        if (n > 1) {
            plan.num_partial_slots += n * kChunkTilesPerItem;
            plan.num_counters += kChunkTilesPerItem;
        }
    }
    plan.cta_item_begin.assign(1, 0);
    for (const auto& list : per_cta) {
        plan.items.insert(plan.items.end(), list.begin(), list.end());
        plan.cta_item_begin.push_back(static_cast<uint32_t>(plan.items.size()));
    }
    return plan;
}

ReplayCapacity replay_capacity(const PlanGeometry& geo, uint32_t max_tokens, uint32_t max_ctas, bool chunks) {
    const uint64_t heads = uint64_t(geo.num_kv_heads) * geo.head_tiles, units = max_tokens * heads;
    ReplayCapacity cap;
    cap.items = units + max_ctas;
    cap.reduces = units;
    cap.slots = cap.items;
    if (chunks) {
        const uint64_t chunk_units = units / 2 + heads;
        cap.chunk_items = chunk_units + 4ull * max_ctas + 8;
        cap.slots += (std::min<uint64_t>(chunk_units + 2ull * max_ctas, 4ull * max_ctas) + 8) * kChunkTilesPerItem;
    }
    return cap;
}

std::vector<DeviceItem> flatten_plan(const WorkPlan& plan, const PlanGeometry& geo) {
    std::vector<DeviceItem> out(plan.items.size());
    for (size_t i = 0; i < plan.items.size(); ++i) {
        const WorkItem& it = plan.items[i];
        const ExecTile& tile = plan.tiles[it.tile];
        const uint32_t head_tile = it.head_sel % geo.head_tiles;
        DeviceItem& d = out[i];
        d.kv_begin = it.kv_begin;
        d.kv_end = it.kv_end;
        d.partial_slot = it.partial_slot;
        d.reduce_unit = it.reduce_unit;
        d.unit_first_slot = it.unit_first_slot;
        d.unit_num_items = it.unit_num_items;
        d.flat_begin = tile.flat_begin;
        d.num_tokens = tile.flat_end - tile.flat_begin;
        d.req_slot = tile.req_slot;
        d.kv_head = it.head_sel / geo.head_tiles;
        d.head0 = d.kv_head * geo.group + head_tile * geo.heads_per_tile;
        d.num_heads = std::min(geo.heads_per_tile, geo.group - head_tile * geo.heads_per_tile);
        d.first_pos = tile.first_pos;
        d.new_begin = tile.new_begin;
        d.flat_req_begin = tile.flat_req_begin;
        d.flags = (head_tile == 0 ? kItemWritesKv : 0u) | (tile.one_position ? kItemOnePosition : 0u);
    }
    return out;
}

// -------------------------------------------------------------------------------------------------------------------
// RoPE inverse frequencies, with the Yarn ramp when scaling is on.
// -------------------------------------------------------------------------------------------------------------------
RopeParameters rope_parameters(const psi_norm_rope_config& c) {
    require(c.rope_dim > 0 && c.rope_dim % 2 == 0, "RoPE dimension must be positive and even");
    require(std::isfinite(c.rope_theta) && c.rope_theta > 0.0f, "rope_theta must be finite and positive");
    RopeParameters out;
    const uint32_t rope_half = c.rope_dim / 2;
    const bool yarn = c.yarn_enabled != 0;
    if (yarn) {
        require(std::isfinite(c.yarn_factor) && c.yarn_factor >= 1.0f, "Yarn factor must be at least 1");
        require(std::isfinite(c.yarn_attention_factor) && c.yarn_attention_factor > 0.0f, "Yarn attention factor must be positive");
        require(c.yarn_beta_fast > 0.0f && c.yarn_beta_slow > 0.0f && c.yarn_beta_fast >= c.yarn_beta_slow,
                "Yarn beta_fast must be at least beta_slow, both positive");
        require(c.yarn_original_max_position_embeddings > 0, "Yarn original context length must be positive");
        require(c.rope_theta > 1.0f, "Yarn rope_theta must be greater than 1");
        auto correction = [&](float rotations) {
            const double two_pi = 6.283185307179586;
            return static_cast<float>(double(c.rope_dim) *
                                      std::log(double(c.yarn_original_max_position_embeddings) / (double(rotations) * two_pi)) /
                                      (2.0 * std::log(double(c.rope_theta))));
        };
        float low = std::max(correction(c.yarn_beta_fast), 0.0f);
        float high = std::min(correction(c.yarn_beta_slow), static_cast<float>(c.rope_dim - 1));
        if (c.yarn_truncate) {
            low = std::floor(low);
            high = std::ceil(high);
        }
        require(low <= high, "Yarn correction range must be ordered");
        if (low == high) high += 0.001f;
        out.correction_low = low;
        out.correction_high = high;
        out.attention_factor = c.yarn_attention_factor;
    }
    out.inverse_frequencies.resize(rope_half);
    for (uint32_t d = 0; d < rope_half; ++d) {
        float inv = std::pow(c.rope_theta, -(static_cast<float>(d) / static_cast<float>(rope_half)));
        if (yarn) {
            float ramp = (static_cast<float>(d) - out.correction_low) / (out.correction_high - out.correction_low);
            ramp = std::min(std::max(ramp, 0.0f), 1.0f);
            inv *= 1.0f + ramp * (1.0f / c.yarn_factor - 1.0f);
        }
        require(std::isfinite(inv) && inv > 0.0f, "RMSNorm/RoPE inverse frequency must be finite and positive");
        out.inverse_frequencies[d] = inv;
    }
    return out;
}

// -------------------------------------------------------------------------------------------------------------------
// Page-ID allocator: freed IDs are handed out first, oldest free first, then fresh IDs from the counter.
// -------------------------------------------------------------------------------------------------------------------
IdAllocator::IdAllocator(uint64_t capacity) : capacity_(capacity), bitmap_(div_ceil(capacity, 64), 0) {
    require(capacity <= kU32Max, "ID allocator capacity must fit u32");
}

void IdAllocator::mark(uint32_t id, bool live) {
    require(id < capacity_, "U32 ID allocator ID is out of range");
    uint64_t bit = 1ull << (id & 63);
    if (live) bitmap_[id >> 6] |= bit; else bitmap_[id >> 6] &= ~bit;
}

void IdAllocator::alloc_many(uint64_t count, uint32_t* out) {
    uint64_t n = 0;
    while (n < count && !free_ids_.empty()) {
        out[n++] = free_ids_.front();
        free_ids_.pop_front();
    }
    if (n < count) {
        uint64_t fresh = count - n;
        if (counter_ + fresh > capacity_) {
            for (uint64_t i = 0; i < n; ++i) free_ids_.push_back(out[i]);
            throw ExhaustedError("not enough ID");
        }
        for (uint64_t i = 0; i < fresh; ++i) out[n + i] = static_cast<uint32_t>(counter_ + i);
        counter_ += fresh;
    }
    for (uint64_t i = 0; i < count; ++i) mark(out[i], true);
}

void IdAllocator::free_many(const uint32_t* ids, uint64_t count) {
    for (uint64_t i = 0; i < count; ++i) {
        mark(ids[i], false);
        free_ids_.push_back(ids[i]);
    }
}

}  // namespace psi
