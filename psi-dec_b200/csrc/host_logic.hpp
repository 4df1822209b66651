// Host-side policy of the paged GQA decode path: replay buckets, SplitKV variant selection, the reference-format
// batch metadata, the device work plan and the page-ID allocator.  Pure C++ (no CUDA), shared by the C ABI.
#pragma once

#include <cstdint>
#include <deque>
#include <stdexcept>
#include <string>
#include <vector>

#include "psi_cuda.h"

#ifdef __CUDACC__
#define PSI_HOST_DEVICE __host__ __device__
#else
#define PSI_HOST_DEVICE
#endif

namespace psi {

// A violated caller contract (the reference panics); mapped to PSI_ERR_INVALID_ARGUMENT at the C ABI.
struct ContractError : std::runtime_error {
    using std::runtime_error::runtime_error;
};
struct ExhaustedError : std::runtime_error {
    using std::runtime_error::runtime_error;
};

inline void require(bool ok, const char* message) {
    if (!ok) throw ContractError(message);
}

constexpr uint32_t kU32Max = 0xFFFFFFFFu;
constexpr uint32_t kKvTile = 16;    // KV tokens per device work tile
constexpr uint32_t kMaxRows = 16;   // query rows (tokens x heads) one work item carries

inline uint32_t dtype_bytes(uint32_t dtype) { return dtype == PSI_DTYPE_F32 ? 4u : 2u; }

// ---- replay buckets (crates/inference-executor-core/src/replay.rs) ------------------------------------------------
class BucketPolicy {
public:
    BucketPolicy(uint32_t max_capacity, const std::vector<uint32_t>& topology_boundaries);
    const std::vector<uint32_t>& buckets() const { return buckets_; }
    uint32_t max_capacity() const { return max_capacity_; }
    uint32_t capacity(uint32_t active) const;

private:
    uint32_t max_capacity_;
    std::vector<uint32_t> buckets_;
};

// ---- SplitKV variant selector (crates/inference-backend-metal/src/components/gqa_split_kv.rs) ---------------------
class SplitKvSelector {
public:
    SplitKvSelector(uint32_t io_dtype, uint32_t page_bytes, uint32_t num_q_heads, uint32_t num_kv_heads,
                    uint32_t head_dim, bool dspark_history);
    psi_split_kv_variant select(uint32_t num_tokens, uint32_t num_q_token_tiles) const;
    uint32_t tiled_q_token_tile_size() const { return 8; }
    uint32_t max_q_tokens_per_partial_output() const { return supports_tiled_ ? 8u : 1u; }
    uint32_t tokens_per_page() const { return tokens_per_page_; }

private:
    uint32_t group_;
    uint32_t tokens_per_page_;
    bool supports_tiled_;
    bool full_group_for_tiled_;
    uint32_t single_threads_;
};

// ---- reference-format batch metadata (crates/inference-executor-metal/src/attn/gqa/batch_metadata.rs) -------------
struct ReferenceMetadata {
    // Capacity-sized host mirrors; only the prefixes the reference writes are touched by update().
    std::vector<uint32_t> req_slots, flat_token_indices, q_token_tiles, kv_splits, cu_kv_splits;
    explicit ReferenceMetadata(uint32_t max_tokens);
    uint32_t max_tokens() const { return static_cast<uint32_t>(req_slots.size()); }
    // The per-token arrays alone (request slot and request-absolute position of every query token), with update()'s
    // checks of the batch; returns the token count.  What a launch needs when no reference-format split plan is asked for.
    uint32_t expand_tokens(const uint32_t* req_slots_by_req, const uint32_t* token_indices, const uint32_t* cu_tokens,
                           uint32_t num_reqs);
    psi_replay_shape update(const uint32_t* req_slots_by_req, const uint32_t* token_indices, const uint32_t* cu_tokens,
                            uint32_t num_reqs, const psi_split_kv_variant& variant, uint32_t capacity_mode,
                            const std::vector<uint32_t>& token_topology_boundaries, uint32_t caller_num_total_tokens);
};

// ---- device work plan ------------------------------------------------------------------------------------------------
// One query tile the kernels execute: consecutive flat tokens of one request, at most tokens_per_tile of them.
struct ExecTile {
    uint32_t flat_begin;
    uint32_t flat_end;
    uint32_t req_slot;
    uint32_t first_pos;       // request-absolute position of the tile's first token
    uint32_t new_begin;       // request-absolute position of the request's first token of this step
    uint32_t flat_req_begin;  // flat index of that token
    bool one_position;        // every token of the tile stands at first_pos (RequestRuns::one_position)
};

// One unit of map work while the plan is being built: the rows of (tile, head_sel) against KV tokens
// [kv_begin, kv_end).
struct WorkItem {
    uint32_t tile;
    uint32_t head_sel;      // kv_head * head_tiles + head_tile
    uint32_t kv_begin;
    uint32_t kv_end;
    uint32_t partial_slot;  // kU32Max: the item covers its unit alone and writes the final output itself
    uint32_t reduce_unit;   // index into the plan's reduce list when partial_slot is set
    uint32_t unit_first_slot;  // partial slot of the unit's first item (slots of one unit are consecutive)
    uint32_t unit_num_items;   // items that share the unit
};

// The same item as the kernels read it: self-contained, 64 bytes, no further indirection.
struct DeviceItem {
    uint32_t kv_begin;
    uint32_t kv_end;
    uint32_t partial_slot;
    uint32_t reduce_unit;
    uint32_t unit_first_slot;
    uint32_t unit_num_items;
    uint32_t flat_begin;      // first flat query token of the tile
    uint32_t num_tokens;      // query tokens in the tile
    uint32_t req_slot;
    uint32_t kv_head;
    uint32_t head0;           // first q head the item carries
    uint32_t num_heads;       // q heads the item carries; row r = (token r / num_heads, head r % num_heads)
    uint32_t first_pos;       // position of the tile's first token: token j sees keys [0, first_pos + j]
    uint32_t new_begin;       // positions at or beyond this belong to this step's appended tokens
    uint32_t flat_req_begin;  // flat index of the token at position new_begin
    uint32_t flags;           // kItemWritesKv, kItemOnePosition
};
constexpr uint32_t kItemWritesKv = 1u;     // the item appends its tile's K/V rows that fall into its KV range (fused step)
constexpr uint32_t kItemOnePosition = 2u;  // every token of the item sees keys [0, first_pos]
static_assert(sizeof(DeviceItem) == 64, "DeviceItem is read as four 16-byte words");

struct ReduceUnit {
    uint32_t first_item;
    uint32_t num_items;
};

struct PlanGeometry {
    uint32_t group;            // q heads per kv head
    uint32_t heads_per_tile;   // q heads of one group one item carries (<= 16)
    uint32_t head_tiles;       // ceil(group / heads_per_tile)
    uint32_t tokens_per_tile;  // query tokens one item carries
    uint32_t num_kv_heads;
};

PlanGeometry plan_geometry(uint32_t num_q_heads, uint32_t num_kv_heads);

// The step's requests as the planners see them: a run of consecutive query tokens of one slot each.  A view of the
// caller's arrays (a step is planned in microseconds; copies of them are a part of that).
struct RequestRuns {
    const uint32_t* req_slots = nullptr;
    const uint32_t* token_indices = nullptr;
    const uint32_t* cu_tokens = nullptr;
    uint32_t num_reqs = 0;
    const uint8_t* one_position_runs = nullptr;  // nullptr: none
    uint32_t size() const { return num_reqs; }
    // the run's tokens all stand at token_indices[r] instead of following one another
    bool one_position(uint32_t r) const { return one_position_runs != nullptr && one_position_runs[r] != 0; }
    uint32_t run(uint32_t r) const { return cu_tokens[r + 1] - cu_tokens[r]; }
    // position of flat token `t` of request r, and the keys its run sees up to and with the token before `end`
    uint32_t position(uint32_t r, uint32_t t) const { return token_indices[r] + (one_position(r) ? 0 : t - cu_tokens[r]); }
    uint32_t context(uint32_t r, uint32_t end) const { return token_indices[r] + (one_position(r) ? 1 : end - cu_tokens[r]); }
};
inline RequestRuns plain_runs(const uint32_t* req_slots, const uint32_t* token_indices, const uint32_t* cu_tokens, uint32_t num_reqs) {
    return {req_slots, token_indices, cu_tokens, num_reqs, nullptr};
}
struct MergedRuns {
    std::vector<uint32_t> req_slots, token_indices, cu_tokens;
    std::vector<uint8_t> one_position;
    RequestRuns view() const {
        return {req_slots.data(), token_indices.data(), cu_tokens.data(), static_cast<uint32_t>(req_slots.size()), one_position.data()};
    }
};
// Adjacent one-token requests of one slot at one position (the rows of a draft block, which all see the same history)
// become one run, so that the history is read once for all of them; false when there are none.  Not for launches that
// take this step's K/V rows from the caller's buffers: there every request reads its own row at that position.
bool merge_one_position_runs(const RequestRuns& runs, MergedRuns& merged);

struct WorkPlan {
    std::vector<ExecTile> tiles;
    std::vector<WorkItem> items;
    std::vector<uint32_t> cta_item_begin;  // [num_ctas + 1]
    std::vector<ReduceUnit> reduces;
    uint32_t num_partial_slots = 0;
    uint64_t total_kv_tiles = 0;
    // what a launch of the plan looks at, where its kernel does: merges_in_launch and item_lengths
    bool merges = false;
    uint32_t item_tiles = 0, least_item_tiles = 0;
    uint32_t num_ctas() const { return cta_item_begin.empty() ? 0u : static_cast<uint32_t>(cta_item_begin.size() - 1); }
};

// Equal-share plan: the (tile, head_sel) units laid end to end in 16-token KV tiles, cut into `max_ctas` (or fewer)
// contiguous shares.  `item_start_cost` (in KV tiles) is what opening one more item costs a CTA; shares are equal in
// KV tiles plus that cost per unit start.
WorkPlan build_balanced_plan(const PlanGeometry& geo, const uint32_t* req_slots, const uint32_t* token_indices,
                             const uint32_t* cu_tokens, uint32_t num_reqs, uint32_t max_ctas,
                             uint32_t min_kv_tiles_per_cta, uint32_t item_start_cost = 0);
// The same over a subset of the batch's requests (indices into the request arrays, ascending).
WorkPlan build_balanced_plan(const PlanGeometry& geo, const RequestRuns& runs, const std::vector<uint32_t>& requests,
                             uint32_t max_ctas, uint32_t min_kv_tiles_per_cta, uint32_t item_start_cost = 0);

// The kernels that take decode rows: the tensor-core kernels of head_dim 64, 128 and 256 and of the odd 16-bit profiles, the f32
// kernel, and the CUDA-core kernels of every other profile and of PSI_KERNEL_GENERIC (staged, or one warp an item).
enum class DecodeKernel : uint32_t { kMma, kMmaAny, kF32, kCudaCore };

// The plan of the kernels that run one CTA of eight warps or more an SM (all but kCudaCore).  Where every unit can be cut into
// equal pieces of one CTA each, no CTA opens a second item, and pieces are whole rounds of a tile a warp: a step that does not
// fill the device is then bounded by its longest piece and the merge, where an equal share may hold the ends of two units or many
// short ones.  The bound on a piece is the one with the smallest modelled cost, and the equal shares stay where theirs is smaller.
// In KV tiles: a piece costs its rounds, a cut unit pays `merge_tiles` for arrival and merge and `group_tiles` for every four
// pieces, and a start counts 16 in the shares where they count less (f32).
struct PieceModel {
    uint32_t round_tiles;  // 0: always the shares
    uint32_t merge_tiles, group_tiles;
};
constexpr uint32_t kPieceStartTiles = 16;
// The tensor-core kernel of the even profiles (eight tiles, a round of all warps, take 1.08 us at head_dim 128), fitted on one
// request of 100 to 8,000 tokens cut in every way: 2.5 us a merge, 0.6 us four pieces.  Replayed steps, equal shares and pieces:
//   one request of 777 tokens, 40/8 heads x 128, six layers: 75.9 and 64.6 us; of 100: 87.4 and 45.6; of 2,500: 82.2 and 77.1;
//   four layers: 16 of 700 tokens 87.7 and 66.1; 8 of 1,000, 16/2 x 256, 76.7 and 64.0; 64 of 300 90.9 and 71.1; 16 of 1,000,
//   32/8 x 64, 77.1 and 58.0; 24/8 x 96 102.9 and 84.3; 16 of 4,000, 16/2 x 256, 126.4 and 125.5.
// Unequal steps it leaves to the shares: 32 of 1,000 to 8,000 tokens, 16/2 x 256, 175.2 and 186.6 us; 16 of 500 to 4,000 87.1 and
// 88.8; f32, 16 of 300 to 2,000, 32/8 x 128, 164.1 and 194.2.
constexpr PieceModel kMmaPieces{8, 14, 4};
// An f32 round is eight tokens a warp, four tiles, and takes longer than a round above, so that a merge is worth fewer tiles; so
// it is in the odd-profile kernel above head_dim 96, where half a round more of warps still saves time.  Replayed, four layers,
// shares, the model above and this one: f32, 16/2 heads x 256, one request of 300 tokens 84, 107 and 63 us; 8 of 370 65, 120 and
// 65; 4 of 600 87, 87 and 71; 16 of 1,000 136, 116 and 117; 32/8 x 128, one of 300 66, 61 and 51; 8 of 370 87, 72 and 65; 16/1 x
// 128, 4 of 300 88, 108 and 71; bf16, 16/2 x 200, 8 of 370 63, 75 and 60; 24/8 x 120, 4 of 700 59, 60 and 54; 24/8 x 96, 8 of 370
// 60, 52 and 53; 16/2 x 48, one of 300 49, 46 and 49.
constexpr PieceModel kSlowRoundPieces{4, 6, 2};
// The CUDA-core kernels have no warps that take a tile each, and run several CTAs an SM.  Four layers, shares and the first model:
// one request of 300 tokens, 40/8 heads, f32 x 80 76 and 112 us, bf16 x 84 112 and 210, x 66 389 and 1,553; 8 of 370, 16/2 heads,
// 71 and 147, 90 and 260, 504 and 2,554.
constexpr PieceModel piece_model(DecodeKernel kernel, uint32_t head_dim) {
    return kernel == DecodeKernel::kCudaCore ? PieceModel{0, 0, 0}
           : kernel == DecodeKernel::kMma || (kernel == DecodeKernel::kMmaAny && head_dim <= 96) ? kMmaPieces : kSlowRoundPieces;
}
WorkPlan build_decode_plan(const PlanGeometry& geo, const RequestRuns& runs, const std::vector<uint32_t>& requests,
                           uint32_t max_ctas, uint32_t min_kv_tiles_per_cta, uint32_t item_start_cost,
                           const PieceModel& model = kMmaPieces);

// How a CTA of `threads` threads merges `pieces` partials of `rows` x head_dim outputs (unit_merge.cuh): `at_once` pieces are loaded
// at a time, `ways` threads share the pieces of four columns, and `trips` is the number of round trips to the L2, one after
// another.  Eight at a time only for more than eight pieces: replayed bf16 steps of 24/8 heads x 96, 8 requests of 100 to 4,000
// tokens, 78.0 us with four and 80.2 with eight; f32 steps of one request of 2,500, 32/8 x 128 (19 pieces), 90 and 84.
struct MergeShape {
    uint32_t at_once, ways, trips;
};
PSI_HOST_DEVICE constexpr MergeShape merge_shape(uint32_t pieces, uint32_t rows, uint32_t head_dim, uint32_t threads) {
    const uint32_t outputs = rows * head_dim / 4, at_once = pieces <= 8 ? 4 : 8;
    uint32_t ways = 1;
    while (pieces > 8 * ways && ways < 4 && 2 * ways * outputs <= threads) ways *= 2;
    return {at_once, ways, (pieces + at_once * ways - 1) / (at_once * ways) * ((outputs * ways + threads - 1) / threads)};
}
// Whether the f32 and the odd-profile kernel merge a plan's cut units in the launch: only where no unit has more than eight pieces
// or takes more than two round trips, since one CTA merges a unit while the reduce launch has one for every row.  Four layers, in
// the launch (four pieces at a time) and by the reduce launch: f32, 32/8 heads x 128, 16 requests of 100 tokens (one or two
// pieces) 42 and 53 us, of 500 94 and 102, 4 of 2,500 (five pieces) 116 and 122, 2 of 8,000 (ten) 168 and 163, one of 20,000 (19)
// 205 and 187; 16/2 x 256, 4 of 2,500 (19 pieces, two outputs a thread) 154 and 120; 16/1 x 128, one of 5,000 (148 pieces) 236 and
// 112; bf16, 24/8 x 96, 8 of 370 52 and 59; 16/1 x 160, one of 5,000 256 and 98.
bool merges_in_launch(const PlanGeometry& geo, const WorkPlan& plan, uint32_t head_dim);
// The same for every plan of up to max_ctas CTAs (a replay reservation, whose launches are the same for all of them): a unit has
// at most max_ctas / (units of a query tile) + 2 pieces, which may be more than eight here, as most steps' units have fewer: 32/8
// heads x 128 as above, replayed, 16 of 500 92 us in the launch and 102 with the reduce launch, one of 2,500 86 and 79.  Rows
// count as one token's.
bool merges_in_launch(const PlanGeometry& geo, uint32_t max_ctas, uint32_t head_dim);

// KV tiles of an item: over the plan, and in the CTA of several items whose are the shortest (kU32Max: every CTA has one).  More
// warps an item pay where items are long, and the CTA of many short ones ends last with them.
struct ItemLengths {
    uint32_t mean, least;
};
ItemLengths item_lengths(const WorkPlan& plan);

// One CTA per (reference KV split, head_sel); reference q tiles wider than tokens_per_tile are cut into sub-tiles
// that share the split boundaries.
WorkPlan build_reference_plan(const PlanGeometry& geo, const ReferenceMetadata& md, const psi_replay_shape& shape,
                              bool tiled_q, const uint32_t* token_indices, const uint32_t* cu_tokens,
                              uint32_t num_reqs);

// Plan of the long-query (chunk) kernel: items are super-tiles of up to eight consecutive query tiles of one request
// and KV head; the warp w of a CTA owns tile w of the super-tile, its partial slot is `partial_slot + w` and its arrival
// counter `reduce_unit + w`; the slots of one unit lie 8 apart (`unit_first_slot + ordinal * 8 + w`).
struct ChunkPlan {
    std::vector<DeviceItem> items;
    std::vector<uint32_t> cta_item_begin;
    uint32_t num_partial_slots = 0;   // slots used beyond slot_base
    uint32_t num_counters = 0;        // counters used beyond counter_base
    uint64_t total_kv_tiles = 0;
    bool fine = false;                // short runs: the kernel holds the softmax weights in two parts
    uint32_t num_ctas() const { return cta_item_begin.empty() ? 0u : static_cast<uint32_t>(cta_item_begin.size() - 1); }
};
constexpr uint32_t kChunkTilesPerItem = 8;  // one query tile per warp
// Requests whose query run spans at least this many query tiles always go to the chunk kernels, which read a request's
// K/V once for all of its query rows; the decode kernel reads it once per query tile.
constexpr uint32_t kChunkMinTiles = 5;
constexpr uint32_t kChunkMinPieceTiles = 64;   // a KV piece of a cut unit is at least this many 16-token tiles
constexpr uint32_t kChunkMaxPieces = 16;      // equal shares: a unit is cut into about this many pieces at most
constexpr uint32_t kChunkWholeTokens = 2 * kChunkMinPieceTiles * 16;  // units of at most this many keys are not worth a cut
constexpr uint32_t kChunkStartCostTiles = 8;   // fixed cost of a work item (query load, epilogue) in KV tiles, stream order
// The same in the other orders, for every piece of a unit: query rows, first tiles and epilogue, in the time of 16-token tiles
// (about 7 us).  0 to 64 measured the same on whole units.  Equal shares, two layers, with 12, 16, 20, 24, 28, 32 and 40: 16 requests
// of 512 to 16,384 tokens, eight rows each, 40/8 heads x 128 169, 164, 164, 161, 163, 160 and 162 us; 64 of 100 to 4,000, four rows
// each, 199, 192, 180, 177, 177, 175 and 177; 24 of 300 to 12,000, eight rows, 32/8 x 128 174, 169, 166, 164, 163, 163 and 166; at
// head_dim 256 a little less is better: 24 of 2,500, eight rows, 16/2 heads 102, 102, 100, 105, 108, 107 and 106.
constexpr uint32_t kChunkUnitCostTiles = 28;

// How the units of a chunk plan are dealt to CTAs.
enum class ChunkOrder {
    kStream,       // in stream order to the CTA that is free first; only long units are cut
    kEqualShares,  // contiguous shares of equal size, units cut where a share ends
    kL2Resident    // any order will do, the K/V stays in L2: whole units, longest first, where no unit is long against a
                   // CTA's share; else equal shares
};

// What decides between the decode kernel and the chunk kernels.
struct ChunkRule {
    uint32_t max_ctas = 1;
    uint32_t head_dim = 0;
    uint64_t token_bytes = 0;   // K and V of one token in one layer
    bool short_runs = false;    // the tcgen05 kernel runs: it may take short runs as well
    uint64_t handicap = 0;      // what taking short runs costs beside the attention, in KV tiles per CTA at head_dim 128
};
// Deals a step's requests.  Runs of kChunkMinTiles query tiles always go to the chunk kernels.  In a step without any, the
// runs of two tiles and more (and rows at one position) go there together, with weights in two parts (the result: true),
// when that pays: the decode kernel reads a request's K/V once per query tile, the tcgen05 kernel once, but a unit
// (request, KV head) that is cut is merged by one CTA, and one that is not occupies one CTA.
bool split_runs(const PlanGeometry& geo, const RequestRuns& runs, const ChunkRule& rule, std::vector<uint32_t>& decode_reqs,
                std::vector<uint32_t>& chunk_reqs);
// The order for the requests `split_runs` left to the chunk kernels.
ChunkOrder chunk_order(const PlanGeometry& geo, const RequestRuns& runs, const std::vector<uint32_t>& requests, uint64_t token_bytes);

// Outside stream order an item (a unit, or a piece of one) counts as its KV tiles plus `unit_start_cost`.
ChunkPlan build_chunk_plan(const PlanGeometry& geo, const RequestRuns& runs, const std::vector<uint32_t>& requests, uint32_t max_ctas,
                           uint32_t slot_base, uint32_t counter_base, ChunkOrder order, uint32_t unit_start_cost = 0);

// What a replay reservation for steps of up to `max_tokens` query tokens sets aside: every token a query tile of its own,
// every unit cut at every CTA boundary; a run of the chunk kernels is at least two tokens long.  Of the chunk items only
// pieces of cut units take partial slots, eight a piece.  In equal shares a CTA holds at most two such pieces.  In stream
// order a unit is cut where it is longer than half a CTA's share, so its pieces are at least a quarter of a share each: at
// most four a CTA, and at most two a CTA and one a unit.
struct ReplayCapacity {
    uint64_t items = 0, reduces = 0, chunk_items = 0, slots = 0;
};
ReplayCapacity replay_capacity(const PlanGeometry& geo, uint32_t max_tokens, uint32_t max_ctas, bool chunks);

// Device form of a finished plan.
std::vector<DeviceItem> flatten_plan(const WorkPlan& plan, const PlanGeometry& geo);

// ---- RoPE parameters (crates/inference-backend-metal/src/components/rms_norm_rope.rs:126-230) ---------------------
struct RopeParameters {
    std::vector<float> inverse_frequencies;  // rope_dim / 2
    float attention_factor = 1.0f;
    float correction_low = 0.0f, correction_high = 0.0f;  // Yarn only
};
RopeParameters rope_parameters(const psi_norm_rope_config& config);

// ---- page-ID allocator (crates/inference-runtime-core/src/memory/u32_id_allocator.rs) --------------------------------
class IdAllocator {
public:
    explicit IdAllocator(uint64_t capacity);
    void alloc_many(uint64_t count, uint32_t* out);
    void free_many(const uint32_t* ids, uint64_t count);
    const std::vector<uint64_t>& bitmap() const { return bitmap_; }
    uint64_t free_count() const { return free_ids_.size() + (capacity_ - counter_); }

private:
    void mark(uint32_t id, bool live);
    uint64_t capacity_;
    uint64_t counter_ = 0;
    std::deque<uint32_t> free_ids_;
    std::vector<uint64_t> bitmap_;
};

}  // namespace psi
