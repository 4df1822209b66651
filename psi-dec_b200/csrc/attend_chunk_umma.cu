// Multi-query attention for long query runs on the 5th-generation tensor cores (tcgen05 / TMEM), K/V staged by TMA.
//
// Same work items as attend_chunk.cu (a super-tile of up to eight 16-row query tiles of one request and KV head: 128
// rows = one native UMMA M tile), different engine.  Per CTA (352 threads at head_dim 256, 384 at 128; 512 TMEM columns, a
// shared-memory ring of K/V tiles of 64 tokens):
//   warps 0-3 and 4-7 (row warpgroups): a thread of the first and one of the second share an accumulator row.  They stage the
//       query rows in TMEM as an MMA A operand, half of the columns each (the next item's rows go in before the current item's
//       output is written), read S rows from TMEM (tcgen05.ld), apply the causal limit and the online softmax without any
//       cross-thread traffic, write P back over the S buffer as the A operand of P V, rescale their O row in TMEM only when the
//       running max ran away from the reference the exponentials are taken against; then the epilogue, half of the columns
//       each, partial slots and last-arriver merge as in attend_chunk.cu.  At head_dim 128 they take alternate tiles, each
//       with a softmax state and an O of its own, merged at the end of the item; at 256 the TMEM holds one O only, the first
//       warpgroup takes all tiles and the second sleeps until the item ends.
//   warp 8 (head_dim 128: 8 and 11): issues the MMAs from converged code with one elected lane (operands then stay in uniform
//       registers)
//         S[128x64]  = Q[128xD] . K^T    (Q from TMEM, K as a K-major shared-memory operand, two or three S buffers)
//         O[128xD]  += P[128x64] . V     (P from TMEM, V as an MN-major shared-memory operand)
//       so that Q K^T of tile i+1 runs under the softmax of tile i and P V of tile i under the softmax of tile i+1.
//   warps 9 and 10: bring the K and V tiles from their pages by TMA, 5-D boxes that land in exactly the order the MMA
//       descriptors read ([8-row group][64-element block][8 rows][64 elements], 128-byte swizzle); an item's last, ragged
//       tile is copied with zero-filling 16-byte cp.async instead.
// What bounds a tile: at head_dim 256 the row threads (1,330 cycles: 512 of the special-function unit, and the latencies of
// loads, maxima and stores around them) a little ahead of the tensor pipe (1,025); at 128 HBM, 6.4 to 7.3 TB/s while tiles
// stream.  Beside its tiles an item costs query rows, the fill of the pipeline and the epilogue (6 us at head_dim 256 with
// gates, 3 without; 11 and 6 with one warpgroup), a cut one also the arrival (1.2 us) and for the last piece the merge (2.5
// us; 4.6 when the eight tiles are merged one by one).  Prompts have many short items, so rows are packed (a group of six
// fills 126 of 128 rows, not 96) and the plan deals whole units.  Three prompts of 611 to 2,500 tokens, 24/4 heads x 256,
// gated: 135 us a layer, 162 with one row warpgroup.  16 requests of 512 to 16,384 tokens, eight rows each, 40/8 heads x
// 128: 72 us a layer, 80.
// All hand-offs are mbarriers (TMA byte counts, tcgen05.commit, thread arrivals); every wait is bounded and reports
// PSI_ERR_TIMEOUT through the status word instead of hanging, and the kernel frees its TMEM on every path.  The kernel
// reads pages only: a step that appends and attends runs the append launch first.
//
// Arithmetic replaced: crates/inference-backend-metal/src/components/metal/gqa_split_kv_tiled_q.metal:49-378.
#include <cuda.h>

#include <mutex>
#include <type_traits>

#include "launch_util.hpp"
#include "mma_common.cuh"
#include "tma_common.cuh"

namespace psi {


namespace {

constexpr uint32_t kRowThreads = 256;   // warps 0-7: half an accumulator row per thread
constexpr uint32_t kRowWarps = kRowThreads / 32;
// + a warp that issues the MMAs (two where the row warpgroups take alternate tiles) and two that bring K and V tiles into the ring
template <int D>
constexpr uint32_t kUmmaThreads = kRowThreads + (D == 128 ? 128 : 96);
constexpr uint32_t kUmmaM = 128;   // query rows per CTA = TMEM lanes
constexpr uint32_t kUmmaN = 64;    // KV tokens per tile

// Shared-memory matrix descriptor of a 128-byte-swizzled operand: start address, leading / stride byte offsets in
// 16-byte units, descriptor version 1, layout type 2 (SWIZZLE_128B).
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t leading_bytes, uint32_t stride_bytes) {
    return static_cast<uint64_t>((addr >> 4) & 0x3FFFu) | (static_cast<uint64_t>((leading_bytes >> 4) & 0x3FFFu) << 16) |
           (static_cast<uint64_t>((stride_bytes >> 4) & 0x3FFFu) << 32) | (1ull << 46) | (2ull << 61);
}

// Instruction descriptor of kind::f16: f32 accumulator, A/B element format (0 = f16, 1 = bf16), B major (0 = K,
// 1 = MN), N >> 3 and M >> 4.
template <typename T>
__device__ __forceinline__ uint32_t umma_idesc(uint32_t n, bool b_mn_major) {
    const uint32_t format = sizeof(T) == 2 && std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
    return (1u << 4) | (format << 7) | (format << 10) | ((b_mn_major ? 1u : 0u) << 16) | ((n >> 3) << 17) |
           ((kUmmaM >> 4) << 24);
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred e;\n\telect.sync _|e, 0xFFFFFFFF;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}\n" ::"r"(bar)
        : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 consecutive f32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_load32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
        "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_load16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// 64 consecutive columns, both loads under way before the wait.
__device__ __forceinline__ void tmem_load64(uint32_t taddr, float (&v)[64]) {
    uint32_t r[64];
#pragma unroll
    for (int h = 0; h < 64; h += 32)
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
            "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
            : "=r"(r[h]), "=r"(r[h + 1]), "=r"(r[h + 2]), "=r"(r[h + 3]), "=r"(r[h + 4]), "=r"(r[h + 5]), "=r"(r[h + 6]), "=r"(r[h + 7]),
              "=r"(r[h + 8]), "=r"(r[h + 9]), "=r"(r[h + 10]), "=r"(r[h + 11]), "=r"(r[h + 12]), "=r"(r[h + 13]), "=r"(r[h + 14]),
              "=r"(r[h + 15]), "=r"(r[h + 16]), "=r"(r[h + 17]), "=r"(r[h + 18]), "=r"(r[h + 19]), "=r"(r[h + 20]), "=r"(r[h + 21]),
              "=r"(r[h + 22]), "=r"(r[h + 23]), "=r"(r[h + 24]), "=r"(r[h + 25]), "=r"(r[h + 26]), "=r"(r[h + 27]), "=r"(r[h + 28]),
              "=r"(r[h + 29]), "=r"(r[h + 30]), "=r"(r[h + 31])
            : "r"(taddr + h));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 64; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_store32(uint32_t taddr, const float (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
        "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};\n" ::"r"(taddr),
        "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])),
        "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])),
        "r"(__float_as_uint(v[8])), "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
        "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])), "r"(__float_as_uint(v[15])),
        "r"(__float_as_uint(v[16])), "r"(__float_as_uint(v[17])), "r"(__float_as_uint(v[18])), "r"(__float_as_uint(v[19])),
        "r"(__float_as_uint(v[20])), "r"(__float_as_uint(v[21])), "r"(__float_as_uint(v[22])), "r"(__float_as_uint(v[23])),
        "r"(__float_as_uint(v[24])), "r"(__float_as_uint(v[25])), "r"(__float_as_uint(v[26])), "r"(__float_as_uint(v[27])),
        "r"(__float_as_uint(v[28])), "r"(__float_as_uint(v[29])), "r"(__float_as_uint(v[30])), "r"(__float_as_uint(v[31]))
        : "memory");
}

__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

__device__ __forceinline__ void row_threads_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

// The two warps that share 32 accumulator rows (warp w and w + 4, `rows` = w % 4).
__device__ __forceinline__ void row_pair_sync(uint32_t rows) {
    __syncwarp();
    asm volatile("bar.sync %0, 64;" ::"r"(rows + 2) : "memory");
}

// One of the two says that it has come this far; the other waits for it.
__device__ __forceinline__ void row_pair_arrive(uint32_t rows) {
    __syncwarp();
    asm volatile("bar.arrive %0, 64;" ::"r"(rows + 6) : "memory");
}
__device__ __forceinline__ void row_pair_wait(uint32_t rows) {
    __syncwarp();
    asm volatile("bar.sync %0, 64;" ::"r"(rows + 6) : "memory");
}

// Executed by a whole converged warp; one elected lane (always the same one for a full warp) issues.
__device__ __forceinline__ void umma_issue_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\telect.sync _|e, 0xFFFFFFFF;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void tmem_store32_bits(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
        "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};\n" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
        "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]),
        "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]),
        "r"(v[31])
        : "memory");
}

__device__ __forceinline__ void tmem_store16_bits(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
        "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}

// Two f32 operations an instruction.
__device__ __forceinline__ uint64_t pack_f32x2(float a, float b) {
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ float2 unpack_f32x2(uint64_t v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
    return v;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
    uint64_t v;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float v;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(v) : "f"(a), "f"(b), "f"(c));
    return v;
}

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Shared-memory ring slots of one K or V tile, and how far the lazily kept softmax reference may lag the running max
// (log2 domain): P then stays below 2^8, well inside bf16/f16, and O is rescaled only on a real jump.
constexpr uint32_t kSlots = 6, kSlotBytes = 32 * 1024;  // a K or a V tile at head_dim 256, both of them at 128
constexpr float kRescaleThreshold = 8.0f;
// Launches over short query runs and rows at one position (kFine) carry the weights as two 16-bit parts, each with a P V of
// its own, over the two halves of the S buffer: the decode kernel, the other one that takes these rows, keeps a maximum per
// warp and rounds less than one part would.  Against 64 bits, seven draft rows a request over a history of 512 to 12,288
// tokens, 40/8 heads x 128: 1.6e-3 with one part, 1.3e-3 on the decode kernel, 8e-6 with two.  The high part is rounded down
// and the low part holds the rest plus 2^-10 of the weight, so that both are positive wherever the weight is (an infinity in
// V stays one instead of meeting 0 x Inf); every weight is then 1 + 2^-10 times itself, which the end of the item divides out.
// Costs 5 to 12 % of such a step (16 requests of 512 to 16,384 tokens, eight rows each, 40/8 heads x 128, two layers, with one
// row warpgroup: 164 us with one part, 184 with two; 275 on the decode kernel).  Long runs keep one part, in code of their own: a branch on the
// kind inside the MMA warp's loop alone cost them 3 %.
constexpr float kFineScale = 1.0009765625f;
static_assert(offsetof(DeviceItem, flat_begin) == 24 && offsetof(DeviceItem, num_tokens) == 28 && offsetof(DeviceItem, head0) == 40 &&
                  offsetof(DeviceItem, num_heads) == 44,
              "the row threads read these fields of the next item as the ends of two 16-byte words");
constexpr uint32_t kUmmaStageColumns = 64;  // columns of the row warps' staging areas

// 8-byte global->shared copy; src_bytes == 0 zero-fills.
__device__ __forceinline__ void cp_async_8(uint32_t dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ uint4 ld_shared_16(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void st_shared_16(uint32_t addr, uint4 v) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};\n" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// What the rounding down of two weights left (see kFineScale).
template <typename T>
__device__ __forceinline__ uint32_t low_part(float a, float b, uint32_t high) {
    const float2 h = Mma<T>::unpack(high);
    return Mma<T>::pack(fmaf(a, kFineScale, -h.x), fmaf(b, kFineScale, -h.y));
}

struct UmmaShared {
    uint64_t bars[3 * kSlots + 5];
    uint32_t tmem_base, abort, last[8];
    uint32_t cleaned[2];  // by item parity: the item (its index + 1) in whose V tiles values were replaced
    float half[2][kUmmaM];  // what the two threads of a row tell each other
};

// Whether one of two packed 16-bit values is infinite or no number.
template <typename T>
__device__ __forceinline__ bool any_not_finite(uint32_t two) {
    constexpr uint32_t kExponent = std::is_same<T, __half>::value ? 0x7C00u : 0x7F80u;
    return (two & kExponent) == kExponent || (two >> 16 & kExponent) == kExponent;
}

template <typename T, int D, bool kFine>
__device__ __forceinline__ void attend_chunk_umma(const AttendParams& p, const CUtensorMap& kv_map, const uint32_t box_rows,
                                                  const bool early, UmmaShared& shared) {
    constexpr uint32_t kChunks = D / 8;               // 16-byte chunks per row of K / V
    constexpr uint32_t kBlocks = D / 64;              // 64-element (128-byte) blocks per row
    constexpr uint32_t kTmemColumns = 512;
    // At head_dim 128 the two row warpgroups take alternate tiles, each into an accumulator of its own (`streams`, merged at
    // the end of an item); at 256, where O takes half of the TMEM, the first takes them all and the second helps at the ends of
    // items.  (Half of every tile's tokens each, with a barrier a tile, was no faster, since the special-function unit takes
    // half of a tile's time for either split, and cost a power-limited step of long runs 2 to 4 %.)
    constexpr uint32_t kStreams = D == 128 ? 2 : 1, kBuffers = D == 128 ? 3 : 2;  // (S buffers)
    // At head_dim 128 a TMA box brings the K and the V rows of a page piece, which share a ring slot, [8-row group][K, V]: boxes of
    // eight-token pages hold 2 KiB otherwise, and as many as a tile then takes keep a producer warp busy for longer than a
    // tile lasts.  kGroupKib: from one 8-row group of a tile to the next; kValues: V in its slot.
    constexpr bool kJoint = D == 128;
    constexpr uint32_t kGroupKib = kJoint ? 2 * kBlocks : kBlocks, kValues = kJoint ? kBlocks * 1024 : 0, kSlotStep = kJoint ? 1 : 2;
    static_assert((kJoint ? 2 : 1) * D * 2 * kUmmaN == kSlotBytes, "what a slot holds");
    // TMEM columns: Q as an MMA A operand (two 16-bit elements per column), the S buffers, whose first half is overwritten
    // by P (again two elements per column), O of every stream
    constexpr uint32_t kColQ = 0, kColS = D / 2, kColO = kColS + kBuffers * kUmmaN;
    static_assert(kColO + kStreams * D <= kTmemColumns, "Q, S and O share one TMEM allocation");
    constexpr uint32_t kStageColumns = kUmmaStageColumns, kStageBytes = 32 * kStageColumns * 2;  // staging area of a row warp
    // barriers
    constexpr uint32_t kBarFull = 0, kBarDone = kSlots, kBarS = kJoint ? 2 * kSlots : kBarDone, kBarP = (kJoint ? 3 : 2) * kSlots,
                       kBarQ = kBarP + 2 * kStreams, kNumBarriers = kBarQ + 1;

    static_assert(kNumBarriers <= sizeof(UmmaShared::bars) / sizeof(uint64_t), "every barrier has a word");

    const uint32_t cta = blockIdx.x;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    uint32_t& tmem_base_s = shared.tmem_base;
    uint32_t& abort_s = shared.abort;
    uint32_t (&last_s)[8] = shared.last;

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // the swizzled operand layouts repeat every 1024 bytes: place them on that boundary whatever the toolchain did
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bar0 = smem_u32(shared.bars);
    auto bar = [&](uint32_t which) { return bar0 + which * 8; };

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)),
                     "r"(kTmemColumns)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (uint32_t b = 0; b < kBarP; ++b) mbar_init(bar(b), kJoint && b < kBarDone ? 2 : 1);  // (a joint slot is filled by two warps)
        for (uint32_t b = kBarP; b < kBarQ; ++b) mbar_init(bar(b), kUmmaM);
        mbar_init(bar(kBarQ), kRowWarps);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        abort_s = 0;
        shared.cleaned[0] = shared.cleaned[1] = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    const uint32_t page_mask = p.geo.tokens_per_page - 1;
    const uint32_t page_shift = 31 - __clz(p.geo.tokens_per_page);
    const unsigned char* pages = static_cast<const unsigned char*>(p.geo.pages);
    const uint64_t page_bytes = p.geo.page_elems * 2;
    const uint64_t v_region_bytes = v_region_offset(p.geo) * 2;

    // A wait that ran out flags the launch and lets every later wait fall through: results are then garbage, the
    // status word says so, and the kernel still frees its TMEM and returns.
    auto wait = [&](uint32_t which, uint32_t parity) {
        if (mbar_try(bar(which), parity & 1)) return;  // the usual case: complete at once or soon
        if (*reinterpret_cast<volatile uint32_t*>(&abort_s) == 0 && !mbar_wait(bar(which), parity & 1)) {
            abort_s = 1;
            if (p.status != nullptr) atomicExch(p.status, static_cast<uint32_t>(PSI_ERR_TIMEOUT));
        }
    };

    // Tiles and items are counted over the whole launch, the same way in every role; tile t belongs to stream t % kStreams.  Its
    // K and V take ring slots 2t and 2t + 1 modulo kSlots, or share slot t modulo kSlots.  The product over a slot's tile
    // completes the slot's "done" barrier, which frees the slot and says that O of the tile is there, or S where K has slots
    // of its own; S has barriers of its own where K and V share a slot.  P has two barriers per stream, taken in turn by its
    // tiles, and Q takes the item count.
    // A parity wait cannot tell two completions from none: nobody waits for a phase whose predecessor may be outstanding or
    // whose successor may be complete.  A slot's next product needs the P of a tile behind this one, so its barrier cannot run
    // ahead of a row thread; S is seen tile by tile, and O is waited for only where it is rescaled or read, but S of tile t
    // says that P V of tile t - kBuffers, whose place it took, is complete, and those before it: the previous use of any V slot
    // lies further back.
    static_assert(kSlots / kSlotStep >= kBuffers + 1 && kSlots % kSlotStep == 0, "the ring holds more tiles than there are S buffers");
    constexpr uint32_t kRingTiles = kSlots / kSlotStep;
    auto v_done = [](uint32_t tile) { return kBarDone + tile % kRingTiles * kSlotStep + (kSlotStep - 1); };
    auto slot_phase = [](uint32_t tile) { return tile / kRingTiles; };
    auto stream_barrier = [](uint32_t tile) { return kStreams == 2 ? (tile & 1u) * 2 + (tile >> 1 & 1u) : tile & 1u; };
    auto stream_phase = [](uint32_t tile) { return kStreams == 2 ? tile >> 2 : tile >> 1; };
    // A tile with its ring slot, that slot's phase and its S buffer, counted along: the divisions are on nobody's chain.
    struct Place {
        uint32_t tile, slot, phase, buffer;
        __device__ __forceinline__ void advance() {
            ++tile;
            slot += kSlotStep;
            if (slot >= kSlots) {
                slot -= kSlots;
                ++phase;
            }
            buffer = buffer + 1 == kBuffers ? 0 : buffer + 1;
        }
    };
    uint32_t tile_base = 0, item_count = 0;
    const uint32_t item_begin = p.cta_item_begin[cta], item_end = p.cta_item_begin[cta + 1];
    if (early && warp >= kRowWarps) await_previous_kernel();  // (the row threads: once they know their first rows)

    if (warp == kRowWarps + 1 || warp == kRowWarps + 2) {
        // ================================ producers: K and V tiles into the ring ========================================
        // A warp each for K and V, or for the rows 0 to 31 and 32 to 63 of joint tiles.
        const uint32_t which = warp - kRowWarps - 1;
        const uint32_t v_groups = p.geo.num_kv_heads * p.geo.tokens_per_page / 8;  // 8-row groups of a page's K region
        constexpr uint32_t kRows = kJoint ? kUmmaN / 2 : kUmmaN;  // of a tile that this warp brings
        const uint32_t row0 = kJoint ? which * kRows : 0;
        Place place{0, kJoint ? 0u : which, 0, 0};
        for (uint32_t index = item_begin; index < item_end; ++index) {
            const ItemView v = view_item(p, index);
            const uint32_t* row_ids = table_row(p.geo, v.req_slot);
            const uint64_t head_bytes = static_cast<uint64_t>(v.kv_head) * p.geo.tokens_per_page * (D * 2);
            const uint32_t head_group = v.kv_head * p.geo.tokens_per_page / 8;
            const uint32_t first_tile = v.kv_begin / kUmmaN;
            const uint32_t num_tiles = (v.kv_end + kUmmaN - 1) / kUmmaN - first_tile;
            const uint32_t last_page = (v.kv_end - 1) >> page_shift;
            // 32 page ids of the request, one per lane, and the 32 behind them, requested a window ahead
            uint32_t window_base = first_tile * kUmmaN >> page_shift;
            auto window_at = [&](uint32_t base) { return base + lane <= last_page ? page_id_or_zero(p.geo, row_ids, base + lane) : 0u; };
            uint32_t window_ids = window_at(window_base), next_ids = window_at(window_base + 32);
            for (uint32_t i = 0; i < num_tiles; ++i, place.advance()) {
                const uint32_t token0 = (first_tile + i) * kUmmaN;
                if ((token0 >> page_shift) >= window_base + 32) {  // (a tile's pages do not straddle windows: both are powers of two)
                    window_base += 32;
                    window_ids = next_ids;
                    next_ids = window_at(window_base + 32);
                }
                const uint32_t slot = place.slot, dst = smem_base + slot * kSlotBytes;
                if (place.phase > 0) wait(kBarDone + slot, place.phase - 1);  // the MMAs that read the slot's previous tile are done
                __syncwarp();
                if (token0 + kUmmaN <= v.kv_end) {
                    if (lane == 0) mbar_expect_tx(bar(kBarFull + slot), kSlotBytes * kRows / kUmmaN);
                    auto load_box = [&](uint32_t row) {
                        const uint32_t token = token0 + row;
                        const uint32_t page = __shfl_sync(0xFFFFFFFFu, window_ids, (token >> page_shift) - window_base);
                        const uint32_t group = head_group + (token & page_mask) / 8, to = dst + (row / 8) * (kGroupKib * 1024);
                        if constexpr (kJoint) tma_load_pair(to, &kv_map, bar(kBarFull + slot), page * (2 * v_groups) + group);
                        else tma_load_groups(to, &kv_map, bar(kBarFull + slot), which * v_groups + group, page);
                    };
                    // (the two small boxes by loops of a known length, whose addresses are worked out side by side)
                    if (box_rows == 8) {
#pragma unroll
                        for (uint32_t row = 0; row < kRows; row += 8) load_box(row0 + row);
                    } else if (box_rows == 16) {
#pragma unroll
                        for (uint32_t row = 0; row < kRows; row += 16) load_box(row0 + row);
                    } else {
                        for (uint32_t row = 0; row < kRows; row += box_rows) load_box(row0 + row);
                    }
                } else {
                    // the item's last tile: rows at and beyond its end are zero
                    for (uint32_t values = kJoint ? 0 : which; values < (kJoint ? 2 : which + 1); ++values) {
                        for (uint32_t c = lane; c < kRows * kChunks; c += 32) {
                            const uint32_t row = row0 + c / kChunks, chunk = c % kChunks;
                            const uint32_t token = token0 + row;
                            const bool valid = token < v.kv_end;
                            const uint32_t page =
                                __shfl_sync(0xFFFFFFFFu, window_ids, valid ? (token >> page_shift) - window_base : 0u);
                            const unsigned char* src = pages + static_cast<uint64_t>(page) * page_bytes + head_bytes +
                                                       (values ? v_region_bytes : 0) + (token & page_mask) * (D * 2) + chunk * 16;
                            cp_async_16(dst + (values ? kValues : 0) + operand_offset(kGroupKib, row, chunk), valid ? src : pages, valid ? 16u : 0u);
                        }
                    }
                    cp_async_commit();
                    cp_async_wait<0>();
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar(kBarFull + slot));
                }
                __syncwarp();
            }
        }
        // the CTA does not go away with its own bulk copies in flight: every slot's last fill has landed (a bounded
        // wait of its own, also after an earlier wait gave up)
        for (uint32_t back = 1; back <= kRingTiles && back <= place.tile; ++back) {
            const uint32_t tile = place.tile - back;
            mbar_wait(bar(kBarFull + tile % kRingTiles * kSlotStep + (kJoint ? 0 : which)), slot_phase(tile) & 1);
        }
    } else if (warp >= kRowWarps) {
        // ================================ MMA issue (converged warp, one elected lane) ================================
        {
            const uint32_t idesc_qk = umma_idesc<T>(kUmmaN, false);
            const uint32_t idesc_pv = umma_idesc<T>(D, true);
            Place qk{0, 0, 0, 0}, pv{0, kSlotStep - 1, 0, 0};
            for (uint32_t index = item_begin; index < item_end; ++index, ++item_count) {
                const ItemView v = view_item(p, index);
                const uint32_t first_tile = v.kv_begin / kUmmaN;
                const uint32_t num_tiles = (v.kv_end + kUmmaN - 1) / kUmmaN - first_tile;
                // S[qk.buffer] = Q K^T of the next tile, whose K tile is there
                auto issue_qk = [&] {
                    // K-major operand: 8-row groups kGroupKib KiB apart; per k-step the start moves to element block ks / 4
                    // and 32 bytes on inside it (the start-address field counts 16-byte units)
                    const uint64_t k_desc = umma_desc(smem_base + qk.slot * kSlotBytes, 16, kGroupKib * 1024);
                    const uint32_t s_tmem = tmem + kColS + qk.buffer * kUmmaN;
#pragma unroll
                    for (uint32_t ks = 0; ks < uint32_t(D) / 16; ++ks)
                        umma_issue_ts(s_tmem, tmem + kColQ + ks * 8, k_desc + ((ks >> 2) * 1024 + (ks & 3) * 32) / 16, idesc_qk, ks > 0);
                    umma_commit(bar(kBarS + qk.slot));
                    qk.advance();
                };
                // O (+)= P V of the next tile, whose V tile and P (over the first half of its S buffer) are there
                auto issue_pv = [&](uint32_t accumulate) {
                    // MN-major operand: 64-element blocks 1 KiB apart, 8-token groups kGroupKib KiB apart, two groups per
                    // k-step
                    const uint64_t v_desc = umma_desc(smem_base + pv.slot * kSlotBytes + kValues, 1024, kGroupKib * 1024);
                    const uint32_t p_tmem = tmem + kColS + pv.buffer * kUmmaN;
                    const uint32_t o_tmem = tmem + kColO + (kStreams == 2 ? (pv.tile & 1u) * D : 0u);
#pragma unroll
                    for (uint32_t ks = 0; ks < kUmmaN / 16; ++ks)
                        umma_issue_ts(o_tmem, p_tmem + ks * 8, v_desc + ks * 2 * (kGroupKib * 1024) / 16, idesc_pv, ks > 0 ? 1u : accumulate);
                    if constexpr (kFine) {  // the low parts of P, over the second half of the S buffer
#pragma unroll
                        for (uint32_t ks = 0; ks < kUmmaN / 16; ++ks)
                            umma_issue_ts(o_tmem, p_tmem + kUmmaN / 2 + ks * 8, v_desc + ks * 2 * (kGroupKib * 1024) / 16, idesc_pv, 1u);
                    }
                    umma_commit(bar(kBarDone + pv.slot));
                    pv.advance();
                };

                if constexpr (kStreams == 2) {
                    // Q K^T and P V from a warp each: the tensor pipe works off a queue of a few products, and a single warp that
                    // looks at its barriers and works out addresses between two batches lets it run dry (500 of 1,450 cycles a
                    // tile).  Three S buffers leave room for Q K^T to wait until P V of the buffer's last tile is complete.
                    if (warp == kRowWarps) {
                        wait(kBarQ, item_count);  // the item's query rows are in TMEM; the rows are done with the previous item
                        for (uint32_t i = 0; i < num_tiles; ++i) {
                            if (qk.tile >= kBuffers) wait(v_done(qk.tile - kBuffers), slot_phase(qk.tile - kBuffers));
                            wait(kBarFull + qk.slot, qk.phase);
                            tc_fence_after();
                            issue_qk();
                        }
                    } else {
                        for (uint32_t i = 0; i < num_tiles; ++i) {
                            wait(kBarFull + pv.slot, pv.phase);
                            wait(kBarP + stream_barrier(pv.tile), stream_phase(pv.tile));
                            tc_fence_after();
                            issue_pv(i >= kStreams);
                        }
                    }
                } else {
                    // One warp, in the order of the pipe: with two S buffers Q K^T of tile i + 2 has to follow P V of tile i, and a second
                    // warp that waits for its completion is slower (2,970 us of long runs against 2,670).
                    auto next_qk = [&] {
                        wait(kBarFull + qk.slot, qk.phase);
                        tc_fence_after();
                        issue_qk();
                    };
                    wait(kBarQ, item_count);  // the item's query rows are in TMEM; the rows are done with the previous item
                    if (num_tiles > 0) next_qk();
                    for (uint32_t i = 0; i < num_tiles; ++i) {
                        if (i + 1 < num_tiles) next_qk();  // runs under the softmax of tile i
                        wait(kBarFull + pv.slot, pv.phase);
                        wait(kBarP + stream_barrier(pv.tile), stream_phase(pv.tile));
                        tc_fence_after();
                        issue_pv(i >= kStreams);
                    }
                }
                tile_base += num_tiles;
            }
        }
    } else {
        // ================================ half an accumulator row per thread ===========================================
        // Warps w and w + 4 share the rows of TMEM lanes 32 w to 32 w + 31 (w < 4): they take the tiles of a stream each, or the
        // first takes all; of Q and the output each takes half of the columns.
        const uint32_t rows_warp = warp & 3u, half = warp >> 2, row_id = tid & (kUmmaM - 1);
        const uint32_t lane_base = (rows_warp * 32u) << 16;  // this warp's TMEM lanes
        const uint32_t tmem_o = tmem + kColO + (kStreams == 2 ? half * D : 0u);  // what this warp rescales
        constexpr uint32_t kHalfD = D / 2;
        const uint32_t column0 = half * kHalfD;
        const bool wide_gates = (reinterpret_cast<uintptr_t>(p.gates) & 15u) == 0;
        const bool wide_out = (reinterpret_cast<uintptr_t>(p.out) & 15u) == 0;
        // Row of this thread in an item: row row_id = (token row_id / heads, head row_id % heads) of the super-tile, packed
        // without gaps; w and rr are its 16-row tile and its row inside it, the unit of partial slots and arrival counters.
        const uint32_t w = row_id >> 4, rr = row_id & 15;
        auto row_of = [&](const ItemView& v, bool& valid) {
            valid = row_id < v.rows;
            return static_cast<uint64_t>(v.flat_begin + (valid ? row_id / v.num_heads : 0)) * p.num_q_heads + v.head0 +
                   (valid ? row_id % v.num_heads : 0);
        };
        // What the other thread of this row has (all threads of both warps take part).  A value goes where this thread has
        // just read the other one's last value and nobody else reads, so one barrier an exchange is enough.
        uint32_t place_of_mine = half;
        auto exchange = [&](float mine) {
            tc_fence_before();
            shared.half[place_of_mine][row_id] = mine;
            row_pair_sync(rows_warp);
            place_of_mine ^= 1u;
            const float theirs = shared.half[place_of_mine][row_id];
            tc_fence_after();
            return theirs;
        };
        auto warp_arrive = [&](uint32_t which) {
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(which));
        };
        // Rows of q, the gates and the output pass through a staging area of this warp, 32 rows x 64 columns: one thread per
        // row would touch 32 lines with every access, so global memory is read and written several rows at a time and
        // every thread reads or writes its own row in shared memory (16-byte chunks XOR-ed with the row: no bank conflicts).
        // Gates and output take it as two buffers of 32 columns, so that gates travel under the arithmetic of the other one.
        const uint32_t stage = smem_base + kSlots * kSlotBytes + warp * kStageBytes;
        constexpr uint32_t kStageChunks = kStageColumns / 8;
        const uint32_t stage_row = lane / kStageChunks, stage_chunk = lane % kStageChunks;  // of a copy of four rows
        auto stage_at = [&](uint32_t row, uint32_t chunk) { return stage + row * (kStageColumns * 2) + ((chunk ^ (row & 7u)) << 4); };
        // Starts the copy of columns [c0, c0 + 64) of this warp's rows; `row` is this thread's row of `base`, and rows at
        // and beyond `rows` become zero.
        auto stage_in = [&](const void* base, uint32_t row, uint32_t rows, uint32_t c0, bool wide) {
#pragma unroll 4
            for (uint32_t i = 0; i < 32; i += 32 / kStageChunks) {
                const uint32_t r = i + stage_row;
                const bool valid = rows_warp * 32 + r < rows;
                const T* src = static_cast<const T*>(base) + static_cast<uint64_t>(__shfl_sync(0xFFFFFFFFu, row, r)) * D + c0 + stage_chunk * 8;
                if (wide) {
                    cp_async_16(stage_at(r, stage_chunk), src, valid ? 16u : 0u);
                } else {
                    cp_async_8(stage_at(r, stage_chunk), src, valid ? 8u : 0u);
                    cp_async_8(stage_at(r, stage_chunk) + 8, src + 4, valid ? 8u : 0u);
                }
            }
            cp_async_commit();
        };
        auto narrow_at = [&](uint32_t row, uint32_t chunk, uint32_t buffer) {
            return stage + buffer * (kStageBytes / 2) + row * kStageColumns + ((chunk ^ (row >> 1 & 3u)) << 4);
        };
        auto stage_gates = [&](uint32_t row, uint32_t rows, uint32_t c0, uint32_t buffer) {
#pragma unroll
            for (uint32_t i = 0; i < 32; i += 8) {
                const uint32_t r = i + (lane >> 2), chunk = lane & 3u;
                const bool valid = rows_warp * 32 + r < rows;
                const T* src = static_cast<const T*>(p.gates) + static_cast<uint64_t>(__shfl_sync(0xFFFFFFFFu, row, r)) * D + c0 + chunk * 8;
                const uint32_t dst = narrow_at(r, chunk, buffer);
                if (wide_gates) {
                    cp_async_16(dst, src, valid ? 16u : 0u);
                } else {
                    cp_async_8(dst, src, valid ? 8u : 0u);
                    cp_async_8(dst + 8, src + 4, valid ? 8u : 0u);
                }
            }
        };
        // This warp's half of its query rows of an item into their TMEM lanes (zero for rows the super-tile does not have),
        // 64 columns at a time, the first of which have been requested into the staging area.  Called when every Q K^T of the
        // previous item has completed.
        auto put_q = [&](uint32_t c0) {
            cp_async_wait<0>();
            __syncwarp();
            uint32_t regs[32];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint4 value = ld_shared_16(stage_at(lane, j));
                regs[4 * j] = value.x;
                regs[4 * j + 1] = value.y;
                regs[4 * j + 2] = value.z;
                regs[4 * j + 3] = value.w;
            }
            __syncwarp();
            tmem_store32_bits(tmem + kColQ + lane_base + c0 / 2, regs);
        };
        auto first_q = [&](uint32_t row, uint32_t rows) {
            put_q(column0);
            if constexpr (kHalfD > kStageColumns) stage_in(p.q, row, rows, column0 + kStageColumns, true);
        };
        auto rest_of_q = [&] {
            if constexpr (kHalfD > kStageColumns) put_q(column0 + kStageColumns);
            tmem_store_wait();
            tc_fence_before();
            warp_arrive(kBarQ);
        };
        static_assert(kHalfD <= 2 * kStageColumns, "a warp's half of the query columns passes in at most two pieces");

        if (item_begin < item_end) {
            const ItemView first = view_item(p, item_begin);
            bool valid;
            const uint32_t row = static_cast<uint32_t>(row_of(first, valid));
            if (early) await_previous_kernel();  // the query rows are requested before the K and V tiles fill the way to memory
            stage_in(p.q, row, first.rows, column0, true);
            first_q(row, first.rows);
            rest_of_q();
        } else if (early) {
            await_previous_kernel();
        }
        // flat_begin, num_tokens (.z, .w) and head0, num_heads (.z, .w) of the item behind the current one.  They are
        // requested an item ahead and the rows staged before the tile loop: a load in flight across the loop, or the staging
        // inside it, cost 9 % of a long run (1,247 TFLOP/s against 1,378 on 512-token chunks of long prompts).
        const uint32_t start = kStreams == 2 ? half : 0u;
        Place place{start, start * kSlotStep, 0, start};  // of this thread's next S
        uint4 next_rows_of = make_uint4(0, 0, 0, 0), next_heads_of = make_uint4(0, 0, 0, 1);
        auto look_ahead = [&](uint32_t index) {
            const uint4* item = reinterpret_cast<const uint4*>(p.items + min(index, item_end - 1));
            next_rows_of = item[1];
            next_heads_of = item[2];
        };
        if (item_begin < item_end) look_ahead(item_begin + 1);
        for (uint32_t index = item_begin; index < item_end; ++index, ++item_count) {
            const ItemView v = view_item(p, index);
            bool row_valid;
            const uint64_t out_row = row_of(v, row_valid);
            const uint32_t limit = row_valid ? item_row_limit(v, row_id) : v.kv_end;
            const uint32_t min_limit = min(v.kv_end, v.first_pos + 1);
            const uint32_t first_tile = v.kv_begin / kUmmaN;
            const uint32_t num_tiles = (v.kv_end + kUmmaN - 1) / kUmmaN - first_tile;

            // softmax state in the log2 domain: `row_ref` is the reference the exponentials are taken against (it
            // trails the true running max by at most kRescaleThreshold); `row_max` and `row_sum` (relative to the reference) are
            // of this thread's tokens until the item ends
            float row_ref = -INFINITY, row_max = -INFINITY, row_sum = 0.0f;
            // A weight of zero does not hide an infinity: 0 x Inf is no number, and an item of a short run holds up to 128
            // rows, of which those of one query token see one of the step's own keys more than those of the one before.
            // Values that are not finite in V rows that some row of the item must not see are therefore set to zero in the
            // tile, by the row threads while S is at hand, and come back at the end of the item in the rows that see them
            // (the decode kernel's items, tiles of 16 rows, keep such a value to themselves); so are those of the keys before
            // the piece's first, which share its first tile.
            [[maybe_unused]] auto clean_values = [&](uint32_t tile, uint32_t token0) {
                const uint32_t before = max(token0, v.kv_begin) - token0, end = min(token0 + kUmmaN, v.kv_end) - token0;
                const uint32_t first = min(max(token0, min_limit) - token0, end);  // rows [0, before) and [first, end)
                const uint32_t slot = tile % kRingTiles * kSlotStep + (kSlotStep - 1);
                wait(kBarFull + slot, slot_phase(tile));
                bool cleaned = false;
                for (uint32_t i = row_id; i < (before + end - first) * kChunks; i += kUmmaM) {
                    const uint32_t row = i / kChunks < before ? i / kChunks : first - before + i / kChunks;
                    const uint32_t at = smem_base + slot * kSlotBytes + kValues + operand_offset(kGroupKib, row, i % kChunks);
                    uint4 value = ld_shared_16(at);
                    if (!any_not_finite<T>(value.x) && !any_not_finite<T>(value.y) && !any_not_finite<T>(value.z) && !any_not_finite<T>(value.w)) continue;
                    uint32_t* two = &value.x;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        if (any_not_finite<T>(two[k] & 0xFFFFu)) two[k] &= 0xFFFF0000u;
                        if (any_not_finite<T>(two[k] >> 16)) two[k] &= 0xFFFFu;
                    }
                    st_shared_16(at, value);
                    cleaned = true;
                }
                if (!cleaned) return;
                fence_async_smem();
                *reinterpret_cast<volatile uint32_t*>(&shared.cleaned[index & 1]) = index + 1;
            };
            uint32_t next_row = 0, next_rows = 0;  // this thread's row of the next item
            if (index + 1 < item_end) {  // the next item's query rows travel under this item's tiles
                next_rows = next_rows_of.w * next_heads_of.w;
                const uint32_t r = row_id < next_rows ? row_id : 0;
                next_row = (next_rows_of.z + r / next_heads_of.w) * p.num_q_heads + next_heads_of.z + r % next_heads_of.w;
                stage_in(p.q, next_row, next_rows, column0, true);
            }
            const bool more = index + 1 < item_end;
            const uint32_t end_tile = kStreams == 2 || half == 0 ? num_tiles : 0;
            for (uint32_t i = kStreams == 2 ? (tile_base ^ half) & 1u : 0u; i < end_tile; i += kStreams) {
                const uint32_t tile = tile_base + i;
                const uint32_t token0 = (first_tile + i) * kUmmaN;
                const uint32_t tmem_s = tmem + kColS + place.buffer * kUmmaN + lane_base;
                wait(kBarS + place.slot, place.phase);
                place.advance();
                if constexpr (kStreams == 2) place.advance();
                __syncwarp();  // the TMEM accesses below are warp-collective
                tc_fence_after();
                if constexpr (kStreams == 1) {
                    // S of the item's last tile is there: every Q K^T of the item is complete, and the next item's query rows
                    // may take the place of this one's while the softmax below runs
                    if (more && i + 1 == num_tiles) {
                        tc_fence_before();
                        row_pair_arrive(rows_warp);
                        first_q(next_row, next_rows);
                    }
                }

                float s[kUmmaN];
                tmem_load64(tmem_s, s);
                if (token0 < v.kv_begin || token0 + kUmmaN > min_limit) {
#pragma unroll
                    for (int c = 0; c < int(kUmmaN); ++c) {
                        const uint32_t token = token0 + c;
                        if (token >= limit || token < v.kv_begin) s[c] = -INFINITY;
                    }
                    if constexpr (kFine) clean_values(tile, token0);
                }
                float m4[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) m4[k] = fmaxf(s[k], s[k + 4]);
#pragma unroll
                for (int c = 8; c < int(kUmmaN); c += 8)
#pragma unroll
                    for (int k = 0; k < 4; ++k) m4[k] = max3(m4[k], s[c + k], s[c + k + 4]);
                const float tile_max = fmaxf(max3(m4[0], m4[1], m4[2]), m4[3]) * p.scale_log2;  // scale > 0
                row_max = fmaxf(row_max, tile_max);
                // O is touched only when a reference of these 32 rows moved (also at the first visible key: -inf reference), and
                // only then does P wait for the previous P V into it.
                const bool moved = row_max > row_ref + kRescaleThreshold, moved_rows = __any_sync(0xFFFFFFFFu, moved);
                float corr = 1.0f;
                if (moved) {
                    corr = row_ref == -INFINITY ? 0.0f : fast_exp2(row_ref - row_max);
                    row_ref = row_max;
                }
                const float base = row_ref == -INFINITY ? 0.0f : row_ref;
                // Two weights an instruction where the two parts of fine weights and two warps a scheduler fill the issue slots
                // (16 verify runs of eight rows, 40/8 heads x 128: 73 us a layer, 76 one by one); one by one at head_dim 256 (a
                // power-limited step of long runs takes 0.9 % longer with pairs).
                [[maybe_unused]] const uint64_t scale2 = pack_f32x2(p.scale_log2, p.scale_log2), base2 = pack_f32x2(-base, -base);
                [[maybe_unused]] uint64_t sum2[2] = {0, 0};
                float sum4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int c0 = 0; c0 < int(kUmmaN); c0 += 32) {
                    uint32_t packed[16];
                    [[maybe_unused]] uint32_t low[16];
#pragma unroll
                    for (int c = 0; c < 32; c += 2) {
                        float e0, e1;
                        if constexpr (kStreams == 2) {
                            const float2 x = unpack_f32x2(fma_f32x2(pack_f32x2(s[c0 + c], s[c0 + c + 1]), scale2, base2));
                            e0 = fast_exp2(x.x);
                            e1 = fast_exp2(x.y);
                            sum2[c >> 1 & 1] = add_f32x2(sum2[c >> 1 & 1], pack_f32x2(e0, e1));
                        } else {
                            e0 = fast_exp2(fmaf(s[c0 + c], p.scale_log2, -base));
                            e1 = fast_exp2(fmaf(s[c0 + c + 1], p.scale_log2, -base));
                            sum4[c & 2] += e0;
                            sum4[(c & 2) + 1] += e1;
                        }
                        if constexpr (kFine) {
                            packed[c / 2] = Mma<T>::pack_down(e0, e1);
                            low[c / 2] = low_part<T>(e0, e1, packed[c / 2]);
                        } else {
                            packed[c / 2] = Mma<T>::pack(e0, e1);
                        }
                    }
                    // P over the first 32 columns of this S buffer, its low part over the rest
                    tmem_store16_bits(tmem_s + c0 / 2, packed);
                    if constexpr (kFine) tmem_store16_bits(tmem_s + kUmmaN / 2 + c0 / 2, low);
                }
                if constexpr (kStreams == 2) {
                    const float2 a = unpack_f32x2(sum2[0]), b = unpack_f32x2(sum2[1]);
                    sum4[0] = a.x;
                    sum4[1] = a.y;
                    sum4[2] = b.x;
                    sum4[3] = b.y;
                }
                row_sum = row_sum * corr + ((sum4[0] + sum4[1]) + (sum4[2] + sum4[3]));

                if (i >= kStreams && moved_rows) {
                    wait(v_done(tile - kStreams), slot_phase(tile - kStreams));
                    __syncwarp();
                    tc_fence_after();
#pragma unroll 1
                    for (uint32_t c = 0; c < uint32_t(D); c += 32) {
                        const uint32_t at = tmem_o + lane_base + c;
                        float o[32];
                        tmem_load32(at, o);
#pragma unroll
                        for (int e = 0; e < 32; ++e) o[e] *= corr;
                        tmem_store32(at, o);
                    }
                }
                tmem_store_wait();
                tc_fence_before();
                mbar_arrive(bar(kBarP + stream_barrier(tile)));
            }
            const bool is_partial = v.partial_slot != kU32Max;
            // The next item's query rows go to TMEM under this item's last P V, and the first Q K^T products of that item run
            // under the epilogue (O is not touched before P of that item's first tile exists).  Where both warps have tiles they
            // have seen their last S where they meet, so all Q K^T of the item are complete there.
            if (kStreams == 1 && half == 1 && more) {
                if (num_tiles > 0) row_pair_wait(rows_warp);
                tc_fence_after();
                first_q(next_row, next_rows);
            }
            const float whole_max = fmaxf(row_max, exchange(row_max));
            if (more) {
                if (kStreams == 2 || (half == 0 && num_tiles == 0)) first_q(next_row, next_rows);
                rest_of_q();
            }
            const bool staged_out = !is_partial && p.ext_o == nullptr, gated = staged_out && p.gates != nullptr;
            if (gated) {
#pragma unroll 1
                for (uint32_t b = 0; b < 2; ++b) {
                    stage_gates(static_cast<uint32_t>(out_row), v.rows, column0 + 32 * b, b);
                    cp_async_commit();
                }
            }
            {
                const uint32_t mine = kStreams == 2 ? (tile_base + num_tiles - 1 - half) & 1u : 0u;  // tiles behind this thread's last one
                if (end_tile > mine) {
                    const uint32_t last = tile_base + num_tiles - 1 - mine;
                    wait(v_done(last), slot_phase(last));
                }
                __syncwarp();
            }
            // Both threads of a row finish it, back at the true max as the reference: l' = l * 2^(ref - max); O / l is unchanged
            // by the shift.  With two streams O is the sum of their O_i * 2^(ref_i - max).  A stream takes no part where it saw no
            // key of the row, and only there: a weight that is no number (a score of +Inf) and the 0 x Inf of an infinity in V
            // under a weight that underflows go into the row as they do with one stream.
            // (The exchange also says that the other warp's last P V is complete.)
            constexpr float kNoKey = -1.0f;
            float sum_at_max, weights[2] = {1.0f, kNoKey};  // of the stream of the item's first tile, and of the other
            if constexpr (kStreams == 2) {
                const bool no_key = row_max == -INFINITY && row_sum == 0.0f;
                // (scores that are no numbers alone leave the maximum at -Inf)
                const float weight = no_key ? kNoKey : (row_max == -INFINITY ? 1.0f : fast_exp2(row_ref - whole_max));
                const float other = exchange(weight);
                if (!no_key) row_sum *= weight;
                row_sum += exchange(row_sum);
                sum_at_max = row_sum;
                const bool first = ((tile_base ^ half) & 1u) == 0;
                weights[0] = first ? weight : other;
                weights[1] = first ? other : weight;
            } else {
                row_sum += exchange(row_sum);  // (0 from the second warp)
                sum_at_max = whole_max == -INFINITY ? row_sum : row_sum * fast_exp2(row_ref - whole_max);
            }
            const uint32_t first_stream = kStreams == 2 ? tile_base & 1u : 0u;
            tile_base += num_tiles;
            look_ahead(index + 2);  // used by the next item, under whose tiles that item's query rows travel

            // ---- epilogue: every thread finishes its half of its row -------------------------------------------------------
            const float inv = row_sum > 0.0f ? 1.0f / (kFine ? row_sum * kFineScale : row_sum) : 0.0f;
            const uint64_t prow = is_partial ? static_cast<uint64_t>(v.partial_slot + w) * kMaxRows + rr : 0;
            // Sixteen columns a pass: a longer body does not stay in the instruction cache, which every warp walks once per item.
#pragma unroll 1
            for (uint32_t c = column0; c < column0 + kHalfD; c += 16) {
                float o[16];
                if (num_tiles > 0) {
                    tmem_load16(tmem + kColO + first_stream * D + lane_base + c, o);
                    if constexpr (kStreams == 2) {
#pragma unroll
                        for (int e = 0; e < 16; ++e) o[e] = weights[0] == kNoKey ? 0.0f : o[e] * weights[0];
                        if (num_tiles > 1) {
                            float other[16];
                            tmem_load16(tmem + kColO + (first_stream ^ 1u) * D + lane_base + c, other);
#pragma unroll
                            for (int e = 0; e < 16; ++e) o[e] = weights[1] == kNoKey ? o[e] : fmaf(other[e], weights[1], o[e]);
                        }
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < 16; ++e) o[e] = 0.0f;
                }
                if constexpr (kFine) {
                    if (row_valid && *reinterpret_cast<volatile uint32_t*>(&shared.cleaned[index & 1]) == index + 1) {
                        const uint32_t* row_ids = table_row(p.geo, v.req_slot);
                        for (uint32_t token = max(min_limit, v.kv_begin); token < limit; ++token) {
                            const uint64_t page = page_id_or_zero(p.geo, row_ids, token >> page_shift);
                            const T* src = reinterpret_cast<const T*>(pages + page * page_bytes + v_region_bytes) +
                                           (static_cast<uint64_t>(v.kv_head) * p.geo.tokens_per_page + (token & page_mask)) * D + c;
#pragma unroll
                            for (int e = 0; e < 16; ++e) {
                                const float value = static_cast<float>(src[e]);
                                if (!isfinite(value)) o[e] += value;
                            }
                        }
                    }
                }
#pragma unroll
                for (int e = 0; e < 16; ++e) o[e] *= inv;
                if (staged_out) {
                    const uint32_t buffer = (c - column0) / 32 & 1u, chunk0 = c / 8 & 2u;  // chunks chunk0 and chunk0 + 1 of the buffer's four
                    const uint32_t at0 = narrow_at(lane, chunk0, buffer), at1 = narrow_at(lane, chunk0 + 1, buffer);
                    if (gated) {
                        if (chunk0 == 0) {
                            cp_async_wait<1>();
                            __syncwarp();
                        }
                        const uint4 raw[2] = {ld_shared_16(at0), ld_shared_16(at1)};
                        const uint32_t two[8] = {raw[0].x, raw[0].y, raw[0].z, raw[0].w, raw[1].x, raw[1].y, raw[1].z, raw[1].w};
                        float factor[16];
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const float2 pair = Mma<T>::unpack(two[e]);
                            factor[2 * e] = pair.x;
                            factor[2 * e + 1] = pair.y;
                        }
                        gate_sigmoids<16>(factor);
#pragma unroll
                        for (int e = 0; e < 16; ++e) o[e] *= factor[e];
                    }
                    st_shared_16(at0, make_uint4(Mma<T>::pack(o[0], o[1]), Mma<T>::pack(o[2], o[3]), Mma<T>::pack(o[4], o[5]), Mma<T>::pack(o[6], o[7])));
                    st_shared_16(at1, make_uint4(Mma<T>::pack(o[8], o[9]), Mma<T>::pack(o[10], o[11]), Mma<T>::pack(o[12], o[13]), Mma<T>::pack(o[14], o[15])));
                    if (chunk0 != 0) {  // the buffer goes out, eight rows per access
                        __syncwarp();
#pragma unroll
                        for (uint32_t i = 0; i < 32; i += 8) {
                            const uint32_t r = i + (lane >> 2), chunk = lane & 3u;
                            const uint32_t row = __shfl_sync(0xFFFFFFFFu, static_cast<uint32_t>(out_row), r);
                            const uint4 value = ld_shared_16(narrow_at(r, chunk, buffer));
                            T* dst = static_cast<T*>(p.out) + static_cast<uint64_t>(row) * D + (c - 16) + chunk * 8;
                            if (rows_warp * 32 + r >= v.rows) continue;
                            if (wide_out) {
                                *reinterpret_cast<uint4*>(dst) = value;
                            } else {
                                reinterpret_cast<uint2*>(dst)[0] = make_uint2(value.x, value.y);
                                reinterpret_cast<uint2*>(dst)[1] = make_uint2(value.z, value.w);
                            }
                        }
                        __syncwarp();
                        if (gated) {
                            if (c + 48 < column0 + kHalfD) stage_gates(static_cast<uint32_t>(out_row), v.rows, c + 48, buffer);
                            cp_async_commit();
                        }
                    }
                } else if (row_valid) {
                    if (is_partial) {
                        // a partial slot of this kernel is stored column-major in float4 units, [D / 4][16 rows]: the
                        // 16 rows of a tile are 16 consecutive lanes here, so every store instruction writes whole
                        // 256-byte runs (the merge below reads them the same way)
                        float4* dst = reinterpret_cast<float4*>(p.partial_o + static_cast<uint64_t>(v.partial_slot + w) * kMaxRows * D) +
                                      static_cast<uint64_t>(c / 4) * kMaxRows + rr;
#pragma unroll
                        for (int e = 0; e < 16; e += 4)
                            dst[static_cast<uint64_t>(e / 4) * kMaxRows] = make_float4(o[e], o[e + 1], o[e + 2], o[e + 3]);
                    } else {
                        float* dst = p.ext_o + out_row * D + c;
#pragma unroll
                        for (int e = 0; e < 16; e += 4)
                            *reinterpret_cast<float4*>(dst + e) = make_float4(o[e], o[e + 1], o[e + 2], o[e + 3]);
                    }
                }
                __syncwarp();  // the TMEM load of the next pass is warp-collective
            }
            // Both warps have read these rows' accumulators before either goes on.  The next item's first P V overwrites an
            // accumulator as soon as four of the eight row warps have delivered its P (at head_dim 256 always the first four,
            // and the others read half of that one O), and its Q K^T may be complete already.
            tc_fence_before();
            row_pair_sync(rows_warp);
            if (row_valid && half == 0) {
                if (is_partial) {
                    p.partial_m[prow] = whole_max;
                    p.partial_l[prow] = sum_at_max;
                } else if (p.ext_o != nullptr) {
                    p.ext_m[out_row] = whole_max * kLn2;
                    p.ext_l[out_row] = sum_at_max;
                }
            }
            tc_fence_before();

            // ---- units shared with other CTAs: whoever delivers a tile's last partial merges it ---------------------------
            if (is_partial) {
                __threadfence();
                row_threads_sync();
                if (tid < 8) {
                    const bool has_rows = tid * kMaxRows < v.rows;
                    last_s[tid] = has_rows && atomicAdd(p.unit_counters + v.reduce_unit + tid, 1u) == v.unit_num_items - 1;
                    __threadfence();  // the other pieces' partials are read (from L2) only after their arrivals were seen
                }
                row_threads_sync();
                // Several tiles at a time, so that their loads share the round trips.  16 rows x D / 4 float4 outputs per tile: a thread
                // takes row tid % 16 and the float4 columns tid / 16 + 16 j (16 consecutive lanes read 256 consecutive bytes of
                // the column-major slots)
                constexpr uint32_t kAtOnce = 512 / D;
                for (uint32_t tile0 = 0; tile0 < 8; tile0 += kAtOnce) {
                    uint32_t some = 8;  // one that is to be merged
#pragma unroll
                    for (uint32_t k = 0; k < kAtOnce; ++k)
                        if (last_s[tile0 + k]) some = tile0 + k;
                    if (some == 8) continue;
                    constexpr uint32_t kPerThread = kMaxRows * (D / 4) / kRowThreads;
                    constexpr uint32_t kColumnStep = kRowThreads / kMaxRows;  // float4 columns between a thread's outputs
                    const uint32_t c4_0 = tid / kMaxRows;
                    // a row beyond the tile's last one is computed on the last row, a tile that is not to be merged on another
                    // one, and both are dropped at the end: the loops below are then straight-line code whose loads all go
                    // out before the first one is used
                    uint32_t r[kAtOnce];
                    bool present[kAtOnce];
                    uint64_t slot_rows[kAtOnce];
#pragma unroll
                    for (uint32_t k = 0; k < kAtOnce; ++k) {
                        const uint32_t tile = last_s[tile0 + k] ? tile0 + k : some;
                        const uint32_t tile_rows = min(kMaxRows, v.rows - tile * kMaxRows);
                        r[k] = min(tid % kMaxRows, tile_rows - 1);
                        present[k] = tile == tile0 + k && tid % kMaxRows < tile_rows;
                        slot_rows[k] = static_cast<uint64_t>(v.unit_first_slot + tile) * kMaxRows;
                    }
                    // one pass over the pieces with the running max of a row carried along (sums are rescaled when
                    // a later piece raises it); the loads of piece s + 1 are in flight while piece s is folded in
                    float4 acc[kAtOnce][kPerThread];
                    float top_all[kAtOnce], sum_all[kAtOnce];  // one row per thread and tile: a single running max and sum for its columns
#pragma unroll
                    for (uint32_t k = 0; k < kAtOnce; ++k) {
                        top_all[k] = -INFINITY;
                        sum_all[k] = 0.0f;
#pragma unroll
                        for (uint32_t j = 0; j < kPerThread; ++j) acc[k][j] = make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                    constexpr uint64_t kPieceRows = 8 * kMaxRows;  // rows between the same tile of consecutive pieces
                    struct Piece {
                        float m[kAtOnce], l[kAtOnce];
                        float4 o[kAtOnce][kPerThread];
                    } piece[2];
                    auto fetch = [&](uint32_t index, Piece& x) {
#pragma unroll
                        for (uint32_t k = 0; k < kAtOnce; ++k) {
                            const uint64_t rows = slot_rows[k] + index * kPieceRows;
                            x.m[k] = __ldcg(p.partial_m + rows + r[k]);
                            x.l[k] = __ldcg(p.partial_l + rows + r[k]);
                            const float4* slot = reinterpret_cast<const float4*>(p.partial_o + rows * D) + r[k];
#pragma unroll
                            for (uint32_t j = 0; j < kPerThread; ++j)
                                x.o[k][j] = __ldcg(slot + static_cast<uint64_t>(c4_0 + j * kColumnStep) * kMaxRows);
                        }
                    };
                    auto fold = [&](const Piece& x) {
#pragma unroll
                        for (uint32_t k = 0; k < kAtOnce; ++k) {
                            const float top = fmaxf(top_all[k], x.m[k]);
                            const float carry = top_all[k] == -INFINITY ? 0.0f : fast_exp2(top_all[k] - top);
                            const float w = x.m[k] == -INFINITY ? 0.0f : fast_exp2(x.m[k] - top) * x.l[k];
                            sum_all[k] = sum_all[k] * carry + w;
#pragma unroll
                            for (uint32_t j = 0; j < kPerThread; ++j) {
                                acc[k][j].x = acc[k][j].x * carry + w * x.o[k][j].x;
                                acc[k][j].y = acc[k][j].y * carry + w * x.o[k][j].y;
                                acc[k][j].z = acc[k][j].z * carry + w * x.o[k][j].z;
                                acc[k][j].w = acc[k][j].w * carry + w * x.o[k][j].w;
                            }
                            top_all[k] = top;
                        }
                    };
                    fetch(0, piece[0]);
                    for (uint32_t s0 = 0; s0 < v.unit_num_items; s0 += 2) {
                        if (s0 + 1 < v.unit_num_items) fetch(s0 + 1, piece[1]);
                        fold(piece[0]);
                        if (s0 + 1 < v.unit_num_items) {
                            if (s0 + 2 < v.unit_num_items) fetch(s0 + 2, piece[0]);
                            fold(piece[1]);
                        }
                    }
#pragma unroll
                    for (uint32_t k = 0; k < kAtOnce; ++k) {
                        if (!present[k]) continue;
                        const float scale = sum_all[k] > 0.0f ? 1.0f / sum_all[k] : 0.0f;
                        const uint64_t row = item_row_index(p, v, (tile0 + k) * kMaxRows + r[k]);
#pragma unroll
                        for (uint32_t j = 0; j < kPerThread; ++j) {
                            const uint32_t c4 = c4_0 + j * kColumnStep;
                            const float4 value =
                                make_float4(acc[k][j].x * scale, acc[k][j].y * scale, acc[k][j].z * scale, acc[k][j].w * scale);
                            if (p.ext_o != nullptr) {
                                *reinterpret_cast<float4*>(p.ext_o + row * D + 4 * c4) = value;
                            } else {
                                store_out4<T>(p, row * D + 4 * c4, value);
                            }
                        }
                        if (p.ext_o != nullptr && c4_0 == 0) {
                            p.ext_m[row] = top_all[k] * kLn2;
                            p.ext_l[row] = sum_all[k];
                        }
                    }
                    if (tid < kAtOnce && last_s[tile0 + tid]) p.unit_counters[v.reduce_unit + tile0 + tid] = 0;  // ready for the next launch
                }
                row_threads_sync();  // the flags are read before the next item overwrites them
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemColumns) : "memory");
    }
}

// kWeights: one of ChunkWeights.
template <typename T, int D, uint32_t kWeights>
__global__ void __launch_bounds__(kUmmaThreads<D>, 1)
    attend_chunk_umma_kernel(const AttendParams p, const __grid_constant__ CUtensorMap kv_map, const uint32_t box_rows) {
    __shared__ UmmaShared shared;
    const bool early = p.plan_ready != 0;  // the set-up runs before the wait for the inputs
    if (!early) await_previous_kernel();
    if (blockIdx.x >= p.scalars[kScalarNumChunkCtas]) {
        if (early) await_previous_kernel();
        return;
    }
    if constexpr (kWeights == kChunkWeightsByPlan) {
        if (p.scalars[kScalarFineChunks] != 0) attend_chunk_umma<T, D, true>(p, kv_map, box_rows, early, shared);
        else attend_chunk_umma<T, D, false>(p, kv_map, box_rows, early, shared);
    } else {
        attend_chunk_umma<T, D, kWeights == kChunkWeightsFine>(p, kv_map, box_rows, early, shared);
    }
}

template <typename T, int D, uint32_t kWeights>
cudaError_t launch_one(const AttendParams& p, uint32_t num_ctas, cudaStream_t stream) {
    constexpr uint32_t kSmem = kSlots * kSlotBytes + kRowThreads * kUmmaStageColumns * 2 + 1024;
    constexpr uint32_t kLargestBox = D == 128 ? kUmmaN / 2 : kUmmaN;
    const uint32_t box_rows = p.geo.tokens_per_page < kLargestBox ? p.geo.tokens_per_page : kLargestBox;
    CUtensorMap map;
    if (!(D == 128 ? make_kv_pair_map(p, box_rows, &map) : make_kv_map(p, box_rows, &map))) return cudaErrorNotSupported;
    auto kernel = attend_chunk_umma_kernel<T, D, kWeights>;
    static std::atomic<uint64_t> configured{0};  // per instantiation, one bit per device
    cudaError_t err = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), static_cast<int>(kSmem), configured);
    if (err != cudaSuccess) return err;
    return launch_overlapped(kernel, num_ctas, kUmmaThreads<D>, kSmem, stream, p, map, box_rows);
}

template <typename T, int D>
cudaError_t launch_for_weights(const AttendParams& p, uint32_t num_ctas, cudaStream_t stream) {
    switch (p.chunk_weights) {
        case kChunkWeightsPlain: return launch_one<T, D, kChunkWeightsPlain>(p, num_ctas, stream);
        case kChunkWeightsFine: return launch_one<T, D, kChunkWeightsFine>(p, num_ctas, stream);
        default: return launch_one<T, D, kChunkWeightsByPlan>(p, num_ctas, stream);
    }
}

template <typename T>
cudaError_t launch_for_dim(const AttendParams& p, uint32_t num_ctas, cudaStream_t stream) {
    switch (p.geo.head_dim) {
        case 128: return launch_for_weights<T, 128>(p, num_ctas, stream);
        case 256: return launch_for_weights<T, 256>(p, num_ctas, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

// cudaErrorNotSupported: the arena cannot be described to the TMA unit (alignment, size); nothing was launched and
// the caller takes launch_attend_chunk instead.

cudaError_t launch_attend_chunk_umma(const AttendParams& p, uint32_t num_ctas, cudaStream_t stream) {
    if (num_ctas == 0) return cudaSuccess;
    return p.dtype == PSI_DTYPE_BF16 ? launch_for_dim<__nv_bfloat16>(p, num_ctas, stream)
                                     : launch_for_dim<__half>(p, num_ctas, stream);
}

}  // namespace psi
