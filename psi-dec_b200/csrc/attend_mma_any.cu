// Split-KV flash-decode map kernel on the tensor cores for the 16-bit profiles attend_mma.cu does not take: head dims
// that are no multiple of 64 (any multiple of eight up to 256) and any page size.
//
// Same work items and partial slots as the CUDA-core kernels (attend_generic.cu), whose arithmetic it keeps: the weights stay f32.  Each is split into three 16-bit parts, and O += P V runs once per part; K, V and q are 16-bit values
// already and all accumulators are f32.  In bf16, which has f32's exponents, the parts add up to the weight exactly.  f16
// ends at steps of 2^-24, so there the weights are taken 2^15 times as large (kWeightShift): exact down to 2^-16 of the
// heaviest key of the warp, and within 2^-40 of it below that, where f32 sums over an item do not see it.  Bound by HBM; the
// tensor pipe has room for the two extra products.  One CTA of eight warps per SM (sixteen for long items up to head_dim 96,
// kLongItemTiles), every warp owning every eighth (sixteenth) 16-token tile of the item and a ring of its own (K tile, V tile,
// K tile, ...) fed by 16-byte cp.async, the next tile's page looked up one tile ahead.  Rows are padded to DP elements plus one 16-byte chunk: an odd number of chunks per row keeps ldmatrix free
// of bank conflicts without a swizzle, and the chunks beyond head_dim hold zeros.
// Units cut into a few pieces are merged by the CTA that delivers the last partial, the others by the reduce launch
// (merges_in_launch), and each warp's first two tiles are requested into the L2 while the append runs.  Measured: 24 requests of 300 to 6,000 tokens, 24/8 heads x 96, pages of 12 (233 MB): 72.7 us a
// step with the append = 3.2 TB/s; 74.2 with eight warps and eight slots each, 79 against 75.7 with twelve and five, 75.0 with
// the reduce as a launch of its own, 466 on the staged kernel.
#include <atomic>

#include "launch_util.hpp"
#include "mma_common.cuh"
#include "unit_merge.cuh"

namespace psi {

namespace {

template <int DP, int NSLOT, int kWarps>
struct AnySmem {
    static constexpr uint32_t kStride = DP * 2 + 16;
    static constexpr uint32_t kTileBytes = kTile * kStride;
    static constexpr uint32_t kRingOffset = kTileBytes;  // the query tile comes first
    static constexpr uint32_t kMergeStride = DP + 8;     // floats per merged row
    static constexpr uint32_t kMergeBytes = kWarps * kTile * kMergeStride * 4;
    static constexpr uint32_t kRingBytes = kWarps * NSLOT * kTileBytes;
    static constexpr uint32_t kTotal = kRingOffset + (kRingBytes > kMergeBytes ? kRingBytes : kMergeBytes);
};

// Two f32 weights as three packed 16-bit parts, each the rounded rest of the ones before it.
template <typename T>
__device__ __forceinline__ void split3(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    hi = Mma<T>::pack(a, b);
    const float2 h = Mma<T>::unpack(hi);
    a -= h.x;
    b -= h.y;
    mid = Mma<T>::pack(a, b);
    const float2 m = Mma<T>::unpack(mid);
    lo = Mma<T>::pack(a - m.x, b - m.y);
}

// Exponent by which the weights (at most 1, the running maximum) are raised: 2^15 is the largest power of two in f16.  The
// row sum is of the raised weights too and is brought back when the item's warps meet; O / l does not change.
template <typename T>
constexpr float kWeightShift = 0.0f;
template <>
constexpr float kWeightShift<__half> = 15.0f;

// Stores those of four consecutive results that are infinite.
template <typename T>
__device__ __forceinline__ void write_infinities(const AttendParams& p, const ItemView& v, uint32_t r, uint32_t d, float4 value) {
    const float x[4] = {value.x, value.y, value.z, value.w};
#pragma unroll
    for (uint32_t e = 0; e < 4; ++e) {
        if (!isinf(x[e])) continue;
        if (v.partial_slot != kU32Max) {
            p.partial_o[(static_cast<uint64_t>(v.partial_slot) * kMaxRows + r) * p.geo.head_dim + d + e] = x[e];
            continue;
        }
        const uint64_t at = item_row_index(p, v, r) * p.geo.head_dim + d + e;
        if (p.ext_o != nullptr) p.ext_o[at] = x[e];
        else store_from_float(p.out, at, p.dtype, x[e] * gate_factor(p, at));
    }
}

__device__ __forceinline__ void st_shared_zero_16(uint32_t dst) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};\n" ::"r"(dst), "r"(0u) : "memory");
}

// 16 bytes from a source on a 2-byte boundary into shared memory.
__device__ __forceinline__ void copy_16_by_elements(uint32_t dst, const void* src, bool present) {
    uint32_t w[4] = {0, 0, 0, 0};
    if (present) {
        const uint16_t* e = static_cast<const uint16_t*>(src);
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = e[2 * i] | static_cast<uint32_t>(e[2 * i + 1]) << 16;
    }
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};\n" ::"r"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
}

// kAligned: the arena lies on a 16-byte boundary.  Off it, and for a q off it, elements are copied one by one: slower than
// cp.async, but the plan is one CTA per SM for this kernel whatever the buffers of a launch, and the CUDA-core kernels
// on such a plan took 1,037 us with an odd q for the step above (541 on a plan of their own; 85 here).
template <typename T, int DP, int NSLOT, int kWarps, bool kAligned>
__global__ void __launch_bounds__(kWarps * 32, 1) attend_mma_any_kernel(AttendParams p) {
    using L = AnySmem<DP, NSLOT, kWarps>;
    constexpr int kThreads = kWarps * 32;
    const uint32_t cta = blockIdx.x;
    // plan and page table are read before the wait for the inputs
    const bool early = p.plan_ready != 0 && p.geo.table_settled != 0;
    if (!early) await_previous_kernel();
    uint32_t item_begin = 0, item_end = 0;
    if (cta < p.scalars[kScalarNumCtas]) {
        item_begin = p.cta_item_begin[cta];
        item_end = p.cta_item_begin[cta + 1];
    }
    if (item_begin >= item_end) {
        if (early) await_previous_kernel();
        return;
    }
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint32_t limit_s[kTile];
    __shared__ float merge_m[kWarps][kTile], merge_l[kWarps][kTile];
    __shared__ uint32_t arrival_s;

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t D = p.geo.head_dim, chunks = D / 8;
    const uint32_t q_base = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    const uint32_t ring_base = q_base + L::kRingOffset + warp * NSLOT * L::kTileBytes;
    float* merge_o = reinterpret_cast<float*>(smem + L::kRingOffset);
    const unsigned char* arena = static_cast<const unsigned char*>(p.geo.pages);
    const uint64_t v_bytes = v_region_offset(p.geo) * 2;
    const uint64_t stream_policy = l2_evict_first_policy();

    // lane roles of the ldmatrix fetches (as in FragmentLanes, rows padded instead of swizzled)
    const uint32_t mat = lane >> 3, mat_row = lane & 7, quad_row = lane >> 2, quad_col = lane & 3;
    const uint32_t q_lane = q_base + (mat_row + 8 * (mat & 1)) * L::kStride + (mat >> 1) * 16;
    const uint32_t k_lane = (mat_row + 8 * (mat >> 1)) * L::kStride + (mat & 1) * 16;
    const uint32_t v_lane = (mat_row + 8 * (mat & 1)) * L::kStride + (mat >> 1) * 16;
    // copy roles: a warp copies two rows at a time while a row has at most 16 chunks, else one
    constexpr uint32_t kRowsPerCopy = DP <= 128 ? 2 : 1;
    const uint32_t copy_row = kRowsPerCopy == 2 ? lane >> 4 : 0, copy_chunk = kRowsPerCopy == 2 ? lane & 15 : lane;

    // An infinity in V meets parts that are zero or negative, and 0 x Inf or Inf - Inf is no number where the weight itself
    // would have kept the infinity.  An item that ends in anything but finite values is therefore done once more with the
    // high parts alone, which have the weight's sign, and its infinities are written over what the first pass left.
    bool again = false;
    const bool wide_q = (reinterpret_cast<uintptr_t>(p.q) & 15u) == 0, wide_out = (reinterpret_cast<uintptr_t>(p.out) & 7u) == 0;
    // columns [d, d + 4) of a finished row
    auto store_row = [&](const ItemView& v, uint32_t r, uint32_t d, float4 value, float top, float sum) {
        const uint64_t row = item_row_index(p, v, r);
        if (p.ext_o != nullptr) {
            *reinterpret_cast<float4*>(p.ext_o + row * D + d) = value;
            if (d == 0) {
                p.ext_m[row] = top * kLn2;
                p.ext_l[row] = sum;
            }
        } else if (wide_out) {
            store_out4<T>(p, row * D + d, value);
        } else {
            const float x[4] = {value.x, value.y, value.z, value.w};
#pragma unroll
            for (uint32_t e = 0; e < 4; ++e) store_from_float(p.out, row * D + d + e, p.dtype, x[e] * gate_factor(p, row * D + d + e));
        }
    };
    bool prefetched = !early;
    for (uint32_t index = item_begin; index < item_end;) {
        const ItemView v = view_item(p, index);
        // (the previous item's merge is done with the ring, q and limit_s: the barrier at the end of this loop)
        bool not_finite = false;
        const uint32_t* row_ids = table_row(p.geo, v.req_slot);
        const uint32_t first_tile = v.kv_begin / kTile;
        const uint32_t item_tiles = (v.kv_end + kTile - 1) / kTile - first_tile;
        const uint32_t my_tiles = item_tiles > warp ? (item_tiles - warp + kWarps - 1) / kWarps : 0;
        const uint32_t my_halves = 2 * my_tiles;
        auto token_of = [&](uint32_t j) { return (first_tile + warp + j * kWarps) * kTile; };
        // byte offset of the K row of token `lane & 15` of local tile j (beyond the range: the last row, which is not read)
        auto lookup = [&](uint32_t j) {
            const uint32_t at = min(token_of(j) + (lane & 15u), v.kv_end - 1);
            const uint32_t page_id = page_id_or_zero(p.geo, row_ids, at / p.geo.tokens_per_page);
            return kv_row_offset(p.geo, page_id, v.kv_head, at % p.geo.tokens_per_page) * 2;
        };
        auto issue = [&](uint32_t h, uint32_t slot, uint64_t offset) {
            const uint32_t in_range = v.kv_end - token_of(h >> 1);
            const uint32_t dst = ring_base + slot * L::kTileBytes + copy_row * L::kStride + copy_chunk * 16;
            if (h & 1) offset += v_bytes;
#pragma unroll
            for (uint32_t r = 0; r < uint32_t(kTile); r += kRowsPerCopy) {
                const unsigned char* src = arena + __shfl_sync(0xFFFFFFFFu, offset, r + copy_row) + copy_chunk * 16;
                if (copy_chunk < chunks) {  // rows beyond the item are zero
                    if constexpr (kAligned) cp_async_16_hinted(dst + r * L::kStride, src, r + copy_row < in_range ? 16u : 0u, stream_policy);
                    else copy_16_by_elements(dst + r * L::kStride, src, r + copy_row < in_range);
                }
            }
        };

        uint64_t cur = 0, next = 0;
        if (my_tiles > 0) cur = lookup(0);
        if (my_tiles > 1) next = lookup(1);
        if (!prefetched) {
            // While the previous kernel finishes, each warp's first two tiles go into the L2: a lane takes the K or V rows of a
            // token of each.
            prefetched = true;
#pragma unroll
            for (uint32_t t = 0; t < 2; ++t) {
                const uint32_t at = token_of(t) + (lane & 15u);
                if (t < my_tiles && at < v.kv_end) {
                    const unsigned char* row = arena + (t == 0 ? cur : next) + (lane & 16u ? v_bytes : 0);
                    for (uint32_t b = 0; b < D * 2; b += 128) prefetch_l2(row + b);
                    prefetch_l2(row + D * 2 - 1);
                }
            }
            await_previous_kernel();
        }

        // query rows (zero beyond the item's) and the zero chunks beyond head_dim of the query tile and of this warp's ring
        // (the merge of the previous item wrote over them)
        for (uint32_t i = tid; i < kTile * (DP / 8); i += kThreads) {
            const uint32_t r = i / (DP / 8), c = i % (DP / 8);
            const bool present = r < v.rows && c < chunks;
            const T* src = static_cast<const T*>(p.q) + (present ? item_row_index(p, v, r) * D + c * 8 : 0);
            if (wide_q) cp_async_16(q_base + r * L::kStride + c * 16, src, present ? 16u : 0u);
            else copy_16_by_elements(q_base + r * L::kStride + c * 16, src, present);
        }
        if (chunks < DP / 8) {
            const uint32_t pad = DP / 8 - chunks;
            for (uint32_t i = lane; i < NSLOT * kTile * pad; i += 32)
                st_shared_zero_16(ring_base + (i / pad) * L::kStride + (chunks + i % pad) * 16);
        }
        if (tid < kTile) limit_s[tid] = tid < v.rows ? item_row_limit(v, tid) : v.kv_end;
        cp_async_commit();

#pragma unroll
        for (uint32_t h = 0; h < NSLOT - 1; ++h) {
            if (h < my_halves) {
                issue(h, h, cur);
                if (h & 1) {
                    cur = next;
                    if ((h >> 1) + 2 < my_tiles) next = lookup((h >> 1) + 2);
                }
            }
            cp_async_commit();
        }
        cp_async_wait<NSLOT - 1>();  // the query rows and the padding (the oldest group) have landed
        __syncthreads();
        const uint32_t limit0 = limit_s[quad_row], limit1 = limit_s[quad_row + 8];
        uint32_t limit_min = v.kv_end;
        for (uint32_t r = 0; r < v.rows; ++r) limit_min = min(limit_min, limit_s[r]);

        RowState<DP> st;
        st.clear();
        uint32_t pa[3][4];
        for (uint32_t h = 0; h < my_halves; ++h) {
            cp_async_wait<NSLOT - 2>();
            __syncwarp();
            const uint32_t ahead = h + NSLOT - 1;
            if (ahead < my_halves) {
                issue(ahead, ahead % NSLOT, cur);
                if (ahead & 1) {
                    cur = next;
                    if ((ahead >> 1) + 2 < my_tiles) next = lookup((ahead >> 1) + 2);
                }
            }
            cp_async_commit();
            const uint32_t tile = ring_base + (h % NSLOT) * L::kTileBytes;
            if ((h & 1) == 0) {
                const uint32_t token0 = token_of(h >> 1);
                float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
                float s_odd[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
                for (int ks = 0; ks < DP / 16; ++ks) {
                    uint32_t a[4], b[4];
                    ldmatrix_x4(a, q_lane + 32 * ks);
                    ldmatrix_x4(b, tile + k_lane + 32 * ks);
                    Mma<T>::run(ks & 1 ? s_odd[0] : s[0], a, b[0], b[1]);
                    Mma<T>::run(ks & 1 ? s_odd[1] : s[1], a, b[2], b[3]);
                }
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) s[n][e] = (s[n][e] + s_odd[n][e]) * p.scale_log2;
                if (token0 < v.kv_begin || token0 + kTile > limit_min) {
#pragma unroll
                    for (int n = 0; n < 2; ++n)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const uint32_t token = token0 + 8 * n + 2 * quad_col + (e & 1);
                            if (token >= (e < 2 ? limit0 : limit1) || token < v.kv_begin) s[n][e] = -INFINITY;
                        }
                }
                float top[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    top[i] = fmaxf(fmaxf(s[0][2 * i], s[0][2 * i + 1]), fmaxf(s[1][2 * i], s[1][2 * i + 1]));
                    top[i] = fmaxf(top[i], __shfl_xor_sync(0xFFFFFFFFu, top[i], 1));
                    top[i] = fmaxf(top[i], __shfl_xor_sync(0xFFFFFFFFu, top[i], 2));
                }
                const float new0 = fmaxf(st.m0, top[0]), new1 = fmaxf(st.m1, top[1]);
                if (__any_sync(0xFFFFFFFFu, new0 > st.m0 || new1 > st.m1)) {
                    const float corr0 = new0 == -INFINITY ? 1.0f : exp2f(st.m0 - new0);
                    const float corr1 = new1 == -INFINITY ? 1.0f : exp2f(st.m1 - new1);
                    st.l0 *= corr0;
                    st.l1 *= corr1;
#pragma unroll
                    for (int j = 0; j < DP / 8; ++j) {
                        st.o[j][0] *= corr0;
                        st.o[j][1] *= corr0;
                        st.o[j][2] *= corr1;
                        st.o[j][3] *= corr1;
                    }
                    st.m0 = new0;
                    st.m1 = new1;
                }
                const float base0 = (st.m0 == -INFINITY ? 0.0f : st.m0) - kWeightShift<T>, base1 = (st.m1 == -INFINITY ? 0.0f : st.m1) - kWeightShift<T>;
                float w[2][4];
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) w[n][e] = exp2f(s[n][e] - (e < 2 ? base0 : base1));
                st.l0 += (w[0][0] + w[0][1]) + (w[1][0] + w[1][1]);
                st.l1 += (w[0][2] + w[0][3]) + (w[1][2] + w[1][3]);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    split3<T>(w[i >> 1][2 * (i & 1)], w[i >> 1][2 * (i & 1) + 1], pa[0][i], pa[1][i], pa[2][i]);
            } else if (!again) {
#pragma unroll
                for (int j = 0; j < DP / 16; ++j) {
                    uint32_t b[4];
                    ldmatrix_x4_trans(b, tile + v_lane + 32 * j);
#pragma unroll
                    for (int part = 2; part >= 0; --part) {  // the smallest first
                        Mma<T>::run(st.o[2 * j], pa[part], b[0], b[1]);
                        Mma<T>::run(st.o[2 * j + 1], pa[part], b[2], b[3]);
                    }
                }
            } else {
#pragma unroll
                for (int j = 0; j < DP / 16; ++j) {
                    uint32_t b[4];
                    ldmatrix_x4_trans(b, tile + v_lane + 32 * j);
                    Mma<T>::run(st.o[2 * j], pa[0], b[0], b[1]);
                    Mma<T>::run(st.o[2 * j + 1], pa[0], b[2], b[3]);
                }
            }
        }

        // ---- merge the warps' partial results ----------------------------------------------------------------------------
        cp_async_wait<0>();
        __syncthreads();  // every warp is done with its ring
        st.l0 += __shfl_xor_sync(0xFFFFFFFFu, st.l0, 1);
        st.l0 += __shfl_xor_sync(0xFFFFFFFFu, st.l0, 2);
        st.l1 += __shfl_xor_sync(0xFFFFFFFFu, st.l1, 1);
        st.l1 += __shfl_xor_sync(0xFFFFFFFFu, st.l1, 2);
        constexpr float kBack = 1.0f / static_cast<float>(1u << static_cast<uint32_t>(kWeightShift<T>));
        st.l0 *= kBack;
        st.l1 *= kBack;
        if (quad_col == 0) {
            merge_m[warp][quad_row] = st.m0;
            merge_m[warp][quad_row + 8] = st.m1;
            merge_l[warp][quad_row] = st.l0;
            merge_l[warp][quad_row + 8] = st.l1;
        }
        float* mine = merge_o + warp * kTile * L::kMergeStride + 2 * quad_col;
#pragma unroll
        for (int j = 0; j < DP / 8; ++j) {
            *reinterpret_cast<float2*>(mine + quad_row * L::kMergeStride + 8 * j) = make_float2(st.o[j][0] * kBack, st.o[j][1] * kBack);
            *reinterpret_cast<float2*>(mine + (quad_row + 8) * L::kMergeStride + 8 * j) = make_float2(st.o[j][2] * kBack, st.o[j][3] * kBack);
        }
        __syncthreads();
        const uint32_t c4_count = D / 4;
        for (uint32_t i = tid; i < v.rows * c4_count; i += kThreads) {
            const uint32_t r = i / c4_count, d = 4 * (i % c4_count);
            float top = -INFINITY;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) top = fmaxf(top, merge_m[w][r]);
            float sum = 0.0f;
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
                const float weight = merge_m[w][r] == -INFINITY ? 0.0f : exp2f(merge_m[w][r] - top);
                const float4 part = *reinterpret_cast<const float4*>(merge_o + (w * kTile + r) * L::kMergeStride + d);
                sum += weight * merge_l[w][r];
                acc.x += weight * part.x;
                acc.y += weight * part.y;
                acc.z += weight * part.z;
                acc.w += weight * part.w;
            }
            const float inv = sum > 0.0f ? 1.0f / sum : 0.0f;
            const float4 value = make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
            not_finite = not_finite || !(isfinite(acc.x) && isfinite(acc.y) && isfinite(acc.z) && isfinite(acc.w));
            if (again) {
                write_infinities<T>(p, v, r, d, value);
                continue;
            }
            if (v.partial_slot != kU32Max) {
                const uint64_t prow = static_cast<uint64_t>(v.partial_slot) * kMaxRows + r;
                *reinterpret_cast<float4*>(p.partial_o + prow * D + d) = value;
                if (d == 0) {
                    p.partial_m[prow] = top;
                    p.partial_l[prow] = sum;
                }
                continue;
            }
            store_row(v, r, d, value, top, sum);
        }
        again = __syncthreads_or(not_finite && !again);
        if (again) continue;
        if (p.merges != 0 && v.partial_slot != kU32Max && delivers_last_partial(p, v, arrival_s)) {
            merge_unit<kThreads>(p, v, [&](uint32_t r, uint32_t d, float4 value, float top, float sum) { store_row(v, r, d, value, top, sum); });
        }
        ++index;
    }
}

template <typename T, int DP, int NSLOT, int kWarps, bool kAligned>
cudaError_t launch_any(const AttendParams& p, uint32_t num_ctas, cudaStream_t stream) {
    auto kernel = attend_mma_any_kernel<T, DP, NSLOT, kWarps, kAligned>;
    constexpr int kBytes = AnySmem<DP, NSLOT, kWarps>::kTotal;
    static_assert(kBytes <= 220 * 1024, "query tile and ring share one CTA's shared memory");
    static std::atomic<uint64_t> configured{0};
    cudaError_t err = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), kBytes, configured);
    if (err != cudaSuccess) return err;
    return launch_overlapped(kernel, num_ctas, kWarps * 32, kBytes, stream, p);
}

// A tile is a chain of latencies, and two warps a scheduler leave 68 % of the issue slots empty; short items have no tiles for
// more.  40 requests, 24/8 heads x 96, pages of 12, four layers: 227 us with sixteen warps and 242 with eight at 1,600 tokens each,
// 165 both at 800, 124 and 120 at 400.  (Above 96 the accumulators leave registers for eight warps.)
// A CTA of many short items beside long ones ends last: 24 requests of 300 to 6,000 tokens, more short than long ones, 194 us with
// sixteen and 189 with eight (16 to 20 tiles an item in that CTA); 40 of 100 to 10,000 301 and 295 (10); as many short as long
// ones, 251 and 256 (24); 80-wide heads, 24 of 400 to 12,000, 270 and 285 (27).
constexpr uint32_t kLongItemTiles = 64, kLeastItemTiles = 20;

template <typename T, bool kAligned>
cudaError_t launch_for_dim(const AttendParams& p, uint32_t num_ctas, cudaStream_t stream) {
    const uint32_t d = p.geo.head_dim;
    if (p.item_tiles >= kLongItemTiles && p.least_item_tiles >= kLeastItemTiles) {
        if (d <= 64) return launch_any<T, 64, 5, 16, kAligned>(p, num_ctas, stream);
        if (d <= 96) return launch_any<T, 96, 4, 16, kAligned>(p, num_ctas, stream);
    }
    if (d <= 64) return launch_any<T, 64, 8, 8, kAligned>(p, num_ctas, stream);
    if (d <= 96) return launch_any<T, 96, 8, 8, kAligned>(p, num_ctas, stream);
    if (d <= 128) return launch_any<T, 128, 6, 8, kAligned>(p, num_ctas, stream);
    if (d <= 192) return launch_any<T, 192, 4, 8, kAligned>(p, num_ctas, stream);
    return launch_any<T, 256, 3, 8, kAligned>(p, num_ctas, stream);
}

template <typename T>
cudaError_t launch_for_arena(const AttendParams& p, uint32_t num_ctas, cudaStream_t stream) {
    return (reinterpret_cast<uintptr_t>(p.geo.pages) & 15u) == 0 ? launch_for_dim<T, true>(p, num_ctas, stream)
                                                                 : launch_for_dim<T, false>(p, num_ctas, stream);
}

}  // namespace

bool attend_mma_any_profile(uint32_t dtype, uint32_t head_dim) {
    return (dtype == PSI_DTYPE_BF16 || dtype == PSI_DTYPE_F16) && head_dim >= 8 && head_dim <= 256 && head_dim % 8 == 0;
}

// (The entry points ask for gates on an 8-byte boundary and partial outputs on a 16-byte one.)
bool attend_mma_any_supported(const AttendParams& p) { return attend_mma_any_profile(p.dtype, p.geo.head_dim); }

cudaError_t launch_attend_mma_any(const AttendParams& p, uint32_t num_ctas, cudaStream_t stream) {
    return p.dtype == PSI_DTYPE_BF16 ? launch_for_arena<__nv_bfloat16>(p, num_ctas, stream)
                                     : launch_for_arena<__half>(p, num_ctas, stream);
}

}  // namespace psi
