// Split-KV flash-decode map kernel for f32 pages: CUDA cores fed from per-warp shared-memory rings.
//
// Same work items and partial slots as the other CUDA-core map kernels (attend_generic.cu); head_dim must be a multiple of 32.
// Bound by HBM: a K and a V row of 2 * 4 * D bytes feed at most 16 query rows, 2 to 8 flop/B, so f32 FMAs keep up as long as
// shared memory does.  One CTA of eight warps per SM (twelve for long items up to head_dim 128, kLongItemTiles); every warp owns
// every eighth (twelfth) 8-token tile of the item and streams it through a ring of its own (K tile, V tile, K tile, ...) by
// 16-byte cp.async, so there is no CTA-wide barrier between the start and the end of an item.  Per tile:
//   scores   lane = (token pair, eighth of the row): two tokens per lane halve the reads of q, which are the larger part
//            of the shared-memory traffic; eight lanes read 128 consecutive bytes, so no access has a bank conflict.  The
//            2 R partial sums are reduced and scattered over the eight lanes in one butterfly, which leaves R / 4 of the
//            R x 8 scores in every lane;
//   softmax  online, in the log2 domain, on those scores; O is rescaled only when a row's maximum moved;
//   values   lane = four (or two times four) columns of every row; the weights are read back as broadcasts.
// The row count is rounded up to 4, 8 or 16 per item, each with code of its own.  All arithmetic is f32.
// Units cut into a few pieces are merged by the CTA that delivers the last partial, the others by the reduce launch
// (merges_in_launch), and each warp's first two tiles are requested into the L2 while the append runs.  Measured: 16 requests of
// 4,096 to 12,288 tokens, 32/8 heads x 128 (1.07 GB), a whole step with the append 203 us = 5.3 TB/s; 224 with eight warps
// and six ring slots each and a reduce launch (map launch alone, with two warps a scheduler, 194 us; 172 with twelve and four
// slots, 178 with sixteen and three), 517 with the staged kernel, whose shared-memory traffic grows with every row.
#include <atomic>

#include "launch_util.hpp"
#include "mma_common.cuh"
#include "unit_merge.cuh"

namespace psi {

namespace {

constexpr uint32_t kF32Tile = 8;  // KV tokens per tile

// Shared memory: q [16][D] | weights [warp][16][8] | ring [warp][NSLOT][8][D], which the merge of the warps reuses as
// [warp][16][D].
__host__ __device__ constexpr uint32_t f32_ring_offset(uint32_t d, uint32_t warps) { return (kMaxRows * d + warps * kMaxRows * kF32Tile) * 4; }
__host__ __device__ constexpr uint32_t f32_smem_bytes(uint32_t d, uint32_t slots, uint32_t warps) {
    return f32_ring_offset(d, warps) + warps * (slots * kF32Tile > kMaxRows ? slots * kF32Tile : kMaxRows) * d * 4;
}

template <int W>
struct F32Shared {
    float m[W][kMaxRows];
    float l[W][kMaxRows];
    uint32_t limit[kMaxRows];
    uint32_t arrival;
};

// One warp's share of an item with at most R rows; leaves the warp's (O, m, l) in the merge area and `shared`.
// DG = float4 columns per lane (head_dim <= 128 DG).
template <int R, int DG, int NSLOT, int W>
__device__ __forceinline__ void f32_item(const AttendParams& p, const ItemView& v, unsigned char* smem, F32Shared<W>& shared) {
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t D = p.geo.head_dim, c4 = D / 4;
    const float* q_s = reinterpret_cast<const float*>(smem);
    float* weight_s = reinterpret_cast<float*>(smem) + kMaxRows * D + warp * (kMaxRows * kF32Tile);
    unsigned char* ring = smem + f32_ring_offset(D, W);
    const uint32_t tile_bytes = kF32Tile * D * 4;
    float* my_ring = reinterpret_cast<float*>(ring + warp * NSLOT * tile_bytes);
    const uint32_t my_ring_u32 = static_cast<uint32_t>(__cvta_generic_to_shared(my_ring));
    const float* arena = static_cast<const float*>(p.geo.pages);
    const uint32_t* row_ids = table_row(p.geo, v.req_slot);
    const uint64_t v_off = v_region_offset(p.geo);

    const uint32_t first_tile = v.kv_begin / kF32Tile;
    const uint32_t item_tiles = (v.kv_end + kF32Tile - 1) / kF32Tile - first_tile;
    const uint32_t my_tiles = item_tiles > warp ? (item_tiles - warp + W - 1) / W : 0;
    const uint32_t my_halves = 2 * my_tiles;
    auto token_of = [&](uint32_t j) { return (first_tile + warp + j * W) * kF32Tile; };
    // element offset of the K row of token `lane & 7` of local tile j (beyond the range: the last row, which is not read)
    auto lookup = [&](uint32_t j) {
        const uint32_t at = min(token_of(j) + (lane & 7u), v.kv_end - 1);
        const uint32_t page_id = page_id_or_zero(p.geo, row_ids, at / p.geo.tokens_per_page);
        return kv_row_offset(p.geo, page_id, v.kv_head, at % p.geo.tokens_per_page);
    };
    auto issue = [&](uint32_t h, uint32_t slot, uint64_t offset) {
        const uint32_t in_range = v.kv_end - token_of(h >> 1);
        const uint32_t dst = my_ring_u32 + slot * tile_bytes + lane * 16;
        if (h & 1) offset += v_off;
#pragma unroll
        for (uint32_t t = 0; t < kF32Tile; ++t) {
            const float* src = arena + __shfl_sync(0xFFFFFFFFu, offset, t) + lane * 4;
            const uint32_t bytes = t < in_range ? 16u : 0u;  // rows beyond the item are zero
#pragma unroll
            for (uint32_t g = 0; g < uint32_t(DG); ++g)
                if (lane + 32 * g < c4) cp_async_16(dst + t * D * 4 + g * 512, src + g * 128, bytes);
        }
    };

    uint64_t cur = 0, next = 0;
    if (my_tiles > 0) cur = lookup(0);
    if (my_tiles > 1) next = lookup(1);
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

    // lane roles: scores of tokens pair and pair + 4 over the chunks eighth, eighth + 8, ... of a row; afterwards the
    // scores of token `my_token` and rows my_row, my_row + 4, ...
    const uint32_t pair = lane >> 3, eighth = lane & 7u;
    const uint32_t my_token = pair + 4 * (eighth >> 2), my_row = eighth & 3u;
    uint32_t limit[R / 4];
    float m[R / 4], l[R / 4];
    float4 o[R][DG];
#pragma unroll
    for (int j = 0; j < R / 4; ++j) {
        limit[j] = shared.limit[my_row + 4 * j];
        m[j] = -INFINITY;
        l[j] = 0.0f;
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int g = 0; g < DG; ++g) o[r][g] = make_float4(0.f, 0.f, 0.f, 0.f);

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
        const float* tile = my_ring + (h % NSLOT) * (kF32Tile * D);
        if ((h & 1) == 0) {
            float s[2][R];
#pragma unroll
            for (int r = 0; r < R; ++r) s[0][r] = s[1][r] = 0.0f;
            const float* k0 = tile + pair * D + eighth * 4;
            const float* k1 = k0 + 4 * D;
            const float* q = q_s + eighth * 4;
#pragma unroll 2
            for (uint32_t d = 0; d < D; d += 32) {
                const float4 a = *reinterpret_cast<const float4*>(k0 + d), b = *reinterpret_cast<const float4*>(k1 + d);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float4 x = *reinterpret_cast<const float4*>(q + r * D + d);
                    s[0][r] += x.x * a.x;
                    s[1][r] += x.x * b.x;
                    s[0][r] += x.y * a.y;
                    s[1][r] += x.y * b.y;
                    s[0][r] += x.z * a.z;
                    s[1][r] += x.z * b.z;
                    s[0][r] += x.w * a.w;
                    s[1][r] += x.w * b.w;
                }
            }
            // reduce and scatter over the eight lanes of a token pair: bit 2 of the lane picks the token, bits 1 and 0
            // the row modulo four
            const bool hi2 = eighth & 4u, hi1 = eighth & 2u, hi0 = eighth & 1u;
            float a[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float keep = hi2 ? s[1][r] : s[0][r], send = hi2 ? s[0][r] : s[1][r];
                a[r] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, 4);
            }
            float dot[R / 4];
#pragma unroll
            for (int j = 0; j < R / 4; ++j) {
                float b[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float keep = hi1 ? a[4 * j + 2 + i] : a[4 * j + i], send = hi1 ? a[4 * j + i] : a[4 * j + 2 + i];
                    b[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, 2);
                }
                const float keep = hi0 ? b[1] : b[0], send = hi0 ? b[0] : b[1];
                dot[j] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, 1);
            }
            const uint32_t pos = token_of(h >> 1) + my_token;
            float x[R / 4], m_new[R / 4];
            bool moved = false;
#pragma unroll
            for (int j = 0; j < R / 4; ++j) {
                x[j] = pos < limit[j] && pos >= v.kv_begin ? dot[j] * p.scale_log2 : -INFINITY;
                float top = fmaxf(x[j], __shfl_xor_sync(0xFFFFFFFFu, x[j], 4));
                top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, 8));
                top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, 16));
                m_new[j] = fmaxf(m[j], top);
                moved = moved || m_new[j] > m[j];
            }
            if (__any_sync(0xFFFFFFFFu, moved)) {
                float corr[R / 4];
#pragma unroll
                for (int j = 0; j < R / 4; ++j) {
                    corr[j] = m_new[j] == -INFINITY ? 1.0f : exp2f(m[j] - m_new[j]);
                    l[j] *= corr[j];
                    m[j] = m_new[j];
                }
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float c = __shfl_sync(0xFFFFFFFFu, corr[r / 4], r % 4);
#pragma unroll
                    for (int g = 0; g < DG; ++g) {
                        o[r][g].x *= c;
                        o[r][g].y *= c;
                        o[r][g].z *= c;
                        o[r][g].w *= c;
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < R / 4; ++j) {
                const float w = x[j] == -INFINITY ? 0.0f : exp2f(x[j] - m[j]);
                l[j] += w;  // this lane's token only; the tokens are summed once at the end
                weight_s[(my_row + 4 * j) * kF32Tile + my_token] = w;
            }
            __syncwarp();
        } else {
#pragma unroll
            for (uint32_t t = 0; t < kF32Tile; t += 4) {
                float4 value[4][DG];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int g = 0; g < DG; ++g)
                        value[i][g] = lane + 32 * g < c4 ? *reinterpret_cast<const float4*>(tile + (t + i) * D + lane * 4 + g * 128)
                                                         : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float4 w = *reinterpret_cast<const float4*>(weight_s + r * kF32Tile + t);
#pragma unroll
                    for (int g = 0; g < DG; ++g) {
                        float4& acc = o[r][g];
                        acc.x += w.x * value[0][g].x;
                        acc.y += w.x * value[0][g].y;
                        acc.z += w.x * value[0][g].z;
                        acc.w += w.x * value[0][g].w;
                        acc.x += w.y * value[1][g].x;
                        acc.y += w.y * value[1][g].y;
                        acc.z += w.y * value[1][g].z;
                        acc.w += w.y * value[1][g].w;
                        acc.x += w.z * value[2][g].x;
                        acc.y += w.z * value[2][g].y;
                        acc.z += w.z * value[2][g].z;
                        acc.w += w.z * value[2][g].w;
                        acc.x += w.w * value[3][g].x;
                        acc.y += w.w * value[3][g].y;
                        acc.z += w.w * value[3][g].z;
                        acc.w += w.w * value[3][g].w;
                    }
                }
            }
            __syncwarp();  // the weights may be overwritten
        }
    }
    cp_async_wait<0>();
    __syncthreads();  // every warp is done with its ring: the merge area may overwrite it
    float* mine = reinterpret_cast<float*>(ring) + warp * kMaxRows * D;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int g = 0; g < DG; ++g)
            if (lane + 32 * g < c4) *reinterpret_cast<float4*>(mine + r * D + lane * 4 + g * 128) = o[r][g];
#pragma unroll
    for (int j = 0; j < R / 4; ++j) {
        l[j] += __shfl_xor_sync(0xFFFFFFFFu, l[j], 4);
        l[j] += __shfl_xor_sync(0xFFFFFFFFu, l[j], 8);
        l[j] += __shfl_xor_sync(0xFFFFFFFFu, l[j], 16);
        if (lane < 4) {
            shared.m[warp][my_row + 4 * j] = m[j];
            shared.l[warp][my_row + 4 * j] = l[j];
        }
    }
}

template <int DG, int NSLOT, int W>
__global__ void __launch_bounds__(W * 32, 1) attend_f32_kernel(AttendParams p) {
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
    extern __shared__ __align__(128) unsigned char f32_smem[];
    __shared__ F32Shared<W> shared;
    const uint32_t tid = threadIdx.x, D = p.geo.head_dim, c4 = D / 4;
    const uint32_t q_base = static_cast<uint32_t>(__cvta_generic_to_shared(f32_smem));

    // columns [d, d + 4) of a finished row
    auto store_row = [&](const ItemView& v, uint32_t r, uint32_t d, float4 value, float top, float sum) {
        const uint64_t row = item_row_index(p, v, r), at = row * D + d;
        if (p.ext_o != nullptr) {
            *reinterpret_cast<float4*>(p.ext_o + at) = value;
            if (d == 0) {
                p.ext_m[row] = top * kLn2;
                p.ext_l[row] = sum;
            }
            return;
        }
        float* out = static_cast<float*>(p.out) + at;
        out[0] = value.x * gate_factor(p, at);
        out[1] = value.y * gate_factor(p, at + 1);
        out[2] = value.z * gate_factor(p, at + 2);
        out[3] = value.w * gate_factor(p, at + 3);
    };
    for (uint32_t index = item_begin; index < item_end; ++index) {
        const ItemView v = view_item(p, index);
        if (early && index == item_begin) {
            // While the previous kernel finishes, each warp's first two tiles go into the L2: a lane takes the K or V row of one token.
            const uint32_t lane = tid & 31u, tile = v.kv_begin / kF32Tile + (tid >> 5) + (lane >> 4) * W;
            const uint32_t at = tile * kF32Tile + (lane & 7u);
            if (at < v.kv_end) {
                const uint32_t page_id = page_id_or_zero(p.geo, table_row(p.geo, v.req_slot), at / p.geo.tokens_per_page);
                const float* row = static_cast<const float*>(p.geo.pages) +
                                   kv_row_offset(p.geo, page_id, v.kv_head, at % p.geo.tokens_per_page) + (lane & 8u ? v_region_offset(p.geo) : 0);
                for (uint32_t d = 0; d < D; d += 32) prefetch_l2(row + d);
            }
            await_previous_kernel();
        }
        __syncthreads();  // the previous item's merge is done with the ring and the statistics
        for (uint32_t i = tid; i < kMaxRows * c4; i += W * 32) {  // query rows, zero beyond the item's
            const uint32_t r = i / c4, c = i % c4;
            const bool present = r < v.rows;
            const float* src = static_cast<const float*>(p.q) + (present ? item_row_index(p, v, r) * D + 4 * c : 0);
            cp_async_16(q_base + i * 16, src, present ? 16u : 0u);
        }
        if (tid < kMaxRows) shared.limit[tid] = tid < v.rows ? item_row_limit(v, tid) : 0u;
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        if (v.rows <= 4) f32_item<4, DG, NSLOT, W>(p, v, f32_smem, shared);
        else if (v.rows <= 8) f32_item<8, DG, NSLOT, W>(p, v, f32_smem, shared);
        else f32_item<16, DG, NSLOT, W>(p, v, f32_smem, shared);
        __syncthreads();

        const float* merge = reinterpret_cast<const float*>(f32_smem + f32_ring_offset(D, W));
        for (uint32_t i = tid; i < v.rows * c4; i += W * 32) {
            const uint32_t r = i / c4, d = 4 * (i % c4);
            float top = -INFINITY;
#pragma unroll
            for (int w = 0; w < W; ++w) top = fmaxf(top, shared.m[w][r]);
            float sum = 0.0f;
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int w = 0; w < W; ++w) {
                const float weight = shared.m[w][r] == -INFINITY ? 0.0f : exp2f(shared.m[w][r] - top);
                const float4 part = *reinterpret_cast<const float4*>(merge + (w * kMaxRows + r) * D + d);
                sum += weight * shared.l[w][r];
                acc.x += weight * part.x;
                acc.y += weight * part.y;
                acc.z += weight * part.z;
                acc.w += weight * part.w;
            }
            const float inv = sum > 0.0f ? 1.0f / sum : 0.0f;
            const float4 value = make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
            if (v.partial_slot != kU32Max) {
                const uint64_t prow = static_cast<uint64_t>(v.partial_slot) * kMaxRows + r;
                *reinterpret_cast<float4*>(p.partial_o + prow * D + d) = value;
                if (d == 0) {
                    p.partial_m[prow] = top;
                    p.partial_l[prow] = sum;
                }
            } else {
                store_row(v, r, d, value, top, sum);
            }
        }
        if (p.merges != 0 && v.partial_slot != kU32Max && delivers_last_partial(p, v, shared.arrival)) {
            merge_unit<W * 32>(p, v, [&](uint32_t r, uint32_t d, float4 value, float top, float sum) { store_row(v, r, d, value, top, sum); });
        }
    }
}

// Two warps a scheduler leave half of the issue slots empty; short items have no tiles for more.  40 requests, 32/8 heads x 128,
// four layers: 406 us with twelve warps and 445 with eight at 1,600 tokens each, 179 and 184 at 400, 142 both at 200, 108 and
// 105 at 100.
// Where a CTA of many short items stands beside those of long ones it ends later still: 64 requests of 20 to 4,000 tokens, mostly
// short, 655 us with twelve and 605 with eight (its items have 3 tiles on average); 32 of 50 to 20,000 791 and 782 (13 to 16); 60
// of 200 to 8,000, 16/4 heads, 456 and 473 (18); 40 of 300 to 3,000 470 and 485 (22).
constexpr uint32_t kLongItemTiles = 20, kLeastItemTiles = 16;

template <int DG, int NSLOT, int W>
cudaError_t launch_f32(const AttendParams& p, uint32_t num_ctas, cudaStream_t stream) {
    auto kernel = attend_f32_kernel<DG, NSLOT, W>;
    static std::atomic<uint64_t> configured{0};
    // the largest head_dim sets the limit once; smaller ones fit under it
    cudaError_t err = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), static_cast<int>(f32_smem_bytes(128 * DG, NSLOT, W)), configured);
    if (err != cudaSuccess) return err;
    return launch_overlapped(kernel, num_ctas, W * 32, f32_smem_bytes(p.geo.head_dim, NSLOT, W), stream, p);
}

}  // namespace

// f32, head_dim a multiple of 32 up to 256 (a row is a whole number of 128-byte pieces), and arena, q and partial buffers
// on 16-byte boundaries.  Other head dims and buffers stay on the staged kernel.
bool attend_f32_profile(uint32_t dtype, uint32_t head_dim) {
    return dtype == PSI_DTYPE_F32 && head_dim >= 32 && head_dim <= 256 && head_dim % 32 == 0;
}

bool attend_f32_supported(const AttendParams& p) {
    auto aligned = [](const void* ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 15u) == 0; };
    return attend_f32_profile(p.dtype, p.geo.head_dim) && aligned(p.geo.pages) && aligned(p.q) && aligned(p.partial_o) && aligned(p.ext_o);
}

cudaError_t launch_attend_f32(const AttendParams& p, uint32_t num_ctas, cudaStream_t stream) {
    if (num_ctas == 0) return cudaSuccess;
    if (p.geo.head_dim > 128) return launch_f32<2, 3, 8>(p, num_ctas, stream);
    const bool long_items = p.item_tiles >= kLongItemTiles && p.least_item_tiles >= kLeastItemTiles;
    return long_items ? launch_f32<1, 4, 12>(p, num_ctas, stream) : launch_f32<1, 6, 8>(p, num_ctas, stream);
}

}  // namespace psi
