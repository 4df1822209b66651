// The stages the reference records directly before the page write, fused with it into one launch: per-head RMSNorm
// and RoPE of q (to q_out) and of k (straight into its page), and the V rows into their pages.
//
// Reference stages: crates/inference-executor-metal/src/attn/gqa/backend.rs:465-513 (q norm/rope, k norm/rope,
// kv_page_write), shader crates/inference-backend-metal/src/components/metal/rms_norm_rope.metal:7-82 and
// metal/gqa_kv_page_write.metal:20-52.  One warp per (token, head) row; the rounding order of the shader is kept:
// T(weight) * T(x * inv_rms) in the storage dtype T, rotation in f32, one final rounding to T.
//
// The inputs are addressed through strides, so the same launch also stands for the stage before those three: the
// de-interleave of the fused projection output (metal/gqa_qgkv_split.metal:14-42 with gates,
// metal/gqa_qkv_split.metal:13-36 without).  Its q, g, k and v rows are read where the projection left them; only the
// gate rows, which the attention epilogue wants contiguous, are copied out.
#include "device_common.cuh"
#include "launch_util.hpp"

namespace psi {

namespace {

template <uint32_t DTYPE>
__device__ __forceinline__ float round_to(float v) {
    if (DTYPE == PSI_DTYPE_BF16) return __bfloat162float(__float2bfloat16_rn(v));
    if (DTYPE == PSI_DTYPE_F16) return __half2float(__float2half_rn(v));
    return v;
}

constexpr int kPrepWarps = 8;

// Bit copy of one element (V rows and gate rows pass through unchanged, NaN payloads included).
__device__ __forceinline__ void copy_element(void* dst, uint64_t dst_index, const void* src, uint64_t src_index,
                                             uint32_t dtype) {
    if (dtype == PSI_DTYPE_F32) {
        static_cast<uint32_t*>(dst)[dst_index] = static_cast<const uint32_t*>(src)[src_index];
    } else {
        static_cast<uint16_t*>(dst)[dst_index] = static_cast<const uint16_t*>(src)[src_index];
    }
}

template <uint32_t DTYPE>
__global__ void __launch_bounds__(kPrepWarps * 32) norm_rope_append_kernel(PrepParams p) {
    await_previous_kernel();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t num_active = min(p.scalars[kScalarNumActiveTokens], p.num_total_tokens);
    const uint32_t hq = p.num_q_heads, hkv = p.geo.num_kv_heads, D = p.geo.head_dim;
    const uint64_t q_rows = static_cast<uint64_t>(num_active) * hq, kv_rows = static_cast<uint64_t>(num_active) * hkv;
    const uint64_t g_rows = p.g_in != nullptr ? q_rows : 0;
    const uint64_t row = static_cast<uint64_t>(blockIdx.x) * kPrepWarps + (threadIdx.x >> 5);
    if (row >= q_rows + 2 * kv_rows + g_rows) return;

    if (row >= q_rows + 2 * kv_rows) {
        // gate row: a bit copy out of the projection into the contiguous [T][Hq][D] the attention epilogue reads
        const uint64_t local = row - q_rows - 2 * kv_rows;
        const uint64_t src_base = (local / hq) * p.q_token_stride + (local % hq) * p.q_head_stride;
        for (uint32_t d = lane; d < D; d += 32) copy_element(p.g_out, local * D + d, p.g_in, src_base + d, DTYPE);
        return;
    }

    // which tensor, which (token, head)
    const bool is_q = row < q_rows, is_v = row >= q_rows + kv_rows;
    const uint64_t local = is_q ? row : (is_v ? row - q_rows - kv_rows : row - q_rows);
    const uint32_t heads = is_q ? hq : hkv;
    const uint32_t token = static_cast<uint32_t>(local / heads), head = static_cast<uint32_t>(local % heads);
    const void* src = is_q ? p.q_in : (is_v ? p.v_in : p.k_in);
    const uint64_t src_base = is_q ? token * p.q_token_stride + head * p.q_head_stride
                                   : token * p.kv_token_stride + static_cast<uint64_t>(head) * D;

    // destination: q_out row, or the row's place in its page
    void* dst = p.q_out;
    uint64_t dst_base = local * D;
    if (!is_q) {
        const uint32_t pos = p.flat_token_indices[token];
        const uint32_t page_index = pos / p.geo.tokens_per_page;
        uint32_t page_id;
        if (!checked_page_id(p.geo, table_row(p.geo, p.req_slots[token]), page_index, page_id)) return;  // write skipped
        dst = const_cast<void*>(p.geo.pages);
        dst_base = kv_row_offset(p.geo, page_id, head, pos % p.geo.tokens_per_page) + (is_v ? v_region_offset(p.geo) : 0);
    }
    if (is_v) {
        for (uint32_t d = lane; d < D; d += 32) copy_element(dst, dst_base + d, src, src_base + d, DTYPE);
        return;
    }

    float acc = 0.0f;
    for (uint32_t d = lane; d < D; d += 32) {
        const float x = load_as_float(src, src_base + d, DTYPE);
        acc += x * x;
    }
    acc = warp_sum(acc);
    const float inv_rms = 1.0f / sqrtf(acc / static_cast<float>(D) + p.eps);
    const __nv_bfloat16* weight = reinterpret_cast<const __nv_bfloat16*>(is_q ? p.q_weight : p.k_weight);
    const float position = static_cast<float>(p.flat_token_indices[token]);
    const uint32_t rope_half = p.rope_dim / 2;
    auto normed = [&](uint32_t d) {
        const float w = round_to<DTYPE>(__bfloat162float(weight[d]));
        return round_to<DTYPE>(w * round_to<DTYPE>(load_as_float(src, src_base + d, DTYPE) * inv_rms));
    };
    for (uint32_t d = lane; d < D; d += 32) {
        if (d < rope_half) {
            const uint32_t d2 = d + rope_half;
            const float x1 = normed(d), x2 = normed(d2);
            float s, c;
            sincosf(position * p.inverse_frequencies[d], &s, &c);
            store_from_float(dst, dst_base + d, DTYPE, p.attention_factor * (x1 * c - x2 * s));
            store_from_float(dst, dst_base + d2, DTYPE, p.attention_factor * (x1 * s + x2 * c));
        } else if (d >= p.rope_dim) {
            store_from_float(dst, dst_base + d, DTYPE, normed(d));
        }
    }
}

// 1 / sqrt(x): the device's own approximation and one Newton step, which leaves the last place of f32.  (A square root and a
// division, each with its range checks, took a fifth of a row's instructions.)  At 0 and infinity the step has no meaning.
__device__ __forceinline__ float inverse_root(float x) {
    const float y = rsqrtf(x), e = fmaf(-x * y, y, 1.0f);
    return isinf(y) || y == 0.0f ? y : fmaf(0.5f * y, e, y);
}

// Eight consecutive elements as a lane holds them.
template <uint32_t DTYPE>
struct Eight {
    static constexpr int kWords = DTYPE == PSI_DTYPE_F32 ? 8 : 4;
    uint4 raw[kWords / 4];
    __device__ __forceinline__ uint32_t* words() { return reinterpret_cast<uint32_t*>(raw); }
    __device__ __forceinline__ const uint32_t* words() const { return reinterpret_cast<const uint32_t*>(raw); }
    __device__ __forceinline__ void load(const void* base, uint64_t index) {
        const uint4* src = reinterpret_cast<const uint4*>(static_cast<const unsigned char*>(base) + index * (kWords / 2));
#pragma unroll
        for (int i = 0; i < kWords / 4; ++i) raw[i] = src[i];
    }
    __device__ __forceinline__ void store(void* base, uint64_t index) const {
        uint4* dst = reinterpret_cast<uint4*>(static_cast<unsigned char*>(base) + index * (kWords / 2));
#pragma unroll
        for (int i = 0; i < kWords / 4; ++i) dst[i] = raw[i];
    }
    __device__ __forceinline__ void widen(float (&v)[8]) const {
#pragma unroll
        for (int j = 0; j < kWords; ++j) {
            if constexpr (DTYPE == PSI_DTYPE_F32) {
                v[j] = __uint_as_float(words()[j]);
            } else {
                const uint32_t w = words()[j];
                const float2 pair = DTYPE == PSI_DTYPE_BF16 ? __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w))
                                                            : __half22float2(*reinterpret_cast<const __half2*>(&w));
                v[2 * j] = pair.x;
                v[2 * j + 1] = pair.y;
            }
        }
    }
    __device__ __forceinline__ void narrow(const float (&v)[8]) {
#pragma unroll
        for (int j = 0; j < kWords; ++j) {
            if constexpr (DTYPE == PSI_DTYPE_F32) {
                words()[j] = __float_as_uint(v[j]);
            } else if constexpr (DTYPE == PSI_DTYPE_BF16) {
                const __nv_bfloat162 pair = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
                words()[j] = *reinterpret_cast<const uint32_t*>(&pair);
            } else {
                const __half2 pair = __floats2half2_rn(v[2 * j], v[2 * j + 1]);
                words()[j] = *reinterpret_cast<const uint32_t*>(&pair);
            }
        }
    }
    // T(weight) * T(x * inv_rms), rounded to T.  In the 16-bit types the product of two such values is exact in f32, so
    // the packed multiplication, which rounds once, gives the same bits as an f32 product rounded to T.
    __device__ __forceinline__ void normalise(const float (&x)[8], float inv_rms, const Eight& weight) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = x[j] * inv_rms;
        narrow(v);
#pragma unroll
        for (int j = 0; j < kWords; ++j) {
            if constexpr (DTYPE == PSI_DTYPE_F32) {
                words()[j] = __float_as_uint(__uint_as_float(weight.words()[j]) * v[j]);
            } else if constexpr (DTYPE == PSI_DTYPE_BF16) {
                const __nv_bfloat162 pair = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(weight.words() + j),
                                                    *reinterpret_cast<const __nv_bfloat162*>(words() + j));
                words()[j] = *reinterpret_cast<const uint32_t*>(&pair);
            } else {
                const __half2 pair = __hmul2(*reinterpret_cast<const __half2*>(weight.words() + j),
                                             *reinterpret_cast<const __half2*>(words() + j));
                words()[j] = *reinterpret_cast<const uint32_t*>(&pair);
            }
        }
    }
};

// The same stage for head sizes whose row is a power-of-two number of lanes of eight elements (LPR lanes, 32 / LPR rows
// per warp) and 16-byte aligned buffers.  A CTA works on rows of one token (blockIdx.x): the token's sines and cosines
// are worked out once into shared memory instead of once per row, its page is looked up once, every lane moves 16 bytes
// at a time, the 16-bit types are rounded and multiplied in pairs, and a warp has kHeld rows in flight.  blockIdx.y deals
// the token's rows (q, k, v, gates) to CTAs.  Bound by issue slots on prompts (three quarters of them) and by latency on
// decode steps.  Measured: 4,667 prompt tokens of 24/4 heads x 256 with gates (267 MB) 63.5 us = 4.2 TB/s, 68 with a square
// root, a division and 64-bit row offsets in every row, 133 with a warp per row and one element per lane (and 65.6 with the
// rows' four sources chosen by selects in place of branches, 87 with a CTA for four tokens); a decode step of 32 tokens 5.2 us
// against 7.5 us.
constexpr int kHeld = 4;
constexpr uint64_t kRowsResidentCtas = 148 * 4;  // of the 16-bit instantiations (three an SM in f32, whose steps are short)

template <uint32_t DTYPE, int LPR>
__global__ void __launch_bounds__(kPrepWarps * 32, DTYPE == PSI_DTYPE_F32 ? 3 : 4) norm_rope_rows_kernel(PrepParams p) {
    constexpr uint32_t D = LPR * 8, kRows = 32 / LPR;
    __shared__ __align__(16) float2 turn_s[D / 2];  // (cosine, sine) of the position at every frequency, read two at a time
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t group = lane / LPR, sub = lane % LPR, d0 = sub * 8;
    const uint32_t token = blockIdx.x;
    if (token >= min(p.scalars[kScalarNumActiveTokens], p.num_total_tokens)) {
        await_previous_kernel();
        return;
    }
    const uint32_t hq = p.num_q_heads, hkv = p.geo.num_kv_heads;
    const uint32_t num_rows = hq + 2 * hkv + (p.g_in != nullptr ? hq : 0);  // q | k | v | gates
    const uint32_t stride = gridDim.y * kPrepWarps * kRows;
    const uint32_t first = (blockIdx.y * kPrepWarps + warp) * kRows + group;
    const uint32_t pos = p.flat_token_indices[token], slot = p.req_slots[token];

    // (a token's rows lie within 2^32 elements of its first one: launch_rows looks)
    const uint32_t q_step = static_cast<uint32_t>(p.q_head_stride);
    const uint64_t q_row = token * p.q_token_stride + d0, kv_row = token * p.kv_token_stride + d0;
    auto fetch = [&](uint32_t row, Eight<DTYPE>& x) {
        if (row < hq) x.load(p.q_in, q_row + row * q_step);
        else if (row < hq + hkv) x.load(p.k_in, kv_row + (row - hq) * D);
        else if (row < hq + 2 * hkv) x.load(p.v_in, kv_row + (row - hq - hkv) * D);
        else if (row < num_rows) x.load(p.g_in, q_row + (row - hq - 2 * hkv) * q_step);
    };
    // everything that needs only the plan, the table and the weights comes before the wait for the inputs
    Eight<DTYPE> q_weight, k_weight;  // the bf16 weights in T
    {
        Eight<PSI_DTYPE_BF16> w;
        float v[8];
        w.load(p.q_weight, d0);
        w.widen(v);
        q_weight.narrow(v);
        w.load(p.k_weight, d0);
        w.widen(v);
        k_weight.narrow(v);
    }
    uint32_t page_id = 0;
    bool page_ok = false;
    auto find_page = [&] { page_ok = checked_page_id(p.geo, table_row(p.geo, slot), pos / p.geo.tokens_per_page, page_id); };
    if (p.geo.table_settled != 0) find_page();
    const uint32_t rope_half = p.rope_dim / 2, half_lanes = rope_half / 8;
    for (uint32_t i = tid; i < rope_half; i += kPrepWarps * 32) {
        float s, c;
        sincosf(static_cast<float>(pos) * p.inverse_frequencies[i], &s, &c);
        turn_s[i] = make_float2(c, s);
    }
    await_previous_kernel();
    if (p.geo.table_settled == 0) find_page();
    const uint64_t page_row = kv_row_offset(p.geo, page_id, 0, pos % p.geo.tokens_per_page) + d0;
    Eight<DTYPE> held[kHeld];
#pragma unroll
    for (int i = 0; i < kHeld; ++i) fetch(first + i * stride, held[i]);
    __syncthreads();
    const bool in_rope = sub < 2 * half_lanes, low = sub < half_lanes;
    const uint32_t partner = in_rope ? (low ? lane + half_lanes : lane - half_lanes) : lane;
    const float2* turns = turn_s + (low ? d0 : d0 - rope_half);
    const uint32_t minus = !low ? 0u : (DTYPE == PSI_DTYPE_F32 ? 0x80000000u : 0x80008000u);  // x1 cos - x2 sin, x2 cos + x1 sin

    for (uint32_t base = first - group; base < num_rows; base += kHeld * stride) {
#pragma unroll
        for (int i = 0; i < kHeld; ++i) {
            if (base + i * stride >= num_rows) break;  // warp-uniform
            const uint32_t row = base + i * stride + group;
            const bool is_q = row < hq, is_k = !is_q && row < hq + hkv;
            Eight<DTYPE> x = held[i];
            fetch(row + kHeld * stride, held[i]);  // the row this place holds next, under the arithmetic of this one
            if (base + i * stride < hq + hkv) {  // warp-uniform: some row of this pass is normalised
                float v[8], acc = 0.0f;
                x.widen(v);
#pragma unroll
                for (int j = 0; j < 8; ++j) acc += v[j] * v[j];
#pragma unroll
                for (int offset = LPR / 2; offset > 0; offset >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, offset);
                const float inv_rms = inverse_root(acc / static_cast<float>(D) + p.eps);
                Eight<DTYPE> n, other;
                n.normalise(v, inv_rms, is_q ? q_weight : k_weight);
#pragma unroll
                for (int j = 0; j < Eight<DTYPE>::kWords; ++j)
                    other.words()[j] = __shfl_sync(0xFFFFFFFFu, n.words()[j], partner) ^ minus;
                if (in_rope) {
                    float mine[8], theirs[8];
                    n.widen(mine);
                    other.widen(theirs);
#pragma unroll
                    for (int j = 0; j < 8; j += 2) {
                        const float4 turn = *reinterpret_cast<const float4*>(turns + j);  // two frequencies
                        mine[j] = theirs[j] * turn.y + mine[j] * turn.x;
                        mine[j + 1] = theirs[j + 1] * turn.w + mine[j + 1] * turn.z;
                    }
                    if (p.attention_factor != 1.0f) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) mine[j] *= p.attention_factor;
                    }
                    n.narrow(mine);
                }
                if (is_q || is_k) x = n;
            }
            if (is_q) {
                x.store(p.q_out, (static_cast<uint64_t>(token) * hq + row) * D + d0);
            } else if (row < hq + 2 * hkv) {
                const uint64_t head_row = static_cast<uint64_t>(row - hq - (is_k ? 0 : hkv)) * p.geo.tokens_per_page * D;
                if (page_ok) x.store(const_cast<void*>(p.geo.pages), page_row + head_row + (is_k ? 0 : v_region_offset(p.geo)));
            } else if (row < num_rows) {
                x.store(p.g_out, (static_cast<uint64_t>(token) * hq + (row - hq - 2 * hkv)) * D + d0);
            }
        }
    }
}

bool aligned16(const void* ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 15u) == 0; }

template <uint32_t DTYPE>
bool launch_rows(const PrepParams& p, cudaStream_t stream, cudaError_t& status) {
    const uint32_t d = p.geo.head_dim;
    if ((d != 64 && d != 128 && d != 256) || p.rope_dim % 16 != 0 || !aligned16(p.q_in) || !aligned16(p.k_in) || !aligned16(p.v_in) ||
        !aligned16(p.g_in) || !aligned16(p.q_out) || !aligned16(p.g_out) || !aligned16(p.geo.pages) || !aligned16(p.q_weight) ||
        !aligned16(p.k_weight)) {
        return false;
    }
    // Rows per warp: one while the device has room for every CTA at once (a decode step: nothing but latency), eight
    // when the step is long: the per-CTA part is then spread over more rows (a prompt step of 4,667 tokens and two
    // layers measured 675 us with one, 551 with four, 538 with eight).
    const uint32_t rows = p.num_q_heads * (p.g_in != nullptr ? 2 : 1) + 2 * p.geo.num_kv_heads;
    const uint32_t rows_per_cta = kPrepWarps * (256 / d);
    const uint64_t ctas = static_cast<uint64_t>(p.num_total_tokens) * ((rows + rows_per_cta - 1) / rows_per_cta);
    const uint32_t per_warp = static_cast<uint32_t>(ctas <= kRowsResidentCtas ? 1 : 8);
    const uint32_t split = (rows + rows_per_cta * per_warp - 1) / (rows_per_cta * per_warp);
    if (split > 65535 || p.q_head_stride * p.num_q_heads > 0xFFFFFFFFull || uint64_t(p.geo.num_kv_heads) * d > 0xFFFFFFFFull) return false;
    const dim3 grid(p.num_total_tokens, split);
    auto kernel = d == 64 ? norm_rope_rows_kernel<DTYPE, 8> : (d == 128 ? norm_rope_rows_kernel<DTYPE, 16> : norm_rope_rows_kernel<DTYPE, 32>);
    status = launch_overlapped(kernel, grid, kPrepWarps * 32, 0, stream, p);
    return true;
}

}  // namespace

cudaError_t launch_norm_rope_append(const PrepParams& p, cudaStream_t stream) {
    const uint64_t rows = static_cast<uint64_t>(p.num_total_tokens) *
                          ((p.g_in != nullptr ? 2ull : 1ull) * p.num_q_heads + 2ull * p.geo.num_kv_heads);
    if (rows == 0) return cudaSuccess;
    cudaError_t status = cudaSuccess;
    if (p.dtype == PSI_DTYPE_F32 ? launch_rows<PSI_DTYPE_F32>(p, stream, status)
                                 : (p.dtype == PSI_DTYPE_BF16 ? launch_rows<PSI_DTYPE_BF16>(p, stream, status)
                                                              : launch_rows<PSI_DTYPE_F16>(p, stream, status))) {
        return status;
    }
    const unsigned blocks = static_cast<unsigned>((rows + kPrepWarps - 1) / kPrepWarps);
    auto kernel = p.dtype == PSI_DTYPE_F32 ? norm_rope_append_kernel<PSI_DTYPE_F32>
                                           : (p.dtype == PSI_DTYPE_BF16 ? norm_rope_append_kernel<PSI_DTYPE_BF16> : norm_rope_append_kernel<PSI_DTYPE_F16>);
    return launch_overlapped(kernel, blocks, kPrepWarps * 32, 0, stream, p);
}

}  // namespace psi
