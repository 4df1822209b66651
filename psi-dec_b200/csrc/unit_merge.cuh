// The end of a unit whose items lie on several CTAs, for the map kernels beside attend_mma.cu: where a launch says so
// (AttendParams::merges), whoever stores a unit's last partial merges the unit, so that no reduce launch follows.
#pragma once

#include "mma_common.cuh"

namespace psi {

// Whether this CTA delivered the last partial of the item's unit.  Called by the whole CTA after its partial stores; the
// barrier orders them before thread 0's fence, which is cumulative, and the second fence orders the count before the reads
// of the other pieces' partials.
__device__ __forceinline__ bool delivers_last_partial(const AttendParams& p, const ItemView& v, uint32_t& arrival_s) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        arrival_s = atomicAdd(p.unit_counters + v.reduce_unit, 1u);
        __threadfence();
    }
    __syncthreads();
    return arrival_s == v.unit_num_items - 1;
}

// Merges the unit's partials: M = max m_i, w_i = 2^(m_i - M) * l_i (0 when m_i is not finite), out = sum w_i o_i / sum w_i
// (0 when empty), as the reduce launch has it (crates/inference-backend-metal/src/components/metal/gqa_split_kv_single_q_reduce.metal:27-48).  A thread owns
// four columns of a row; the pieces' statistics and values go out four pieces at a time.  `store(r, d, value, m, l)` takes
// columns [d, d + 4) of row r.
template <int kThreadCount, typename Store>
__device__ __forceinline__ void merge_few(const AttendParams& p, const ItemView& v, const Store& store) {
    const uint32_t D = p.geo.head_dim, columns = D / 4, n = v.unit_num_items;
    for (uint32_t i = threadIdx.x; i < v.rows * columns; i += kThreadCount) {
        const uint32_t r = i / columns, d = 4 * (i % columns);
        const uint64_t row0 = static_cast<uint64_t>(v.unit_first_slot) * kMaxRows + r;
        float top = -INFINITY, sum = 0.0f;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (uint32_t s0 = 0; s0 < n; s0 += 4) {
            float pm[4], pl[4];
            float4 part[4];
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
                const uint64_t row = row0 + static_cast<uint64_t>(min(s0 + k, n - 1)) * kMaxRows;
                pm[k] = __ldcg(p.partial_m + row);
                pl[k] = __ldcg(p.partial_l + row);
                part[k] = __ldcg(reinterpret_cast<const float4*>(p.partial_o + row * D + d));
            }
            float group_top = top;
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k)
                if (s0 + k < n) group_top = fmaxf(group_top, pm[k]);
            const float carry = top == group_top ? 1.0f : exp2f(top - group_top);  // (also at +Inf, whose pieces weigh 0)
            sum *= carry;
            acc.x *= carry;
            acc.y *= carry;
            acc.z *= carry;
            acc.w *= carry;
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
                if (s0 + k >= n) break;
                const float weight = isfinite(pm[k]) ? exp2f(pm[k] - group_top) * pl[k] : 0.0f;
                sum += weight;
                acc.x += weight * part[k].x;
                acc.y += weight * part[k].y;
                acc.z += weight * part[k].z;
                acc.w += weight * part[k].w;
            }
            top = group_top;
        }
        const bool any = sum > 0.0f;
        store(r, d, make_float4(any ? acc.x / sum : 0.0f, any ? acc.y / sum : 0.0f, any ? acc.z / sum : 0.0f, any ? acc.w / sum : 0.0f), top, sum);
    }
}

// The same for units of many pieces: eight at a time, and where the rows leave threads idle, two or four of them (`ways`) share the
// pieces of a column.
template <int kThreadCount, typename Store>
__device__ __forceinline__ void merge_many(const AttendParams& p, const ItemView& v, uint32_t ways, const Store& store) {
    constexpr uint32_t kAtOnce = 8;
    const uint32_t D = p.geo.head_dim, columns = D / 4, n = v.unit_num_items, outputs = v.rows * columns;
    const uint32_t way = threadIdx.x & (ways - 1), step = kThreadCount / ways;
    for (uint32_t first = 0; first < outputs; first += step) {
        const uint32_t mine = first + threadIdx.x / ways, i = min(mine, outputs - 1);
        const uint32_t r = i / columns, d = 4 * (i % columns);
        const uint64_t row0 = static_cast<uint64_t>(v.unit_first_slot) * kMaxRows + r;
        float top = -INFINITY, sum = 0.0f;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (uint32_t s0 = way; s0 < n; s0 += kAtOnce * ways) {
            float pm[kAtOnce], pl[kAtOnce];
            float4 part[kAtOnce];
#pragma unroll
            for (uint32_t k = 0; k < kAtOnce; ++k) {
                const uint64_t row = row0 + static_cast<uint64_t>(min(s0 + k * ways, n - 1)) * kMaxRows;
                pm[k] = __ldcg(p.partial_m + row);
                pl[k] = __ldcg(p.partial_l + row);
                part[k] = __ldcg(reinterpret_cast<const float4*>(p.partial_o + row * D + d));
            }
            float group_top = top;
#pragma unroll
            for (uint32_t k = 0; k < kAtOnce; ++k)
                if (s0 + k * ways < n) group_top = fmaxf(group_top, pm[k]);
            const float carry = top == group_top ? 1.0f : exp2f(top - group_top);  // (also at +Inf, whose pieces weigh 0)
            sum *= carry;
            acc.x *= carry;
            acc.y *= carry;
            acc.z *= carry;
            acc.w *= carry;
#pragma unroll
            for (uint32_t k = 0; k < kAtOnce; ++k) {
                if (s0 + k * ways >= n) break;
                const float weight = isfinite(pm[k]) ? exp2f(pm[k] - group_top) * pl[k] : 0.0f;
                sum += weight;
                acc.x += weight * part[k].x;
                acc.y += weight * part[k].y;
                acc.z += weight * part[k].z;
                acc.w += weight * part[k].w;
            }
            top = group_top;
        }
        for (uint32_t x = 1; x < ways; x *= 2) {  // (the same number for the whole CTA)
            const float other = __shfl_xor_sync(0xFFFFFFFFu, top, x), both = fmaxf(top, other);
            const float carry = top == both ? 1.0f : exp2f(top - both);
            auto add_other = [&](float& value) {
                value *= carry;
                value += __shfl_xor_sync(0xFFFFFFFFu, value, x);
            };
            add_other(sum);
            add_other(acc.x);
            add_other(acc.y);
            add_other(acc.z);
            add_other(acc.w);
            top = both;
        }
        if (way != 0 || mine >= outputs) continue;
        const bool any = sum > 0.0f;
        store(r, d, make_float4(any ? acc.x / sum : 0.0f, any ? acc.y / sum : 0.0f, any ? acc.z / sum : 0.0f, any ? acc.w / sum : 0.0f), top, sum);
    }
}

// (Both inline: a call takes 6 us a layer.  A launch of sixteen warps, whose items are long, keeps to the first form: what the second
// one does to the rest of its code took 1 to 2 % of a step.)
template <int kThreadCount, typename Store>
__device__ __forceinline__ void merge_unit(const AttendParams& p, const ItemView& v, const Store& store) {
    if constexpr (kThreadCount > 384) {
        merge_few<kThreadCount>(p, v, store);
    } else {
        const MergeShape shape = merge_shape(v.unit_num_items, v.rows, p.geo.head_dim, kThreadCount);
        if (shape.at_once == 4) merge_few<kThreadCount>(p, v, store);
        else merge_many<kThreadCount>(p, v, shape.ways, store);
    }
    if (threadIdx.x == 0) p.unit_counters[v.reduce_unit] = 0;  // ready for the next launch
}

}  // namespace psi
