// The end of a unit whose items lie on several CTAs, for the map kernels beside attend_mma.cu: whoever stores a unit's last
// partial merges the unit, so that no reduce launch follows.
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
// (0 when empty), crates/inference-backend-metal/src/components/metal/gqa_split_kv_single_q_reduce.metal:27-48.  A thread owns
// four columns of a row; the pieces' statistics and values go out four pieces at a time.  `store(r, d, value, m, l)` takes
// columns [d, d + 4) of row r.
template <int kThreadCount, typename Store>
__device__ __forceinline__ void merge_unit(const AttendParams& p, const ItemView& v, const Store& store) {
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
            const float carry = top == -INFINITY ? 0.0f : exp2f(top - group_top);
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
    if (threadIdx.x == 0) p.unit_counters[v.reduce_unit] = 0;  // ready for the next launch
}

}  // namespace psi
